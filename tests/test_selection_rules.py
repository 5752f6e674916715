"""Rules by which the launchers choose a kernel, on the host: the sides that were measured stay on the side that was faster."""


def test_float32_products_of_few_rows_stay_with_the_library():
    """Up to 32 rows the library is the faster one whatever the columns (9 rows, 49,152 x 576: 50 us against 79); from 33 on it is not (csrc/products_f32.cu)."""
    from velomind_b200.kernels.library import library
    pays = library().vm_products_f32_pays
    for rows, columns, want in ((9, 49152, 0), (32, 49152, 0), (32, 1 << 20, 0), (33, 49152, 1), (64, 5632, 1), (446, 3072, 1), (446, 576, 0), (130, 960, 0), (0, 0, 0)):
        assert pays(rows, columns) == want, (rows, columns)
