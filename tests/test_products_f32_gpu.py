"""Float32 products of many rows on the tensor cores (csrc/products_f32.cu) against the same in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _product(x, w, rows=None):
    from velomind_b200.kernels.library import library
    T, K = x.shape
    out = torch.full((T + 1, w.shape[0]), float("nan"), device=DEV)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (x, w, out)]
    rc = library().vm_products_f32(p[0], ctypes.c_longlong(x.stride(0)), p[1], p[2], T, w.shape[0], K, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and bool(torch.isnan(out[T]).all())
    return out[:T]


# one tile and several, rows, columns and K at the edges of theirs, 32 and 64 columns a block, columns that are no multiple of four, K below one step
SIZES = [(1, 32, 4), (9, 33, 60), (127, 128, 64), (128, 576, 576), (129, 100, 68), (300, 960, 1000), (446, 3072, 576), (257, 97, 1536), (500, 5632, 1024), (1100, 1030, 132)]


@pytest.mark.parametrize("T,N,K", SIZES)
def test_products(T, N, K):
    """What the three parts leave out is below 2^-24 of a product, a sum of K of them in 32 bits off by at most K 2^-24 of the sum of magnitudes; on the whole
    the sums, rounded every 64 places, stay within a few units of the last place."""
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    wide = torch.randn(T, K + 8, generator=g, device=DEV)
    x, w = wide[:, :K], torch.randn(N, K, generator=g, device=DEV) * 0.1
    got, want = _product(x, w).double(), x.double() @ w.double().T
    assert bool(((got - want).abs() <= (x.double().abs() @ w.double().abs().T) * (K + 1) * 2.0 ** -24).all())
    assert float((got - want).norm() / want.norm()) < 2.0 ** -22
    again = _product(x[: (T + 1) // 2], w)                           # a row's result does not depend on the other rows
    assert torch.equal(again.double(), got[: (T + 1) // 2])


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38, 1e-38, 0.0])
def test_values_beyond_the_parts(value):
    """Infinities, NaN and values that bfloat16 rounds to infinity come out as in any float32 product, in x and in W; the smallest ones as far as 32 bits go."""
    g = torch.Generator(device=DEV).manual_seed(5)
    T, N, K = 150, 70, 200
    x, w = torch.randn(T, K, generator=g, device=DEV) * 0.01, torch.randn(N, K, generator=g, device=DEV) * 0.01
    x[140, 77] = value
    w[3, 5] = value
    got, want = _product(x, w).double(), x.double() @ w.double().T
    top = torch.finfo(torch.float32).max
    finite = torch.isfinite(want) & (want.abs() <= top)
    bound = (x.double().abs() @ w.double().abs().T) * (K + 1) * 2.0 ** -24
    assert bool(((got - want).abs() <= bound)[finite].all())
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])


@pytest.mark.parametrize("scale_x,scale_w", [(1e-36, 0.1), (1e-38, 1.0), (1e-42, 30.0), (0.1, 1e-37), (1e-20, 1e-18), (1e-30, 1e-10), (1e-42, 1e30)])
@pytest.mark.parametrize("T,N,K", [(150, 70, 200), (40, 33, 576)])
def test_the_smallest_values(T, N, K, scale_x, scale_w):
    """Rows below what the parts hold, in x and in W, and products below the smallest normal number: as far as 32 bits go, and half of the smallest number a term."""
    g = torch.Generator(device=DEV).manual_seed(6)
    x, w = torch.randn(T, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    x[::2] *= scale_x
    w[::3] *= scale_w
    x[4], w[6] = 0.0, 0.0
    got, want = _product(x, w).double(), x.double() @ w.double().T
    assert bool(((got - want).abs() <= (x.double().abs() @ w.double().abs().T) * (K + 1) * 2.0 ** -24 + K * 2.0 ** -150).all())
    assert bool((got[4] == 0).all()) and bool((got[:, 6] == 0).all())


@pytest.mark.parametrize("big_x,big_w", [(1e32, 1e10), (1.7e38, 3.1), (1e30, 1e20), (-3e38, 2e38)])
def test_products_beyond_the_range(big_x, big_w):
    """Finite operands whose product passes float32's range, with low mantissa bits of either sign: an infinity of the product's sign, no NaN."""
    g = torch.Generator(device=DEV).manual_seed(7)
    T, N, K = 140, 96, 192
    x, w = torch.randn(T, K, generator=g, device=DEV) * 0.01, torch.randn(N, K, generator=g, device=DEV) * 0.01
    x[5:60, 100] = big_x * (1 + torch.rand(55, generator=g, device=DEV) * 0.01)
    w[3:40, 100] = big_w * (1 + torch.rand(37, generator=g, device=DEV) * 0.01)
    w[20:40, 100] *= -1
    got, want = _product(x, w), x.double() @ w.double().T
    beyond = torch.zeros(T, N, dtype=torch.bool, device=DEV)
    beyond[5:60, 3:40] = True
    assert bool((want[beyond].abs() > torch.finfo(torch.float32).max).all()) and torch.equal(got[beyond].double(), torch.sign(want[beyond]) * float("inf"))
    bound = (x.double().abs() @ w.double().abs().T) * (K + 1) * 2.0 ** -24
    assert bool(((got.double() - want).abs() <= bound)[~beyond].all())


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38, 1e-41])
def test_rows_beside_an_odd_one_keep_their_bits(value):
    """A row's result does not depend on the others of its tile, nor a column's on its neighbours, whatever those hold."""
    g = torch.Generator(device=DEV).manual_seed(8)
    x, w = torch.randn(200, 300, generator=g, device=DEV), torch.randn(130, 300, generator=g, device=DEV)
    plain = _product(x, w)
    x[40], x[150, 7], w[65, 299] = value, value, value
    got = _product(x, w)
    rows, columns = torch.ones(200, dtype=torch.bool, device=DEV), torch.ones(130, dtype=torch.bool, device=DEV)
    rows[40], rows[150], columns[65] = False, False, False
    assert torch.equal(got[rows][:, columns], plain[rows][:, columns])
