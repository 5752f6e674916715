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
