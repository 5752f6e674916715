"""Products of a few rows that lie ready (csrc/skinny_direct.cu): plain rows in every form of the launch, the rows that a residual product leaves for the
norm behind it, and products of such rows, against the same in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _lib():
    from velomind_b200.kernels.library import library
    return library()


def _p(t):                                                          # (of a tensor that a name holds until the kernel has run)
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _i(v):
    return ctypes.c_int(int(v))


def _f(v):
    return ctypes.c_float(v)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _bf(x):
    return x.to(torch.bfloat16).to(DEV)


# eight and sixteen warps (items up to the number of SMs, K to 1,024 and beyond), one and two pairs of column tiles, blocks of K that a warp has not (K = 32),
# has one of and refills, an odd last pair, N of whole pairs and not, rows at the edges of their tiles
SIZES = [(1, 200, 32), (8, 576, 576), (9, 960, 960), (16, 144, 1536), (17, 328, 2560), (32, 576, 4128), (3, 2416, 1024), (8, 2400, 96), (25, 3072, 576), (12, 2576, 736), (5, 2512, 2080)]


@pytest.mark.parametrize("M,N,K", SIZES)
def test_products_of_plain_rows(M, N, K):
    """Products of bfloat16 are exact in 32 bits; a sum of K of them in 32 bits is off by at most K 2^-24 of the sum of magnitudes, a store to bfloat16 by 2^-8."""
    g = torch.Generator().manual_seed(M + N + K)
    x, w = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g) * 0.1)
    want, bound = x.double() @ w.double().T, (x.double().abs() @ w.double().abs().T) * K * 2.0 ** -24 + 1e-30
    out = torch.full((M, N + 3), float("nan"), device=DEV)
    assert _lib().vm_skinny_linear(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(N), _i(K), _p(out), _i(N + 3), _i(1), _p(None), _p(None), _stream()) == 0
    assert bool(((out[:, :N].double() - want).abs() <= bound).all()) and bool(torch.isnan(out[:, N:]).all())
    low = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert _lib().vm_skinny_linear(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(N), _i(K), _p(low), _i(N), _i(0), _p(None), _p(None), _stream()) == 0
    assert bool(((low.double() - want).abs() <= bound + want.abs() * 2.0 ** -8).all())
    half = N // 16 * 8
    unit = torch.full((M, half), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert _lib().vm_skinny_gated(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(half), _i(K), _i(0), _p(unit), _p(None), _stream()) == 0
    gate, up = want[:, :half], want[:, half:2 * half]
    silu = gate / (1 + torch.exp(-gate))                             # (slope at most 1.1; the exponential and the quotient: a few 2^-24 of the result)
    loose = 1.1 * bound[:, :half] * up.abs() + (silu.abs() + bound[:, :half]) * bound[:, half:2 * half]
    assert bool(((unit.double() - silu * up).abs() <= loose + (silu * up).abs() * (2.0 ** -8 + 2.0 ** -20) + 1e-30).all())


# either side of the rule: 8 rows and 9 of 18 MB and more, 17 of 10 MB and more, column tiles of eight, two pairs of tiles a block, blocks for one SM and a half
@pytest.mark.parametrize("form,M,N,K,ring", [("gated", 9, 6144, 2048, True), ("gated", 8, 6144, 2048, False), ("sum", 16, 6144, 1536, True), ("sum", 17, 5632, 960, True), ("sum", 17, 5120, 960, False),
                                             ("gated", 32, 16384, 1024, True), ("gated", 17, 12288, 960, False), ("store", 17, 4088, 1280, True), ("store", 5, 4088, 4096, True), ("store", 9, 4088, 2048, True),
                                             ("store", 16, 3200, 4096, False), ("sum", 32, 3072, 2048, False)])
def test_plain_rows_of_many_weights(form, M, N, K, ring):
    """Where memory sets the time, plain rows take the kernel that stages them once a CTA: its bits; and either kernel's sums are right, bounds as above."""
    g = torch.Generator().manual_seed(M + N + K)
    x, w = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g) * 0.1)
    h0, err = torch.randn(M, N, generator=g).to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(variant):
        out, h = torch.full((M, N), float("nan"), device=DEV), h0.clone()
        unit = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
        _lib().vm_skinny_variant(_i(variant))
        try:
            if form == "gated":
                rc = _lib().vm_skinny_gated(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(N // 2), _i(K), _i(0), _p(unit), _p(err), _stream())
            else:
                rc = _lib().vm_skinny_linear(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(N), _i(K), _p(out), _i(N), _i(1), _p(h if form == "sum" else None), _p(err), _stream())
        finally:
            _lib().vm_skinny_variant(_i(0))
        assert rc == 0
        return {"gated": unit, "sum": h, "store": out}[form]

    got = run(0)
    if ring:
        assert torch.equal(got, run(2))
    want = x.double() @ w.double().T
    bound = (x.double().abs() @ w.double().abs().T + (h0.double().abs() if form == "sum" else 0)) * (K + 1) * 2.0 ** -24
    if form == "gated":
        gate, up = want[:, :N // 2], want[:, N // 2:]
        bg, bu = bound[:, :N // 2], bound[:, N // 2:]
        silu = gate / (1 + torch.exp(-gate))
        want, bound = silu * up, 1.1 * bg * up.abs() + (silu.abs() + bg) * bu + (silu * up).abs() * (2.0 ** -8 + 2.0 ** -20) + 1e-30
    elif form == "sum":
        want = want + h0.double()
    assert bool(((got.double() - want).abs() <= bound).all()) and int(err.item()) == 0


@pytest.mark.parametrize("M,N,K", SIZES)
def test_rows_left_ready(M, N, K):
    """The residual sum, the rows for the next product and their sums of squares."""
    g = torch.Generator().manual_seed(2 * M + N + K)
    x, w = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g) * 0.1)
    h0, nw = torch.randn(M, N, generator=g).to(DEV), (torch.rand(N, generator=g) + 0.5).to(DEV)
    want = h0.double() + x.double() @ w.double().T
    bound = (x.double().abs() @ w.double().abs().T + h0.double().abs()) * (K + 1) * 2.0 ** -24
    plain = h0.clone()
    assert _lib().vm_skinny_linear(_p(x), _i(0), _p(None), _f(0), _p(w), _i(M), _i(N), _i(K), _p(None), _i(N), _i(0), _p(plain), _p(None), _stream()) == 0
    assert bool(((plain.double() - want).abs() <= bound).all())
    parts = _lib().vm_skinny_ready_parts(_i(N))
    assert parts % 4 == 0 and parts >= N // 16
    h, ready, squares = h0.clone(), torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV), torch.full((M, parts), float("nan"), device=DEV)
    assert _lib().vm_skinny_residual_ready(_p(x), _p(w), _i(M), _i(N), _i(K), _p(h), _p(nw), _p(ready), _p(squares), _stream()) == 0
    assert torch.equal(h, plain)
    assert torch.equal(ready, (h * nw).to(torch.bfloat16))
    full = (h.double() ** 2).sum(1)
    assert bool(((squares.double().sum(1) - full).abs() <= full * 20 * 2.0 ** -24).all())      # (16 squares and their sums in 32 bits a part)


@pytest.mark.parametrize("M", [1, 8, 9, 32])
@pytest.mark.parametrize("H,Hkv,D,K", [(9, 3, 64, 576), (2, 1, 16, 224), (32, 32, 64, 2048)])
def test_products_of_ready_rows(M, H, Hkv, D, K):
    """Norm, product, rotation and cache write from rows that carry the norm's weight: the same as from the float32 rows, to the last bits of the sums."""
    g = torch.Generator().manual_seed(M + H)
    h, nw = torch.randn(M, K, generator=g).to(DEV), (torch.rand(K, generator=g) + 0.5).to(DEV)
    w = _bf(torch.randn((H + 2 * Hkv) * D, K, generator=g) * 0.05)
    parts = _lib().vm_skinny_ready_parts(_i(K))
    ready, squares = (h * nw).to(torch.bfloat16), torch.zeros(M, parts, device=DEV)
    squares[:, 0] = (h.double() ** 2).sum(1).float() * 0.25
    squares[:, -1] = squares[:, 0] * 3
    pos = torch.randint(0, 120, (M,), generator=g).int().to(DEV)
    seq = torch.arange(M, dtype=torch.int32, device=DEV)
    table = torch.randperm(2 * M, generator=g).int().reshape(M, 2).to(DEV)
    freq = (10000.0 ** (-torch.arange(D // 2) / (D // 2))).float().to(DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(a, pro, weight):
        q = torch.full((M, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        kp, vp = (torch.zeros(2 * M, Hkv, 64, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        rc = _lib().vm_skinny_qkv_rope(_p(a), _i(pro), _p(weight), _f(1e-5), _p(w), _i(M), _i(K), _p(q), _p(pos), _p(seq), _p(table), _i(2), _p(freq), _i(D), _i(0),
                                       _p(kp), _p(vp), _i(H), _i(Hkv), _i(D), _i(2 * M), _p(err), _stream())
        assert (rc, int(err.item())) == (0, 0)
        return q, kp, vp
    for a, b in zip(run(ready, 2, squares), run(h, 1, nw)):
        scale = float(b.double().abs().max())
        # the same bfloat16 operands and 32-bit sums in another order: results differ by one rounding to bfloat16 at most
        assert float((a.double() - b.double()).abs().max()) <= scale * 2.0 ** -8
    out, plain = (torch.full((M, w.shape[0]), float("nan"), device=DEV) for _ in range(2))
    for o, a, pro, weight in ((out, ready, 2, squares), (plain, h, 1, nw)):
        assert _lib().vm_skinny_linear(_p(a), _i(pro), _p(weight), _f(1e-5), _p(w), _i(M), _i(w.shape[0]), _i(K), _p(o), _i(w.shape[0]), _i(1), _p(None), _p(None), _stream()) == 0
    assert float((out - plain).abs().max()) <= K * 2.0 ** -22 * float((ready.double().abs() @ w.double().abs().T).max())


def test_more_rows_than_the_kernel_takes():
    """33 rows and more: the rows stay with the other kernel, the ready forms are refused."""
    g = torch.Generator().manual_seed(5)
    x, w = _bf(torch.randn(40, 96, generator=g)), _bf(torch.randn(64, 96, generator=g))
    out = torch.zeros(40, 64, device=DEV)
    assert _lib().vm_skinny_linear(_p(x), _i(0), _p(None), _f(0), _p(w), _i(40), _i(64), _i(96), _p(out), _i(64), _i(1), _p(None), _p(None), _stream()) == 0
    assert float((out.double() - x.double() @ w.double().T).abs().max()) <= 1e-3
    h, nw, squares = torch.zeros(40, 64, device=DEV), torch.ones(64, device=DEV), torch.zeros(40, 8, device=DEV)
    assert _lib().vm_skinny_residual_ready(_p(x), _p(w), _i(40), _i(64), _i(96), _p(h), _p(nw), _p(out), _p(squares), _stream()) == -1
    assert _lib().vm_skinny_linear(_p(x), _i(2), _p(squares), _f(1e-5), _p(w), _i(40), _i(64), _i(96), _p(out), _i(64), _i(1), _p(None), _p(None), _stream()) == -1


@pytest.mark.parametrize("M,N,K", [(1, 64, 96), (8, 576, 576), (32, 144, 1536)])
def test_ready_rows_into_a_residual_sum_are_refused(M, N, K):
    g = torch.Generator().manual_seed(6)
    x, w, h = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g)), torch.randn(M, N, generator=g).to(DEV)
    squares, before = torch.ones(M, _lib().vm_skinny_ready_parts(_i(K)), device=DEV), h.clone()
    assert _lib().vm_skinny_linear(_p(x), _i(2), _p(squares), _f(1e-5), _p(w), _i(M), _i(N), _i(K), _p(None), _i(N), _i(0), _p(h), _p(None), _stream()) == -1
    torch.cuda.synchronize()
    assert torch.equal(h, before)
