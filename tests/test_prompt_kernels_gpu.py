"""Kernels of a prompt's mixers at the places where their launches change form: the preparation with a norm over the whole projection
(csrc/mixer_prep.cu)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _lib():
    from velomind_b200.kernels.library import library
    lib = library()
    for name in ("vm_delta_scratch_floats", "vm_mlstm_chunk_scratch_floats"):
        getattr(lib, name).restype = ctypes.c_longlong
    return lib


def _p(t):                                                          # (of a tensor that a name holds until the kernel has run)
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _i(v):
    return ctypes.c_int(int(v))


def _l(v):
    return ctypes.c_longlong(int(v))


def _f(v):
    return ctypes.c_float(v)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ints(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _cu(new):
    return _ints([sum(new[:i]) for i in range(len(new) + 1)])


@pytest.mark.parametrize("H,G,D", [(3, 1, 64), (22, 10, 64), (20, 12, 32), (32, 0, 64), (25, 8, 64)])
@pytest.mark.parametrize("K", [0, 3])
@pytest.mark.parametrize("T", [7, 140, 320, 1100])
def test_the_normed_preparation(T, K, H, G, D):
    """One block a token with a warp per head (more heads with the values than warps: two turns), and the kernel of many tokens: queries, keys and values
    of a prompt against 64 bits.  Sums of up to 2,048 squares and three taps in 32 bits; angles up to T rounded to 2^-24 of themselves."""
    g = torch.Generator().manual_seed(T + H)
    C, pages = (H + 2 * G) * D, -(-T // 64)
    x, bias = torch.randn(T, C, generator=g).to(DEV), torch.randn(C, generator=g).to(DEV)
    taps = torch.randn(C, K, generator=g).to(DEV) if K else None
    qn, kn = (torch.rand(n * D, generator=g).to(DEV) + 0.5 for n in (H, max(G, 1)))
    freq = (10000.0 ** (-torch.arange(D // 2) / (D // 2))).float().to(DEV)
    state = torch.zeros(1, max(K - 1, 1) * C, device=DEV)
    q = torch.full((T, H * D), float("nan"), device=DEV)
    kp, vp = (torch.full((pages, G, 64, D), float("nan"), device=DEV) if G else None for _ in range(2))
    table, err, zero = _ints([list(range(pages))]), _ints([0]), _ints([0])
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seq, cu = torch.zeros_like(pos), _cu([T])
    rc = _lib().vm_mixer_prepare(_p(x), _i(C), _p(bias), _p(taps), _i(K), _p(state if K else None), _l(state.shape[1]), _i(0), _p(qn), _p(kn), _f(1e-5), _p(freq), _i(D), _i(0),
                                 _p(pos), _p(seq), _p(cu), _p(zero), _p(table), _i(pages), _p(q), _p(kp), _p(vp), _i(pages), _i(T), _i(1), _i(H), _i(G),
                                 _i(D), _i(D), _i(0), _i(0), _i(0), _i(0), _p(err), _stream())
    assert (rc, int(err.item())) == (0, 0)
    y = x.double() + bias.double()
    if K:
        past = torch.cat([torch.zeros(K - 1, C, device=DEV, dtype=torch.float64), y])
        y = sum(past[j:j + T] * taps.double()[:, j] for j in range(K))
    angle = (pos.float()[:, None] * freq).double()
    cos, sin = (f(angle)[:, None] for f in (torch.cos, torch.sin))

    def turned(z, w, n):
        z = z / torch.sqrt((z ** 2).mean(-1, keepdim=True) + 1e-5) * w.double()
        a, b = z.reshape(T, n, 2, D // 2).unbind(2)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    assert float((q.reshape(T, H, D).double() - turned(y[:, :H * D], qn, H)).abs().max()) <= 2e-5
    if G:
        rows = lambda pool: pool.transpose(1, 2).reshape(pages * 64, G, D)[:T].double()
        assert float((rows(kp) - turned(y[:, H * D:(H + G) * D], kn, G)).abs().max()) <= 2e-5
        assert float((rows(vp) - y[:, (H + G) * D:].reshape(T, G, D)).abs().max()) <= 2e-5
    if K > 1:
        assert torch.equal(state.reshape(K - 1, C), x[T - K + 1:])
