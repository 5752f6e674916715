"""Kernels of a prompt's mixers at the places where their launches change form: the preparation with a norm over the whole projection
(csrc/mixer_prep.cu), the delta rule's chunks with one or two stages (csrc/delta_rule.cu), the matrix memory's chunks with and without 16-byte loads
(csrc/mlstm.cu)."""
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


@pytest.mark.parametrize("new,H,G,Dk,Dv", [([130, 65, 1, 64], 40, 20, 64, 64), ([200, 30], 10, 10, 128, 128), ([70, 129], 12, 6, 128, 100), ([300], 2, 1, 80, 48), ([64, 3, 90], 30, 15, 80, 32),
                                           ([100, 140], 13, 13, 96, 96)])
def test_delta_rule_in_chunks(new, H, G, Dk, Dv):
    """Blocks of one stage side by side (more blocks than SMs, keys of 96 and 128), two blocks of two stages an SM (64 and 80), and one wave: against the
    recurrence in 64 bits."""
    g = torch.Generator().manual_seed(Dk + H)
    T, B, C = sum(new), len(new), 2 * G * Dk + H * Dv
    rows = torch.randn(T, C, generator=g)
    for a in (0, G * Dk):
        rows[:, a:a + G * Dk] = torch.nn.functional.normalize(rows[:, a:a + G * Dk].reshape(T, G, Dk), dim=-1).reshape(T, G * Dk)
    gates = torch.cat([torch.rand(T, H, generator=g), -torch.rand(T, H, generator=g) * 0.2], 1)
    start = torch.randn(B, H, Dk, Dv, generator=g) * 0.3
    state = start.reshape(B, -1).clone().to(DEV)
    chunks = sum(-(-n // 64) for n in new)
    scratch = torch.full((_lib().vm_delta_scratch_floats(_i(chunks), _i(H), _i(Dk), _i(Dv)),), float("nan"), device=DEV)
    o = torch.full((T, H * Dv), float("nan"), device=DEV)
    d_rows, d_gates, cu, slots = rows.to(DEV), gates.contiguous().to(DEV), _cu(new), _ints(list(range(B)))
    assert _lib().vm_delta_chunks(_p(d_rows), _p(d_gates), _p(state), _l(H * Dk * Dv), _i(0), _p(cu), _p(slots), _p(o), _p(scratch), _i(chunks), _i(T), _i(B), _i(H),
                                  _i(G), _i(Dk), _i(Dv), _stream()) == 0
    z = d_rows.double()
    q, k = (z[:, a:a + G * Dk].reshape(T, G, Dk).repeat_interleave(H // G, 1) for a in (0, G * Dk))
    v, beta, keep = z[:, 2 * G * Dk:].reshape(T, H, Dv), d_gates[:, :H].double(), torch.exp(d_gates[:, H:].double())
    S, t = start.to(DEV).double(), 0
    for b, n in enumerate(new):
        for t in range(t, t + n):
            s = S[b] * keep[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", s, k[t]))
            S[b] = s + k[t][:, :, None] * u[:, None]
            want = torch.einsum("hkv,hk->hv", S[b], q[t])
            if t % 37 == 0 or t + 1 == sum(new[:b + 1]):
                assert float((o[t].reshape(H, Dv).double() - want).abs().max()) <= 2e-5, t
        t += 1
    assert float((state.reshape(S.shape).double() - S).abs().max()) <= 2e-5


@pytest.mark.parametrize("new,H,D,V", [([64, 1, 63, 100], 4, 128, 256), ([129], 2, 64, 128), ([130, 7], 2, 32, 64), ([200], 3, 20, 36), ([65, 65], 1, 48, 40), ([127], 8, 24, 100)])
def test_matrix_memory_in_chunks_however_its_rows_lie(new, H, D, V):
    """With 16-byte loads where the rows allow them and without (the same rows one value further on): the same bits; and what the memory read and
    written token by token gives, up to sums in another order."""
    g = torch.Generator().manual_seed(D + V)
    T, B = sum(new), len(new)
    ld = 2 * H * D + 2 * H * V + 2 * H
    ld += -ld % 4
    proj = torch.randn(T, ld, generator=g)
    bi, bf = torch.randn(H, generator=g).to(DEV), (torch.randn(H, generator=g) + 3).to(DEV)
    nw = torch.rand(H * V, generator=g).to(DEV) + 0.5
    words = H * (D * V + D + 1)
    slots, cu = _ints(list(range(B))), _cu(new)
    got = []
    for kind in ("aligned", "one on", "token by token"):
        pool = torch.full((T * ld + 4,), float("nan"), device=DEV)
        rows = pool[1:1 + T * ld] if kind == "one on" else pool[:T * ld]
        rows.copy_(proj.reshape(-1))
        state = torch.zeros(B, words, device=DEV)
        out = torch.full((T, H * V), float("nan"), device=DEV)
        head = (_p(rows), _i(ld), _p(bi), _p(bf), _p(nw), _p(state), _p(cu), _p(slots), _p(out))
        sizes = (_i(B), _i(H), _i(D), _i(V), _f(15.0), _f(1e-6), _i(0), _stream())
        if kind == "token by token":
            if not _lib().vm_mlstm_scan_fits(_i(D), _i(V)):
                continue
            assert _lib().vm_mlstm_scan(*head, *sizes) == 0
        else:
            scratch = torch.full((_lib().vm_mlstm_chunk_scratch_floats(_i(T), _i(B), _i(H), _i(D), _i(V)),), float("nan"), device=DEV)
            assert _lib().vm_mlstm_chunks(*head, _p(scratch), _i(T), *sizes) == 0
        got.append((out, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    # (sums of up to 228 tokens and 128 channels in another order, 2^-24 each of their largest term, through a norm over the head: a few hundred of them)
    for out, _ in got[2:]:
        assert float((out - got[0][0]).abs().max()) <= 5e-5 * float(out.abs().max())
