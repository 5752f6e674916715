"""The kernels of a decode step's few rows against the same in 64 bits: float32 products (csrc/skinny_f32.cu), the routers (csrc/expert_router.cu)
and the experts on tensor-core tiles (csrc/routed_experts_tile.cu)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _lib():
    from velomind_b200.kernels.library import library
    return library()


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _i(v):
    return ctypes.c_int(int(v))


def _f(v):
    return ctypes.c_float(v)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 4), (5, 36), (7, 576), (960, 576), (33, 1028), (64, 4096)])
def test_skinny_f32(T, N, K):
    """A row of a product does not depend on the others; error: K terms of 2^-24 of values of rms 1."""
    g = torch.Generator().manual_seed(T * K)
    x, w = torch.randn(T, K + 8, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    out = torch.full((T, N), float("nan"), device=DEV)
    assert _lib().vm_skinny_f32(_p(x), ctypes.c_longlong(K + 8), _p(w), _p(out), _i(T), _i(N), _i(K), _stream()) == 0
    want = x[:, :K].double() @ w.double().T
    assert float((out.double() - want).abs().max()) <= 1e-6 * K ** 0.5 * 4
    one = torch.empty(1, N, device=DEV)
    assert _lib().vm_skinny_f32(_p(x[T - 1:]), ctypes.c_longlong(K + 8), _p(w), _p(one), _i(1), _i(N), _i(K), _stream()) == 0
    assert float((one - out[T - 1:]).abs().max()) == 0.0


@pytest.mark.parametrize("T", [1, 2, 3, 8])
@pytest.mark.parametrize("N,K", [(6, 36), (1152, 576), (130, 1028)])
def test_skinny_f32_with_its_neighbours(T, N, K):
    """The norm in front, the sum into a residual stream and the gated unit behind."""
    g = torch.Generator().manual_seed(T + K)
    x, w, nw, h = (torch.randn(*s, generator=g).to(DEV) for s in ((T, K), (N, K), (K,), (T, N)))
    xn = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5) * nw.double()
    for norm in (True, False):
        y = (xn if norm else x.double()) @ w.double().T
        args = (_p(x), ctypes.c_longlong(K), _p(nw if norm else None), _f(1e-5), _p(w))
        tol = 1e-6 * K ** 0.5 * 8
        for add in (0, 1):
            out = h.clone()
            assert _lib().vm_skinny_f32_fused(*args, _p(out), _i(T), _i(N), _i(K), _i(add), _i(0), _stream()) == 0
            assert float((out.double() - (y + h.double() if add else y)).abs().max()) <= tol
        out = torch.full((T, N // 2), float("nan"), device=DEV)
        assert _lib().vm_skinny_f32_fused(*args, _p(out), _i(T), _i(N), _i(K), _i(0), _i(1), _stream()) == 0
        gate, up = y.chunk(2, -1)
        want = torch.nn.functional.silu(gate) * up
        assert float((out.double() - want).abs().max()) <= tol * float(y.abs().max())


def _choice(z, kind, top, groups, keep, gtop, correction, normalize, scale):
    if kind == "chosen":
        v, i = z.topk(top, -1)
        return i, torch.softmax(v, -1)
    s = torch.softmax(z, -1) if kind == "softmax" else torch.sigmoid(z)
    c = s if correction is None else s + correction
    if groups > 1:
        by = c.reshape(len(z), groups, -1)
        best = by.topk(gtop, -1).values.sum(-1).topk(keep, -1).indices
        mask = torch.zeros(len(z), groups, dtype=torch.bool, device=z.device).scatter_(1, best, True)
        c = by.masked_fill(~mask[..., None], -1e9).reshape(c.shape)
    i = c.topk(top, -1).indices
    w = s.gather(1, i)
    return i, w / (w.sum(-1, keepdim=True) + 1e-20) * scale if normalize else w * scale


def _check_choice(x, w, z, chosen, kind, groups, gtop, correction):
    """Every output was the best one left to choose, up to the error of 32-bit sums: hidden / 16 + 16 additions in a row, however the kernels cut
    them, of 2^-23 (the tensor cores cut off, 2^-24 where they round) of the sum of the products' magnitudes."""
    n = chosen.long()
    assert bool((n.sort(-1).values.diff(dim=-1) > 0).all())
    e = (w.shape[1] / 16 + 16) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T).max(-1, keepdim=True).values
    s = z if kind == "chosen" else torch.softmax(z, -1) if kind == "softmax" else torch.sigmoid(z)
    with_corr = s if correction is None else s + correction.double()
    c = z if kind == "sigmoid" and correction is None else with_corr
    e = e if c is z else 2.1 * e + 2.0 ** -22                           # a softmax moves by at most twice its logits
    left = torch.ones_like(c, dtype=torch.bool)
    if groups > 1:
        per = c.shape[1] // groups
        mine = n // per
        assert bool((mine == mine[:, :1]).all())
        score = with_corr.reshape(len(c), groups, per).topk(gtop, -1).values.sum(-1)
        assert bool((score.gather(1, mine[:, :1]) >= score.max(-1, keepdim=True).values - 2 * gtop * e).all())
        left = torch.arange(c.shape[1], device=c.device) // per == mine[:, :1]
    for k in range(n.shape[1]):
        best = c.masked_fill(~left, -1e30).max(-1, keepdim=True).values
        assert bool((c.gather(1, n[:, k:k + 1]) >= best - 2 * e).all()), k
        left = left & ~torch.zeros_like(left).scatter_(1, n[:, k:k + 1], True)


@pytest.mark.parametrize("T", [1, 8, 149, 163, 700, 905, 1201])
@pytest.mark.parametrize("hidden,n_out,top,kind", [(1024, 16, 4, "chosen"), (96, 18, 4, "softmax"), (2048, 32, 4, "sigmoid"), (64, 5, 2, "chosen"), (160, 64, 6, "sigmoid"), (72, 9, 3, "softmax")])
def test_routers(T, hidden, n_out, top, kind):
    """One block per token and tiles of sixteen tokens, with a gate row behind the outputs (`chosen`) and with groups: the choice, where no two
    outputs come closer than the sums' error, and the weights (float32 sums of `hidden` terms)."""
    g = torch.Generator().manual_seed(T + hidden)
    x = torch.randn(T, hidden, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(n_out, hidden, generator=g) * 2.0 / hidden ** 0.5).to(DEV)
    chosen, weight = torch.full((T, top), -1, dtype=torch.int32, device=DEV), torch.full((T, top), float("nan"), device=DEV)
    z = x.double() @ w.double().T
    if kind == "chosen":
        b, gate = torch.randn(n_out, generator=g).to(DEV), torch.randn(hidden, generator=g).to(DEV) / hidden ** 0.5
        sg = torch.full((T,), float("nan"), device=DEV)
        assert _lib().vm_expert_router(_p(x), None, _f(0), _p(w), _p(b), _p(gate), _i(T), _i(hidden), _i(n_out), _i(top), _p(chosen), _p(weight), _p(sg), _i(1), _stream()) == 0
        want = _choice(z + b.double(), kind, top, 1, 1, 1, None, False, 1.0)
        assert float((sg.double() - torch.sigmoid(x.double() @ gate.double())).abs().max()) <= 1e-6
    else:
        groups = 2 if n_out % 2 == 0 and n_out // 2 >= top else 1
        corr = (torch.randn(n_out, generator=g) * 0.01).to(DEV) if kind == "softmax" else None
        gtop = 2 if kind == "sigmoid" and groups > 1 else 1
        assert _lib().vm_expert_router_groups(_p(x), None, _f(0), _p(w), _p(corr), _i(T), _i(hidden), _i(n_out), _i(top), _i(groups), _i(1), _i(gtop), _f(1.5),
                                              _i(0 if kind == "softmax" else 1), _i(1 if kind == "sigmoid" else 0), _p(chosen), _p(weight), _i(1), _stream()) == 0
        want = _choice(z, kind, top, groups, 1, gtop, None if corr is None else corr.double(), kind == "sigmoid", 1.5)
    same = (chosen.long() == want[0]).all(-1)
    assert float(same.float().mean()) >= 0.99                       # (near ties may fall either way)
    assert float((weight.double() - want[1])[same].abs().max()) <= 4e-6
    if kind == "chosen":
        _check_choice(x, w, z + b.double(), chosen, kind, 1, 1, None)
    else:
        _check_choice(x, w, z, chosen, kind, groups, gtop, corr)


@pytest.mark.parametrize("hidden,n_out", [(1024, 16), (2048, 64), (96, 40)])
def test_a_router_row_in_a_long_step_and_in_short_ones(hidden, n_out):
    """The same rows in one step (tiles of tokens) and a hundred at a time (a block per token) add their products up in another order: weights agree to 8e-6
    (4e-6 each against 64 bits), and a choice differs only where the scores are as close as the sums' error."""
    g = torch.Generator().manual_seed(hidden)
    T, top = 1500, 4
    x = torch.randn(T, hidden, generator=g).to(torch.bfloat16).to(DEV)
    w, b = (torch.randn(n_out, hidden, generator=g) * 2.0 / hidden ** 0.5).to(DEV), torch.randn(n_out, generator=g).to(DEV)
    out = []
    for piece in (T, 100):
        chosen, weight = torch.full((T, top), -1, dtype=torch.int32, device=DEV), torch.full((T, top), float("nan"), device=DEV)
        for a in range(0, T, piece):
            assert _lib().vm_expert_router(_p(x[a:]), None, _f(0), _p(w), _p(b), None, _i(min(piece, T - a)), _i(hidden), _i(n_out), _i(top), _p(chosen[a:]), _p(weight[a:]), None,
                                           _i(1), _stream()) == 0
        _check_choice(x, w, x.double() @ w.double().T + b.double(), chosen, "chosen", 1, 1, None)
        out.append((chosen, weight))
    same = (out[0][0] == out[1][0]).all(-1)
    assert float(same.float().mean()) >= 0.99
    assert float((out[0][1] - out[1][1])[same].abs().max()) <= 8e-6


@pytest.mark.parametrize("T", [1, 8, 17, 33, 70])
@pytest.mark.parametrize("hidden,ff,sff,top,E,ident,glu", [(64, 32, 0, 2, 6, 0, 0), (1024, 512, 1024, 4, 16, 0, 0), (128, 288, 0, 4, 16, 2, 1), (96, 64, 32, 3, 5, 0, 2), (2400, 96, 64, 4, 40, 0, 3)])
def test_experts_tile(T, hidden, ff, sff, top, E, ident, glu):
    """Few and many tokens of an expert, pieces of the contraction that end early, identity experts, every kind of gate; the unit and the result are
    rounded to bfloat16."""
    g = torch.Generator().manual_seed(T + ff)
    bf = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(torch.bfloat16).to(DEV)
    x, up, down = bf(T, hidden), bf(E, (2 if glu else 1) * ff, hidden, scale=hidden ** -0.5), bf(E, hidden, ff, scale=ff ** -0.5)
    s_gated = glu >= 2
    s_up = bf((2 if s_gated else 1) * sff, hidden, scale=hidden ** -0.5) if sff else None
    s_down = bf(hidden, sff, scale=sff ** -0.5) if sff else None
    chosen = torch.stack([torch.randperm(E + ident, generator=g)[:top] for _ in range(T)]).int().to(DEV)
    weight = torch.rand(T, top, generator=g).to(DEV)
    sg = torch.rand(T, generator=g).to(DEV) if glu == 0 and sff else None
    limit, alpha = 1.0, 1.702
    r = lambda t: t.to(torch.bfloat16).double()

    def unit(z, w, gated, kind):
        if not gated:
            return r(torch.relu(z) ** 2)
        a, b = z.chunk(2, -1)
        if kind == 1:
            a, b = r(a).clamp(max=limit), r(b).clamp(-limit, limit)
            return r(a * torch.sigmoid(alpha * a) * (b + 1))
        a, b = w * r(a), w * r(b)
        return r(a * torch.sigmoid(a) * b)

    want = torch.zeros(T, hidden, dtype=torch.float64, device=DEV)
    for t in range(T):
        for k in range(top):
            e, w = int(chosen[t, k]), weight[t, k].double()
            if e >= E:
                want[t] += w * x[t].double()
                continue
            a = unit(up[e].double() @ x[t].double(), w if glu == 2 else 1.0, bool(glu), glu)
            want[t] += (1.0 if glu == 2 else w) * (down[e].double() @ a)
        if sff:
            a = unit(s_up.double() @ x[t].double(), 1.0, s_gated, glu)
            want[t] += (sg[t].double() if sg is not None else 1.0) * (s_down.double() @ a)
    cols = top * ff + sff + (hidden if ident else 0)
    act = torch.full((T, cols), float("nan"), dtype=torch.bfloat16, device=DEV)
    out = torch.full((T, hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
    h = torch.randn(T, hidden, generator=g).to(DEV)
    assert _lib().vm_experts_few_tile_fits(_i(T), _i(hidden), _i(ff), _i(sff), _i(top), _i(E), _i(ident)) == 1
    for residual in (None, h.clone()):
        rc = _lib().vm_experts_few_tile(_p(x), _p(up), _p(down), _p(s_up), _p(s_down), _p(chosen), _p(weight), _p(sg), _i(T), _i(hidden), _i(ff), _i(sff), _i(top), _i(2), _i(2),
                                        _i(E), _i(ident), _i(glu), _f(limit), _f(alpha), _p(act), _p(out), _p(residual), _stream())
        assert rc == 0
        got = out.double() if residual is None else (residual - h).double()
        # one rounding of the result (2^-9 of it), and now and then a unit that falls to the other side of a rounding
        assert float((got - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-2 * float(want.std())


@pytest.mark.parametrize("T,top", [(895, 8), (896, 8), (1024, 8), (2048, 4), (512, 16)])
def test_experts_tile_of_large_decode_batches(T, top):
    """As many (token, expert) pairs as the list of a block holds, around the sizes from which it needs more shared memory than a launch gets
    unasked; one more token is refused."""
    g = torch.Generator().manual_seed(T)
    hidden, ff, E = 64, 32, 18
    bf = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(torch.bfloat16).to(DEV)
    x, up, down = bf(T, hidden), bf(E, ff, hidden, scale=hidden ** -0.5), bf(E, hidden, ff, scale=ff ** -0.5)
    chosen = torch.rand(T, E, generator=g).topk(top, -1).indices.int().to(DEV)
    weight = torch.rand(T, top, generator=g).to(DEV)
    z = torch.einsum("efh,th->tef", up.double(), x.double())
    a = (torch.relu(z) ** 2).to(torch.bfloat16).double()
    y = torch.einsum("ehf,tef->teh", down.double(), a)
    want = (y.gather(1, chosen.long()[..., None].expand(-1, -1, hidden)) * weight.double()[..., None]).sum(1)
    act = torch.full((T, top * ff), float("nan"), dtype=torch.bfloat16, device=DEV)
    out = torch.full((T, hidden), float("nan"), dtype=torch.bfloat16, device=DEV)

    def run(T):
        sizes = _i(T), _i(hidden), _i(ff), _i(0), _i(top)
        fits = _lib().vm_experts_few_tile_fits(*sizes, _i(E), _i(0))
        return fits, _lib().vm_experts_few_tile(_p(x), _p(up), _p(down), None, None, _p(chosen), _p(weight), None, *sizes, _i(2), _i(2), _i(E), _i(0), _i(0), _f(0),
                                                _f(0), _p(act), _p(out), None, _stream())
    assert run(T) == (1, 0)
    # one rounding of the result (2^-9 of it), and now and then a unit that falls to the other side of a rounding
    assert float((out.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-2 * float(want.std())
    fits, rc = run(8192 // top + 1)                                # (refused before anything is launched)
    assert fits == 0 and rc != 0


@pytest.mark.parametrize("sizes", [[(1, 0)], [(3, 1), (40000, 0), (5, 3)], [(7, 0)] * 33])
def test_clear_areas(sizes):
    """State areas of any size and start become zeros, and nothing beside them does."""
    pool = torch.ones(sum(n + off + 8 for n, off in sizes), device=DEV)
    at, left = [], torch.ones_like(pool)
    start = 0
    for n, off in sizes:
        at.append((start + off, n))
        left[start + off:start + off + n] = 0
        start += n + off + 8
    for k in range(0, len(at), 32):
        part = at[k:k + 32]
        where = (ctypes.c_void_p * len(part))(*[pool.data_ptr() + 4 * a for a, _ in part])
        n = (ctypes.c_longlong * len(part))(*[n for _, n in part])
        assert _lib().vm_clear_areas(where, n, _i(len(part)), _stream()) == 0
    assert torch.equal(pool, left)
    assert _lib().vm_clear_areas(None, None, _i(33), _stream()) != 0
