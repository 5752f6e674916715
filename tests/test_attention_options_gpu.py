"""The attention kernels that share a query's keys out (csrc/attention_rows.cu in float32, csrc/attention_decode_tile.cu for decode steps in
bfloat16) against the same attention in 64 bits, with every option: bias by bucketed distance, slopes, sink, window, kept first tokens, chunked
mask, values inside the key rows.  Rows that no query sees hold NaN."""
import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PAGE = 64


def _lib():
    from velomind_b200.kernels.library import library
    return library()


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _i(v):
    return ctypes.c_int(int(v))


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


class Step:
    """Sequences of `before` cached and `new` tokens, paged in a shuffled order, and the options' tables."""

    def __init__(self, H, Hkv, Dk, Dv, before, new, dtype, in_keys=False, far=40, seed=0):
        g = torch.Generator().manual_seed(seed)
        self.H, self.Hkv, self.Dk, self.Dv, self.before, self.new, self.dtype, self.in_keys = H, Hkv, Dk, Dv, before, new, dtype, in_keys
        lens = [a + n for a, n in zip(before, new)]
        width = max(-(-n // PAGE) for n in lens) + 1
        pages = sum(-(-n // PAGE) for n in lens) + 2
        order = torch.randperm(pages, generator=g).tolist()
        kp = torch.full((pages, Hkv, PAGE, Dk), float("nan"))
        vp = torch.full((pages, Hkv, PAGE, Dv), float("nan"))
        self.table = torch.full((len(lens), width), -1, dtype=torch.int32)
        self.k, self.v = [], []
        for s, n in enumerate(lens):
            k = torch.randn(n, Hkv, Dk, generator=g).to(dtype)
            v = k[..., :Dv] if in_keys else torch.randn(n, Hkv, Dv, generator=g).to(dtype)
            self.k.append(k.double()); self.v.append(v.double())
            for b in range(-(-n // PAGE)):
                pg = order.pop()
                self.table[s, b] = pg
                m = min(PAGE, n - PAGE * b)
                kp[pg, :, :m] = k[PAGE * b:PAGE * b + m].transpose(0, 1).float()
                vp[pg, :, :m] = v[PAGE * b:PAGE * b + m].transpose(0, 1).float()
        self.kp = kp.to(dtype).to(DEV)
        self.vp = self.kp if in_keys else vp.to(dtype).to(DEV)
        self.T = sum(new)
        self.stride = H * Dk + 16
        self.q = (torch.randn(self.T, self.stride, generator=g) * 1.5).to(dtype)
        self.positions = torch.cat([torch.arange(a, a + n) for a, n in zip(before, new)]).int()
        self.seq = torch.cat([torch.full((n,), s) for s, n in enumerate(new)]).int()
        self.far = far
        self.rel = torch.randn(7, H, generator=g)
        self.bucket = (torch.arange(far + 1) % 7).int()
        self.sink = torch.randn(H, generator=g)
        self.slopes = torch.rand(H, generator=g) * 0.1

    def want(self, window, keep, chunk, rel, sink, slopes, scale):
        out = torch.empty(self.T, self.H, self.Dv, dtype=torch.float64)
        for t in range(self.T):
            s, i = int(self.seq[t]), int(self.positions[t])
            j = torch.arange(i + 1)
            see = torch.ones(i + 1, dtype=torch.bool)
            if window:
                see &= i - j < window
            if chunk:
                see &= j // chunk == i // chunk
            see |= j < keep
            for h in range(self.H):
                g = h // (self.H // self.Hkv)
                x = (self.k[s][:i + 1, g] @ self.q[t, h * self.Dk:(h + 1) * self.Dk].double()) * scale
                if rel:
                    x = x + self.rel[self.bucket[(i - j).clamp(max=self.far)].long(), h].double()
                if slopes:
                    x = x - self.slopes[h].double() * (i - j)
                x = x[see]
                top = max(float(x.max()), float(self.sink[h]) if sink else -math.inf)
                e = torch.exp(x - top)
                den = e.sum() + (math.exp(float(self.sink[h]) - top) if sink else 0.0)
                out[t, h] = (e / den) @ self.v[s][:i + 1, g][see]
        return out

    def want_some(self, tokens, heads, *options):
        """`want` for some tokens and heads."""
        few = Step.__new__(Step)
        few.__dict__.update(self.__dict__)
        few.T, few.positions, few.seq, few.q = len(tokens), self.positions[tokens], self.seq[tokens], self.q[tokens]
        n = len(range(*heads.indices(self.H)))
        few.H, few.Hkv = n, max(1, n // (self.H // self.Hkv)) if n < self.H else self.Hkv
        return few.want(*options)

    def call(self, name, window, keep, chunk, rel, sink, slopes, scale, tokens=None, n_seqs=0, width=None):
        """The kernel's outputs, its status and the error word; width: columns of the block table."""
        at = slice(0, self.T) if tokens is None else tokens
        n = len(range(*at.indices(self.T)))
        out = torch.full((n, self.H, self.Dv), float("nan"), dtype=self.dtype, device=DEV)
        err = torch.zeros(1, dtype=torch.int32, device=DEV)
        blocks = self.table if width is None else torch.nn.functional.pad(self.table, (0, max(0, width - self.table.shape[1])), value=-1)[:, :width].contiguous()
        dev = [t.to(DEV) for t in (self.q[at].contiguous(), blocks, self.positions[at].contiguous(), self.seq[at].contiguous(), self.rel, self.bucket, self.sink, self.slopes)]
        q, table, pos, seq, r, b, sk, sl = dev
        head = [_p(q), _i(self.stride), _p(self.kp), _p(self.vp), _p(table), _i(table.shape[1]), _p(pos)]
        opts = [_p(r if rel else None), _p(b if rel else None), _i(self.far if rel else 0), _p(sk if sink else None), _p(sl if slopes else None),
                _i(self.Dk if self.in_keys else 0), _p(out)]
        sizes = [_i(self.H), _i(self.Hkv), _i(self.Dk), _i(self.Dv), ctypes.c_float(scale), _i(window), _i(keep), _i(chunk), _i(self.kp.shape[0])]
        if name == "prompt":
            new = torch.bincount(self.seq.long(), minlength=len(self.new)).tolist()
            cu = torch.tensor([0] + list(np.cumsum(new)), dtype=torch.int32, device=DEV)
            rc = _lib().vm_attention_sink_prefill_bf16(*head, _p(cu), _i(len(new)), _i(sum(-(-m // 64) for m in new)), *opts[:3], _i(7 if rel else 0), *opts[3:], *sizes, _p(err), _stream())
        elif name == "rows":
            rc = _lib().vm_attention_sink_generic_seqs(*head, _p(seq), *opts, _i(n), *sizes, _i(0 if self.dtype == torch.float32 else 1), _p(err), _i(n_seqs), _stream())
        else:
            rc = _lib().vm_attention_sink_decode_bf16(*head, *opts, _i(n), *sizes, _p(err), _stream())
        return out.cpu(), rc, int(err.item())

    def run(self, *args, **more):
        out, rc, err = self.call(*args, **more)
        assert (rc, err) == (0, 0)
        return out


# window, kept first tokens, chunk, bias, sink, slopes
OPTIONS = [(0, 0, 0, False, False, False), (33, 0, 0, True, False, False), (64, 5, 0, True, True, False), (0, 0, 96, False, False, True), (40, 70, 0, False, True, True),
           (0, 3, 64, False, False, False)]


@pytest.mark.parametrize("H,Hkv,Dk,Dv,in_keys", [(3, 3, 64, 64, False), (9, 3, 64, 64, False), (16, 1, 160, 128, True), (10, 1, 20, 6, False), (4, 2, 128, 66, False), (17, 1, 4, 2, False)])
@pytest.mark.parametrize("options", OPTIONS)
def test_rows_float32(H, Hkv, Dk, Dv, in_keys, options):
    """Whole prompts across chunk and page edges, a continued sequence, single tokens; error: 64 or more terms of 2^-24 each."""
    s = Step(H, Hkv, Dk, Dv, [0, 130, 63, 0, 255], [100, 5, 2, 1, 1], torch.float32, in_keys)
    scale = Dk ** -0.5
    got, want = s.run("rows", *options, scale), s.want(*options, scale)
    assert float((got.double() - want).abs().max()) <= 1e-5


def test_rows_do_not_depend_on_the_batch_or_the_cut():
    """Few tokens (a CTA per token) and many (a CTA for several), in one step and in pieces: the same bits."""
    s = Step(6, 3, 64, 64, [0, 70, 0, 200], [150, 31, 64, 1], torch.float32)
    whole = s.run("rows", 50, 3, 0, False, True, False, 0.125)
    for a, b in ((0, 1), (149, 152), (140, 160), (245, 246)):
        assert torch.equal(whole[a:b], s.run("rows", 50, 3, 0, False, True, False, 0.125, slice(a, b)))


@pytest.mark.parametrize("H,Hkv,D", [(32, 32, 64), (9, 3, 64), (16, 1, 128), (12, 12, 20)])
@pytest.mark.parametrize("before,new,widths", [([0, 7, 31, 32, 50, 62, 63] * 6, [1] * 42, (1, 2, 3)), ([0, 33, 64, 100, 126, 127] * 6, [1] * 36, (2, 3)),
                                               ([70, 128, 300, 511, 90] * 8, [1] * 40, (8, 9)), ([0, 20, 3] * 12, [3, 40, 1] * 12, (1, 2, 3)), ([0, 1, 60], [30, 2, 4], (1, 4))])
def test_rows_of_many_sequences(H, Hkv, D, before, new, widths):
    """Decode batches and prompts side by side, in tables of one page, two and more: however tokens are dealt out to CTAs and keys to
    warps, the same bits; and the right ones."""
    s = Step(H, Hkv, D, D, before, new, torch.float32)
    options = (0, 0, 0, False, False, False, D ** -0.5)
    got = s.run("rows", *options, n_seqs=len(new), width=widths[0])
    for width in widths:
        for n_seqs in (0, len(new)):
            assert torch.equal(got, s.run("rows", *options, n_seqs=n_seqs, width=width)), (width, n_seqs)
    some = torch.arange(0, s.T, max(1, s.T // 40))
    heads = slice(0, H // Hkv) if Hkv > 1 else slice(0, H)             # (heads compared: the reference is slow)
    assert float((got[some][:, heads].double() - s.want_some(some, heads, *options)).abs().max()) <= 1e-5


@pytest.mark.parametrize("H,Hkv,Dk,Dv,in_keys", [(8, 8, 64, 64, False), (16, 4, 64, 64, False), (4, 2, 64, 128, False), (6, 2, 96, 64, False), (4, 4, 128, 64, False), (3, 1, 96, 128, False),
                                                 (16, 1, 128, 128, True), (20, 1, 160, 128, True), (33, 1, 192, 128, True)])
@pytest.mark.parametrize("options", OPTIONS)
def test_decode_tile(H, Hkv, Dk, Dv, in_keys, options):
    """Lengths around the 32-key turns, the pages and a cluster's first round; the result is rounded to bfloat16 once (half of 2^-8 of it), and
    sums of 32-bit terms leave 1e-5."""
    s = Step(H, Hkv, Dk, Dv, [0, 31, 32, 63, 64, 300, 1111], [1] * 7, torch.bfloat16, in_keys, far=700)
    scale = Dk ** -0.5
    got, want = s.run("tile", *options, scale), s.want(*options, scale)
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all())


def test_decode_tile_with_more_sequences_than_sms():
    """One CTA per sequence and head group, several turns of every warp."""
    s = Step(4, 4, 64, 64, [700 - 3 * i for i in range(70)], [1] * 70, torch.bfloat16)
    got, want = s.run("tile", 0, 0, 0, False, False, False, 0.125), s.want(0, 0, 0, False, False, False, 0.125)
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all())


def test_an_infinite_value_stays_infinite():
    s = Step(4, 1, 64, 64, [40], [1], torch.bfloat16)
    page, row = int(s.table[0, 0]), 7
    s.vp[page, 0, row, 3] = float("inf")
    got = s.run("tile", 0, 0, 0, False, False, False, 0.125)
    assert bool(torch.isposinf(got[0, :, 3]).all()) and bool(torch.isfinite(got[0, :, 4:]).all()) and bool(torch.isfinite(got[0, :, :3]).all())


@pytest.mark.parametrize("name", ["tile", "rows"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_biases_at_the_ends_of_the_type(name, dtype):
    """The lowest float as a mask: on the far keys (they get no weight), on every key (they all get the same, as in float32 arithmetic), and a sink of
    the lowest and the largest float."""
    if name == "tile" and dtype == torch.float32:
        pytest.skip("bfloat16 only")
    least = torch.finfo(torch.float32).min
    for rel, sink in ((torch.arange(7)[:, None].expand(7, 4) > 2, None), (torch.ones(7, 4, dtype=torch.bool), None), (None, least), (None, -least)):
        s = Step(4, 1, 64, 64, [0, 40, 300], [1] * 3, dtype)
        if rel is not None:
            s.rel = torch.where(rel, torch.full((7, 4), least), s.rel)
            s.bucket = (torch.arange(s.far + 1) * 7 // (s.far + 1)).int()
        if sink is not None:
            s.sink = torch.full((4,), sink)
        options = (0, 0, 0, rel is not None, sink is not None, False, 0.125)
        got, want = s.run(name, *options), s.want(*options)
        assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all())


@pytest.mark.parametrize("name,dtype,page", [("tile", torch.bfloat16, -1), ("rows", torch.bfloat16, -1), ("rows", torch.float32, 4096), ("prompt", torch.bfloat16, -1)])
def test_a_missing_page_is_reported(name, dtype, page):
    """A page that is not there, or outside the pool: the launch is accepted, and the error word says that a page was missing."""
    s = Step(4, 1, 64, 64, [200], [1], dtype)
    s.table[0, 1] = page
    assert s.call(name, 0, 0, 0, False, False, False, 0.125)[1:] == (0, 3)


@pytest.mark.parametrize("H,Hkv,Dk,Dv,in_keys", [(4, 2, 64, 64, False), (80, 20, 64, 64, False), (3, 1, 96, 64, True), (2, 1, 160, 128, True), (70, 1, 128, 128, True), (2, 2, 64, 128, False),
                                                 (4, 4, 32, 16, False)])
@pytest.mark.parametrize("options", OPTIONS + [(0, 0, 0, True, False, True)])
def test_prompt(H, Hkv, Dk, Dv, in_keys, options):
    """Prompts around the edges of the 64-row tiles and of the masks: blocks that every row of a warp sees whole and blocks that it does not.  Probabilities are rounded to
    bfloat16 (2^-9 each of values around 1) and so is the result."""
    s = Step(H, Hkv, Dk, Dv, [0, 130, 63, 0, 0], [130, 5, 70, 1, 129], torch.bfloat16, in_keys, far=300)
    scale = Dk ** -0.5
    keep = slice(0, 2) if H > 8 else slice(0, H)                       # (heads compared: the reference is slow)
    got = s.run("prompt", *options, scale)
    t = torch.tensor([0, 63, 64, 127, 128, 129, 130, 134, 135, 204, 205, 206, 270, 334])
    whole = s.want_some(t, keep, *options, scale)
    assert bool(((got[t][:, keep].double() - whole).abs() <= whole.abs() * 2.0 ** -8 + 6e-3 * float(whole.abs().max())).all())
