"""Float32 attention of prompts (csrc/attention_tiles_f32.cu): the bits of the kernel that shares a query's keys over a CTA (csrc/attention_rows.cu)."""
import ctypes

import pytest
import torch

from test_attention_options_gpu import DEV, OPTIONS, Step, _i, _lib, _p, _stream

pytestmark = pytest.mark.gpu


# ragged prompts beside continued ones and single tokens: chunks of more than one round of the eight classes, tiles that cross sequences, chunk and page edges
@pytest.mark.parametrize("H,Hkv,Dk,Dv,in_keys", [(6, 2, 64, 64, False), (4, 4, 20, 8, False), (3, 1, 96, 128, False), (16, 1, 160, 128, True), (3, 3, 64, 32, True)])
@pytest.mark.parametrize("before,new", [([0, 130, 63, 0, 255], [300, 5, 2, 1, 33]), ([0] * 7, [8, 16, 31, 32, 33, 64, 65])])
@pytest.mark.parametrize("options", OPTIONS)
def test_same_bits_as_the_rows_kernel(H, Hkv, Dk, Dv, in_keys, before, new, options):
    s = Step(H, Hkv, Dk, Dv, before, new, torch.float32, in_keys)
    scale = Dk ** -0.5
    want = s.run("rows", *options, scale)                            # (sequences not counted: that kernel)
    window, keep, chunk, rel, sink, slopes = options
    dev = [t.to(DEV) for t in (s.q, s.table, s.positions, s.seq, s.rel, s.bucket, s.sink, s.slopes)]
    q, table, pos, seq, r, b, sk, sl = dev
    for rows in (2, 4, 0) if Dv > 64 else (2, 4, 8, 0):              # (what eight wide rows keep does not fit)
        out, err = torch.full((s.T, H, Dv), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        rc = _lib().vm_attention_tiles_f32(_p(q), _i(s.stride), _p(s.kp), _p(s.vp), _p(table), _i(table.shape[1]), _p(pos), _p(seq), _p(r if rel else None),
                                           _p(b if rel else None), _i(s.far if rel else 0), _p(sk if sink else None), _p(sl if slopes else None), _i(Dk if in_keys else Dv), _p(out), _i(s.T),
                                           _i(H), _i(Hkv), _i(Dk), _i(Dv), ctypes.c_float(scale), _i(window), _i(keep), _i(chunk), _i(s.kp.shape[0]), _p(err), _i(rows),
                                           _stream())
        assert rc == 0 and int(err.item()) == 0
        assert torch.equal(out.cpu(), want), rows


def test_a_page_that_is_missing_is_reported():
    s = Step(16, 16, 64, 64, [0], [200], torch.float32)          # (with the sequences counted: that kernel)
    s.table = s.table.clone()
    s.table[0, 1] = -1
    for n_seqs in (0, 1):
        assert s.call("rows", 0, 0, 0, False, False, False, 0.125, n_seqs=n_seqs)[1:] == (0, 3)


@pytest.mark.parametrize("H,Hkv,Dk,Dv,in_keys", [(16, 1, 160, 128, True), (9, 3, 64, 64, False)])
@pytest.mark.parametrize("options", OPTIONS)
def test_prompts_that_are_counted_take_it_with_the_same_bits(H, Hkv, Dk, Dv, in_keys, options):
    """Through the launcher that chooses: prompts of eight tokens a sequence and more, 2,000 rows and more, go to it once the sequences are counted."""
    s = Step(H, Hkv, Dk, Dv, [0, 0], [200, 130], torch.float32, in_keys)
    scale = Dk ** -0.5
    assert s.T * H >= 2000 and 16 * s.table.shape[1] * 2 <= s.T
    counted = s.run("rows", *options, scale, n_seqs=2)
    assert torch.equal(counted, s.run("rows", *options, scale))
    some = torch.tensor([0, 31, 32, 150, 199, 200, 263, 264, 329])
    assert float((counted[some].double() - s.want_some(some, slice(0, H), *options, scale)).abs().max()) <= 1e-5
