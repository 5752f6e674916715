"""Decode attention over wide block tables (csrc/attn_decode_body.cuh): ten warps with a further page fetched under the work on the page at hand, and the same
sequences shared out over several CTAs, against 64 bits."""
import math

import pytest
import torch

from test_attention_options_gpu import DEV, Step

pytestmark = pytest.mark.gpu

# pages: the first width that is fetched ahead and the next one, a table of several turns; lengths at the edges of pages and of a turn of ten pages, sequences
# of one page and of none but the new token beside them
TABLES = [[1343, 1280, 1279, 640, 639, 63, 0], [1344, 1407, 704, 1], [2715, 2560, 2559, 1919, 1300, 90]]


def _decode(s, splits, window, in_step=False):
    from velomind_b200.kernels import ops
    B, H, D = len(s.new), s.H, s.Dk
    out = torch.full((B, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    partial, counters = torch.full((B * H * splits * (D + 2),), float("nan"), device=DEV), torch.zeros(B * H, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    # (Step's last column names no page: it goes, so that the width is the longest sequence's)
    q, table, positions = s.q.to(DEV), s.table[:, :-1].contiguous().to(DEV), s.positions.to(DEV)
    ops.attention_decode_bf16(q, s.stride, s.kp, s.vp, table, positions, out, partial, counters, H, s.Hkv, D, splits, 1 / math.sqrt(D), window, err, in_step=in_step)
    torch.cuda.synchronize()
    assert int(counters.abs().sum()) == 0
    return out.view(B, H, D).cpu(), int(err.item())


def _step(H, Hkv, D, before):
    s = Step(H, Hkv, D, D, before, [1] * len(before), torch.bfloat16)
    s.kp, s.vp = s.kp.nan_to_num(3.0), s.vp.nan_to_num(3.0)              # (pages hold finite values from the start)
    return s


@pytest.mark.parametrize("H,Hkv,D", [(9, 3, 64), (20, 1, 48), (3, 3, 16)])
@pytest.mark.parametrize("before", TABLES)
@pytest.mark.parametrize("window", [0, 70, 700])
def test_wide_tables(H, Hkv, D, before, window):
    """Products of bfloat16 are exact and summed in 32 bits; a probability is rounded to bfloat16 (2^-9 of it) before it meets its value, the result once more."""
    s = _step(H, Hkv, D, before)
    want = s.want(window, 0, 0, False, False, False, 1 / math.sqrt(D))
    bound = 2.0 ** -9 * (max(float(v.abs().max()) for v in s.v) + want.abs()) + 1e-4
    for splits, in_step in ((1, False), (1, True), (4, False), (16, True)):
        got, err = _decode(s, splits, window, in_step)
        assert err == 0 and bool(((got.double() - want).abs() <= bound).all()), (splits, in_step)


@pytest.mark.parametrize("page", [0, 7, 15, 30, 42])
def test_a_missing_page_is_reported(page):
    """A page of the first turn, of a further one, the last one: the error word; the other sequence's result does not change."""
    s = _step(9, 3, 64, [2715, 1300])
    whole, err = _decode(s, 1, 0)
    assert err == 0
    s.table = s.table.clone()
    s.table[0, page] = -1
    got, err = _decode(s, 1, 0)
    assert err == 3 and torch.equal(got[1], whole[1])
