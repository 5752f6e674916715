"""Launchers called one behind the other on a stream, with nothing between the tokens of a sequence: programmatic launch changes no result."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one page; a table that is fetched ahead; several CTAs a sequence
@pytest.mark.parametrize("width,at,splits", [(1, 40, 1), (24, 1500, 1), (24, 1400, 4)])
@pytest.mark.parametrize("M", [1, 5])
def test_two_tokens_in_one_chain(M, width, at, splits, H=9, Hkv=3, D=64, K=576):
    """q/k/v and cache write of token t, its attention, the same of token t + 1: the last attention reads the row that the first kernel writes, while all four
    may be resident behind a long product.  The rows hold large values until they are written, so a row fetched too early shows in every output."""
    from velomind_b200.kernels import ops
    from velomind_b200.kernels.library import library
    g = torch.Generator(device=DEV).manual_seed(width + M)
    w = (torch.randn((H + 2 * Hkv) * D, K, generator=g, device=DEV) * 0.05).bfloat16()
    x = [torch.randn(M, K, generator=g, device=DEV).bfloat16() for _ in range(2)]
    cache = [torch.randn(M * width, Hkv, 64, D, generator=g, device=DEV).bfloat16() for _ in range(2)]
    table = torch.arange(M * width, dtype=torch.int32, device=DEV).view(M, width)
    positions = [torch.full((M,), at + i, dtype=torch.int32, device=DEV) for i in range(2)]
    for i in range(2):
        for c in cache:
            c.view(M, width, Hkv, 64, D)[:, (at + i) // 64, :, (at + i) % 64] = 300.0
    seq = torch.arange(M, dtype=torch.int32, device=DEV)
    freq = (10000.0 ** (-torch.arange(D // 2, device=DEV) / (D // 2))).float()
    partial = torch.empty(M * H * 16 * (D + 2), device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    counters = ops.decode_counters(DEV)
    long = torch.randn(4096, 4096, generator=g, device=DEV).bfloat16()
    product = torch.empty_like(long)

    def chain(kp, vp, q, out):
        torch.mm(long, long, out=product)
        for i in range(2):
            ops.skinny_qkv_rope(x[i], None, w, q[i], positions[i], seq, table, freq, D, kp, vp, H, Hkv, D, err=err)
            ops.attention_decode_bf16(q[i], H * D, kp, vp, table, positions[i], out[i], partial, counters, H, Hkv, D, splits, 1 / math.sqrt(D), err=err)

    def run(programmatic):
        kp, vp = (c.clone() for c in cache)
        q, out = ([torch.full((M, H * D), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2)] for _ in range(2))
        library().vm_set_pdl(1 if programmatic else 0)
        try:
            chain(kp.clone(), vp.clone(), q, out)                    # (what a first launch sets up is not part of a recording)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                chain(kp, vp, q, out)
            graph.replay()
            torch.cuda.synchronize()
        finally:
            library().vm_set_pdl(1)
        return out + [kp, vp]

    want = run(False)
    for _ in range(3):
        for a, b in zip(run(True), want):
            assert torch.equal(a, b)
    assert int(err.item()) == 0
