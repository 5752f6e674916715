"""Prompt attention with its tiles dealt out by their length (csrc/tile_order.cuh): the same bits as tile by tile along the prompts."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _i(v):
    return ctypes.c_int(int(v))


# one tile; fewer items than SMs; an odd last wave that is not full; sequences without new tokens between others; rows at the edges of a tile; more tiles than the
# list holds (the walk over the sequences)
@pytest.mark.parametrize("new,H,Hkv", [([1], 1, 1), ([300], 9, 3), ([2048], 9, 3), ([64, 0, 65, 63, 0, 700], 15, 5), ([130 + 54 * i for i in range(8)], 16, 4), ([5] * 257, 2, 1),
                                       ([64] * 256, 1, 1), ([64 * 256], 1, 1), ([64 * 256 + 1], 1, 1)])
def test_same_bits_as_along_the_prompts(new, H, Hkv, D=64):
    from velomind_b200.kernels.library import library
    lib = library()
    g = torch.Generator(device=DEV).manual_seed(sum(new))
    T, B, width = sum(new), len(new), max(1, max(-(-n // 64) for n in new))
    q = torch.randn(T, H * D, generator=g, device=DEV).bfloat16()
    k, v = (torch.randn(B * width, Hkv, 64, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    table = torch.randperm(B * width, generator=torch.Generator().manual_seed(1)).int().view(B, width).to(DEV)
    positions = torch.cat([torch.arange(n) for n in new]).int().to(DEV)
    offsets = torch.tensor([0] + new).cumsum(0).int()
    on_device, err = offsets.to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    tiles, stream = sum(-(-n // 64) for n in new), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    head = [_p(q), _i(H * D), _p(k), _p(v), _p(table), _i(width), _p(positions), _p(on_device)]
    want = torch.empty(2, T, H * D)
    for host in (None, offsets):
        plain, biased = (torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
        assert lib.vm_attention_prefill_seqs_bf16(*head, _p(host), _i(B), _i(tiles), _p(plain), _i(H), _i(Hkv), _i(D), ctypes.c_float(0.125), _i(0), _i(B * width), _p(err),
                                                  _i(1), stream) == 0
        assert lib.vm_attention_sink_prefill_seqs_bf16(*head, _p(host), _i(B), _i(tiles), _p(None), _p(None), _i(0), _i(0), _p(None), _p(None), _i(0), _p(biased), _i(H), _i(Hkv),
                                                       _i(D), _i(D), ctypes.c_float(0.125), _i(100), _i(3), _i(0), _i(B * width), _p(err), stream) == 0
        got = torch.stack([plain, biased]).float().cpu()
        assert int(err.item()) == 0 and not bool(torch.isnan(got).any())
        if host is None:
            want = got
        assert torch.equal(got, want)
