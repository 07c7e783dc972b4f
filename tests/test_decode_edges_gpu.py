"""Lengths at the edges of what the head_dim 64 decode kernel cuts requests into (32-token chunks,
sixteen of them in flight per CTA, 256-token planner tiles), and values at the rounding boundaries
of the writer's division-free quantizer."""
import numpy as np
import pytest
import torch

from helpers import assert_pools_equal, cpu_twin, paged_batch
from test_decode_gpu import _run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [2, 4])
@pytest.mark.parametrize("hq,hkv", [(64, 8), (8, 8), (24, 8), (32, 2)])
@pytest.mark.parametrize("scale_dtype", [None, torch.bfloat16])
def test_head_dim_64_chunk_edges(bits, hq, hkv, scale_dtype):
    """GQA 8, 1, 3 and 16 (two head tiles): one token, around one chunk, around a page, around a
    lap of the CTA's warps, and uniform splits whose last piece is short."""
    _run_case(bits, 64, hq, hkv, [1, 31, 32, 33, 63, 65, 511, 513, 1025], seed=71,
              scale_dtype=scale_dtype)
    _run_case(bits, 64, hq, hkv, [257, 3000], seed=72, kv_splits=3, host_lens=False,
              scale_dtype=scale_dtype)


@pytest.mark.parametrize("bits", [2, 4])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_codes_at_rounding_boundaries(bits, d):
    """Rows whose scale is exactly one and whose values lie on half integers or one bf16 step beside
    them (both sides of every rounding boundary, where the quantizer has to divide), next to rows
    that stay clear of them: the bytes are the oracle's."""
    from foscar_b200 import QuantKVLayout
    hkv, seq, top = 2, [64, 128], (1 << bits) - 1
    _, _, slots, npages = paged_batch(seq, seed=73)
    gen = torch.Generator().manual_seed(73)
    half = (torch.randint(0, top, (len(slots), hkv, d), generator=gen) + 0.5).bfloat16()
    step = torch.randint(-1, 2, half.shape, generator=gen).to(torch.int16)
    k = (half.view(torch.int16) + step).view(torch.bfloat16)
    k[..., 0], k[..., 1] = 0.0, float(top)
    v = k.flip(0).contiguous()
    v[::2] = torch.randn(v[::2].shape, generator=gen).bfloat16()
    layout = QuantKVLayout.create(bits=bits, head_dim=d, num_kv_heads=hkv, device="cuda")
    cache = layout.allocate(npages)
    cache.append(k.cuda(), v.cuda(), torch.from_numpy(slots).cuda())
    torch.cuda.synchronize()
    assert cache.last_status() == 0
    assert_pools_equal(cache, cpu_twin(cache, k.cuda(), v.cuda(), slots))
