"""Decode attention where the split of the keys can go wrong: unsplit, clusters of 2..8 CTAs, splits with a merge kernel; lengths at
the edges of key tiles, empty sequences, splits that get no tile; rings that wrap while K and V come from L2 (the reuse of a
stage), so every call is repeated and has to give the same bits."""

import numpy as np
import pytest
import torch

from kernelforge import ops

from helpers import ATTN_ATOL, attn_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,hk,d,cap,lens", [
    (1, 32, 4, 64, 449, (449,)),                         # 8 tiles: the smallest split group, a last tile of one key
    (1, 32, 4, 64, 448, (448,)),                         # 7 tiles: one CTA per group
    (4, 8, 4, 64, 1024, (0, 1, 64, 65)),                 # most of a cluster has no tile; no key at all
    (2, 16, 8, 128, 800, (800, 577)),
    (8, 32, 4, 64, 4608, (1000, 4096, 4608, 63, 2047, 2048, 2049, 3333)),
    (5, 8, 4, 64, 2048, (2048, 2000, 1, 129, 640)),      # 20 groups: clusters of six
    (3, 8, 8, 128, 1500, (1500, 64, 1437)),              # 24 groups: clusters of five
    (11, 4, 4, 64, 700, tuple(range(640, 651))),         # 44 groups, 11 tiles: too short for clusters of three
    (11, 4, 4, 64, 705, tuple(range(640, 706, 6))),      # 12 tiles: clusters of three
    (16, 8, 4, 128, 1000, tuple(range(0, 1000, 63))),    # 64 groups, 16 tiles: too short for pairs
    (16, 8, 4, 128, 1473, tuple(range(1, 1473, 95))),   # 24 tiles: pairs
    (37, 2, 2, 64, 1600, tuple(range(0, 1600, 44))),     # 74 groups: as many pairs as there are
    (12, 4, 4, 64, 16321, tuple(range(1, 16321, 1483))), # 48 groups of very long caches: clusters of six on the shallow ring
    (20, 4, 4, 64, 8129, tuple(range(0, 8129, 427))),    # 80 groups of long caches: clusters of four on the shallow ring
    (40, 4, 4, 64, 4033, tuple(range(64, 4033, 100))),   # 160 groups of long caches: pairs on the shallow ring
    (1, 34, 2, 64, 16384, (16321,)),                     # 34 / 2 = 17 heads: two chunks; splits and a merge kernel
    (40, 8, 4, 64, 2000, tuple(range(1, 2000, 50))),     # more groups than SMs: the shallow ring, three CTAs per SM
    (40, 8, 8, 128, 900, tuple(range(20, 900, 22))),     # the same at D = 128, two per SM
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_decode_splits(b, h, hk, d, cap, lens, dtype):
    g = torch.Generator(device="cuda").manual_seed(b * cap + d)
    q = torch.randn(b, h, 1, d, generator=g, device="cuda").to(dtype)
    k, v = (torch.randn(b, hk, cap, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    for i, n in enumerate(lens):
        k[i, :, n:], v[i, :, n:] = float("nan"), float("nan")   # rows past the length are never used
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out = [ops.flash_attn_decode(q, k, v, kv_len) for _ in range(12)]
    for o in out[1:]:
        assert torch.equal(o, out[0])
    q, k, v = q.cpu(), k.cpu(), v.cpu()
    for i, n in enumerate(lens):
        if n == 0:
            assert not out[0][i].any()
            continue
        want = attn_oracle(q[i:i + 1], k[i:i + 1, :, :n].contiguous(), v[i:i + 1, :, :n].contiguous(), False)
        assert np.abs(out[0][i:i + 1].float().cpu().numpy() - want).max() <= ATTN_ATOL[dtype]
