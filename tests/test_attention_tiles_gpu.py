"""Prefill attention where its cutting into tiles can go wrong: several heads of a group in one tile, tiles without a partner,
key splits (with pieces that a causal row never reaches), head dim 128 on the two-tile kernel."""

import pytest
import torch

from helpers import ATTN_ATOL, attn_oracle, qkv_case
from kernelforge import _capi, ops

pytestmark = pytest.mark.gpu

# (B, H, Hk, Nq, Nk): packed heads (16 x 8 = a full tile; 5 x 6; 43 x 2 of 4; 128 x 1 of 3), one tile per head (G = 1) on few
# and on many heads, odd numbers of tiles, one key more than a step, long caches that are split
SHAPES = [(1, 8, 1, 16, 513), (2, 6, 1, 5, 129), (1, 4, 1, 43, 700), (1, 3, 1, 128, 128), (2, 2, 2, 2, 1030), (20, 8, 8, 70, 140),
          (1, 2, 2, 129, 129), (1, 2, 1, 300, 900), (1, 1, 1, 257, 4097), (1, 4, 2, 100, 3000), (3, 2, 1, 385, 640)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,h,hk,nq,nk", SHAPES)
def test_tiles_and_splits(b, h, hk, nq, nk, d, causal, dtype):
    q, k, v = qkv_case(b, h, hk, nq, nk, d, dtype, seed=nq + nk + d)
    got = ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=causal)
    ref = torch.from_numpy(attn_oracle(q, k, v, causal))
    assert (got.float().cpu() - ref).abs().max().item() <= ATTN_ATOL[dtype]
    assert _capi.device_status(torch.device("cuda", 0)) == 0


# One step of keys per CTA (one buffer of scores) next to two (two buffers), grids below and above one CTA per SM, splits of one step
ONE_STEP = [(1, 1, 1, 2, 2), (11, 8, 8, 3, 3), (2, 4, 1, 32, 127), (1, 32, 32, 128, 128), (1, 4, 4, 128, 129), (18, 8, 8, 50, 50), (19, 8, 8, 50, 50),
            (1, 1, 1, 2, 1000), (1, 2, 2, 6, 1480), (2, 32, 4, 2, 422), (1, 8, 8, 20, 385), (1, 8, 8, 100, 512)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h,hk,nq,nk", ONE_STEP)
def test_one_step_of_keys(b, h, hk, nq, nk, causal, dtype):
    q, k, v = qkv_case(b, h, hk, nq, nk, 128, dtype, seed=3 * nq + nk)
    ref = torch.from_numpy(attn_oracle(q, k, v, causal))
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    got = [ops.flash_attn(q, k, v, causal=causal) for _ in range(3)]
    assert (got[0].float().cpu() - ref).abs().max().item() <= ATTN_ATOL[dtype]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert _capi.device_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("d", [64, 128])
def test_large_scores_and_growing_maxima(d):
    """Rows whose maximum grows by far more than the rescale threshold from step to step, and rows far below zero."""
    q, k, v = qkv_case(1, 2, 1, 260, 1000, d, torch.float16, seed=1)
    k = k * torch.linspace(0.1, 30.0, 1000).view(1, 1, -1, 1).half()
    got = ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=True)
    ref = torch.from_numpy(attn_oracle(q, k, v, True))
    s = (q.float()[:, :, -1:] @ k.float().expand(1, 2, -1, -1).transpose(2, 3)).abs().max().item() / d ** 0.5
    assert (got.float().cpu() - ref).abs().max().item() <= 2e-3 + 8 * 2.0 ** -24 * s * v.abs().max().item()


def test_the_workspace_is_optional():
    q, k, v = (t.cuda() for t in qkv_case(1, 2, 1, 200, 3000, 64, torch.float16, seed=2))
    lib = _capi.lib()
    assert lib.kfb_flash_attn_ws_bytes(1, 2, 1, 200, 3000, 64) > 0
    o = torch.empty_like(q)
    _capi.check(lib.kfb_flash_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), 0, 1, 2, 1, 200, 3000, 64, 1, 0.125, None,
                                       None, 0, _capi.stream_ptr(q.device)))
    assert (o.float() - ops.flash_attn(q, k, v, causal=True).float()).abs().max().item() <= 1e-3
