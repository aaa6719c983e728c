"""Prefill exponentials are taken with the base of the steps before and again where a maximum outgrows it: maxima that jump in
one step, in one chunk of it, for some rows only.  And one-tile CTAs with two buffers of scores over many lengths."""

import ctypes

import pytest
import torch

from helpers import ATTN_ATOL, attn_oracle, qkv_case
from kernelforge import _capi, ops

pytestmark = pytest.mark.gpu


def tiles_per_cta(b, h, hk, nq, nk, d, causal):
    t, s = ctypes.c_int(), ctypes.c_int()
    _capi.check(_capi.lib().kfb_flash_attn_plan(b, h, hk, nq, nk, d, int(causal), 1 << 40, ctypes.byref(t), ctypes.byref(s)))
    return t.value


# (B, H, Hk, Nq, Nk, D, causal, tiles per CTA)
KINDS = [(1, 1, 1, 130, 700, 64, True, 1), (3, 16, 16, 1500, 1500, 64, False, 1),
         (2, 1, 1, 3907, 3907, 64, True, 2), (1, 2, 2, 130, 700, 128, False, 1),
         (12, 16, 16, 300, 300, 128, False, 1), (3, 16, 16, 1500, 1500, 128, True, 2)]


@pytest.mark.parametrize("key", [3, 128 + 40, 128 + 75, 256 + 127, -1])
@pytest.mark.parametrize("b,h,hk,nq,nk,d,causal,tiles", KINDS)
def test_a_maximum_that_jumps(b, h, hk, nq, nk, d, causal, tiles, key):
    assert tiles_per_cta(b, h, hk, nq, nk, d, causal) == tiles
    q, k, v = qkv_case(b, h, hk, nq, nk, d, torch.float16, seed=d + nq)
    key = min(key, nk - 1)
    k[:, :, key] *= 12.0           # scores of this key are 12 times as large: above the base for half of the rows, far below for the rest
    got = ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=causal).float().cpu()
    pick = [(0, 0), (b - 1, h - 1)]
    for i, j in pick:
        ref = torch.from_numpy(attn_oracle(q[i:i + 1, j:j + 1], k[i:i + 1, j:j + 1], v[i:i + 1, j:j + 1], causal))
        s = (q[i, j].float() @ k[i, j].float().T).abs().max().item() / d ** 0.5
        # the reference's bound, and the rounding of scores of this size (as in the test of growing maxima)
        assert (got[i, j] - ref[0, 0]).abs().max().item() <= 2e-3 + 8 * 2.0 ** -24 * s * v.abs().max().item()
    assert _capi.device_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("deviation", [6.0, 30.0])
@pytest.mark.parametrize("b,h,hk,nq,nk,d,causal,tiles", KINDS)
def test_maxima_that_keep_growing(b, h, hk, nq, nk, d, causal, tiles, deviation):
    """Sharp scores: in every second step and more some row of a warp outgrows its base, in any of the four chunks."""
    assert tiles_per_cta(b, h, hk, nq, nk, d, causal) == tiles
    q, k, v = qkv_case(b, h, hk, nq, nk, d, torch.float16, seed=nq, scale_q=deviation)
    got = ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=causal).float().cpu()
    for i, j in [(0, 0), (b - 1, h - 1)]:
        ref = torch.from_numpy(attn_oracle(q[i:i + 1, j:j + 1], k[i:i + 1, j:j + 1], v[i:i + 1, j:j + 1], causal))
        s = (q[i, j].float() @ k[i, j].float().T).abs().max().item() / d ** 0.5
        # the reference's bound, and the rounding of scores of this size (as above); P is rounded to 11 bits: 2^-11 of the largest |v|
        vmax = v.abs().max().item()
        assert (got[i, j] - ref[0, 0]).abs().max().item() <= 2e-3 + (8 * 2.0 ** -24 * s + 2.0 ** -11) * vmax
    assert _capi.device_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("nk", [2, 128, 129, 256, 257, 384, 500, 640, 1100, 2048])
def test_two_buffers_of_scores(nk):
    """One tile per CTA at head dim 128, from one step to sixteen; with 256 CTAs, which follow one another on an SM; often."""
    q, k, v = qkv_case(1, 16, 16, nk, nk, 128, torch.bfloat16, seed=nk)
    assert tiles_per_cta(1, 16, 16, nk, nk, 128, True) == 1
    ref = torch.from_numpy(attn_oracle(q[:, :2], k[:, :2], v[:, :2], True))
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    outs = [ops.flash_attn(q, k, v, causal=True) for _ in range(20)]
    assert all(torch.equal(o, outs[0]) for o in outs)
    assert (outs[0][:, :2].float().cpu() - ref).abs().max().item() <= ATTN_ATOL[torch.bfloat16]
    assert _capi.device_status(torch.device("cuda", 0)) == 0
