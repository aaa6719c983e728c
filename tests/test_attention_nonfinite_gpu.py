"""Scores that are NaN or +infinity: softmax makes their rows NaN, wherever the key lies in its block, and leaves the others alone."""

import pytest
import torch

from helpers import ATTN_ATOL, attn_oracle, qkv_case
from kernelforge import ops

pytestmark = pytest.mark.gpu

# one-tile and two-tile CTAs, several heads of a group in one tile, key splits
SHAPES = [(1, 2, 2, 130, 200), (4, 16, 16, 300, 300), (1, 8, 1, 16, 700), (1, 1, 1, 40, 4097)]
PLACES = [0, 5, 7, 31, 130]   # of the key; 130: past the first step


def expected(q, k, v, causal):
    clean = torch.where(torch.isfinite(k.float()) & (k.float().abs() < 1e30), k, torch.zeros((), dtype=k.dtype))
    ref = torch.from_numpy(attn_oracle(q, clean, v, causal))
    group = q.shape[1] // k.shape[1]
    s = q.float() @ k.float().repeat_interleave(group, 1).transpose(2, 3)
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[2:], dtype=torch.bool).tril(k.shape[2] - q.shape[2]), 0.0)
    bad = ~torch.isfinite(s).all(-1)
    return ref, bad


def check(got, ref, bad, tol):
    assert bad.any()
    assert torch.isnan(got[bad]).all()
    if (~bad).any():
        assert (got - ref)[~bad].abs().max().item() <= tol


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,h,hk,nq,nk", SHAPES)
def test_nan_key_makes_the_rows_that_see_it_nan(b, h, hk, nq, nk, d, place, dtype):
    q, k, v = qkv_case(b, h, hk, nq, nk, d, dtype, seed=place + d)
    k[0, 0, place] = float("nan")
    ref, bad = expected(q, k, v, True)
    check(ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=True).float().cpu(), ref, bad, ATTN_ATOL[dtype])


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("d", [64, 128])
def test_score_of_plus_infinity_makes_its_row_nan(d, place):
    q, k, v = qkv_case(2, 2, 2, 150, 200, d, torch.bfloat16, seed=place)
    q[..., 0] = 0.0
    k[..., 0] = 0.0
    q[0, 1, 140, 0] = k[0, 1, place, 0] = 3e38    # their product overflows FP32; no other row has a first feature
    ref, bad = expected(q, k, v, True)
    assert bad.sum() == 1
    check(ops.flash_attn(q.cuda(), k.cuda(), v.cuda(), causal=True).float().cpu(), ref, bad, ATTN_ATOL[torch.bfloat16])


# (sequences, heads, KV heads, keys): one CTA per group; clusters of splits; more than eight splits and the merge kernel
DECODE = [(40, 8, 4, 300), (8, 32, 4, 2000), (1, 34, 2, 16384)]


@pytest.mark.parametrize("score", ["nan", "inf", "all nan"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,h,hk,nk", DECODE)
def test_decode_makes_the_rows_that_see_it_nan(b, h, hk, nk, d, score):
    q, k, v = qkv_case(b, h, hk, 1, nk, d, torch.bfloat16, seed=d)
    lens = torch.full((b,), nk, dtype=torch.int32)
    lens[-1] = nk - 70
    k[-1, :, nk - 70:] = float("nan")          # not valid keys: nothing sees them
    v[-1, :, nk - 70:] = float("nan")
    valid = torch.arange(nk)[None, :] < lens[:, None]
    clean = lambda t: torch.where(valid[:, None, :, None], t, torch.zeros((), dtype=t.dtype))
    ref = torch.cat([torch.from_numpy(attn_oracle(q[i:i + 1], clean(k)[i:i + 1, :, :lens[i]], clean(v)[i:i + 1, :, :lens[i]], False)) for i in range(b)])
    group = h // hk
    bad = torch.zeros(b, h, 1, dtype=torch.bool)
    if score == "inf":      # the product overflows FP32 for one head; the others of its group have no such feature
        q[..., 0] = 0.0
        k[:, :, :, 0] = 0.0
        ref = torch.cat([torch.from_numpy(attn_oracle(q[i:i + 1], clean(k)[i:i + 1, :, :lens[i]], clean(v)[i:i + 1, :, :lens[i]], False)) for i in range(b)])
        q[0, 1, 0, 0] = k[0, 1 // group, 77, 0] = 3e38
        bad[0, 1] = True
    else:                   # one key, or the first 64 keys: the first piece of the row then has no number at all
        k[0, 0, 0 if score == "nan" else slice(0, nk // 16)] = float("nan")
        bad[0, :group] = True
    got = ops.flash_attn_decode(q.cuda(), k.cuda(), v.cuda(), lens.cuda()).float().cpu()
    check(got, ref, bad, ATTN_ATOL[torch.bfloat16])
    if b == 1:
        return
    none = ops.flash_attn_decode(q.cuda(), k.cuda(), v.cuda(), torch.zeros_like(lens).cuda())
    assert not none.any()      # no valid key: zeros, whatever the cache holds
