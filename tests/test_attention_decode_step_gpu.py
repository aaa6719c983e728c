"""Decode attention that reads old cache rows before the kernel in front has finished: the same bits as the plain call, whichever
kernel wrote the last row, with the last row first or last in its tile, empty and partly empty splits, clusters and single CTAs."""

import pytest
import torch

from kernelforge import _capi, ops

pytestmark = pytest.mark.gpu

# (B, H, Hk, D, capacity): one CTA per group, shallow and deep rings; clusters; more than eight splits and the merge kernel
CASES = [(3, 8, 2, 64, 300), (40, 8, 4, 128, 300), (2, 32, 4, 64, 1200), (3, 4, 4, 128, 900), (24, 8, 4, 64, 4600), (1, 34, 2, 64, 16384)]


@pytest.mark.parametrize("b,h,hk,d,cap", CASES)
def test_same_bits_as_the_plain_call(b, h, hk, d, cap):
    g = torch.Generator(device="cuda").manual_seed(cap + d)
    rn = lambda *size: torch.randn(*size, generator=g, device="cuda").half()
    q, k, v = rn(b, h, 1, d), rn(b, hk, cap, d), rn(b, hk, cap, d)
    edges = [1, 2, 63, 64, 65, 128, 129, 193, cap - 63, cap - 1, cap]
    for shift in range(len(edges)):
        lens = torch.tensor([min(cap, max(1, edges[(i + shift) % len(edges)])) for i in range(b)], dtype=torch.int32, device="cuda")
        assert torch.equal(ops.flash_attn_decode_step(q, k, v, lens), ops.flash_attn_decode(q, k, v, lens)), lens
    none = torch.zeros(b, dtype=torch.int32, device="cuda")
    assert not ops.flash_attn_decode_step(q, k, v, none).any()
    assert _capi.device_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("b,h,hk,d,cap", [(2, 32, 4, 64, 1200), (8, 8, 4, 128, 300)])
def test_the_kernel_in_front_writes_the_last_row(b, h, hk, d, cap):
    """A chain of RoPE + cache write and attention, as in a decode step; every position checked against a call that waits."""
    g = torch.Generator(device="cuda").manual_seed(d)
    rn = lambda *size: torch.randn(*size, generator=g, device="cuda")
    cos, sin = rn(cap, d), rn(cap, d)
    k, v = torch.zeros(b, hk, cap, d, device="cuda", dtype=torch.float16), torch.zeros(b, hk, cap, d, device="cuda", dtype=torch.float16)
    steps = [i for i in range(cap - 1) if i < 140 or i % 64 in (0, 63)]
    qkvs = [rn(b, (h + 2 * hk) * d).half() for _ in steps]
    poss = [torch.tensor([i], device="cuda") for i in steps]
    lens = [torch.full((b,), i + 1, dtype=torch.int32, device="cuda") for i in steps]
    torch.cuda.synchronize()
    got, want = [], []
    for qkv, pos, n in zip(qkvs, poss, lens):
        got.append(ops.flash_attn_decode_step(ops.rope_kv_write(qkv, cos, sin, pos, k, v, h), k, v, n))
    k.zero_(), v.zero_()
    for qkv, pos, n in zip(qkvs, poss, lens):
        q = ops.rope_kv_write(qkv, cos, sin, pos, k, v, h)
        torch.cuda.synchronize()
        want.append(ops.flash_attn_decode(q, k, v, n))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
