"""The kernels of a prompt's prefill against the torch formulation of the same steps (the roundings are the same, so bit for
bit where no transcendental is involved)."""

import pytest
import torch

from kernelforge import _capi, ops

pytestmark = pytest.mark.gpu


def rand(*size, seed=0):
    return torch.randn(*size, generator=torch.Generator().manual_seed(seed)).half().cuda()


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("b,t,h,hk,d,lmax", [(1, 1, 1, 1, 64, 1), (2, 5, 4, 2, 64, 9), (3, 67, 6, 1, 128, 80)])
def test_rope_tokens_and_attention_tokens(b, t, h, hk, d, lmax, pairs):
    qkv = rand(b * t, (h + 2 * hk) * d)
    ang = torch.rand(lmax, d // 2, generator=torch.Generator().manual_seed(1)).repeat(1, 2) * 6
    cos, sin = ang.cos().cuda(), ang.sin().cuda()
    kc, vc = rand(b, hk, lmax, d, seed=2), rand(b, hk, lmax, d, seed=3)
    k_old, v_old = kc.clone(), vc.clone()
    q = ops.rope_tokens(qkv, cos, sin, kc, vc, b, h, pairs)
    x = qkv.view(b, t, h + 2 * hk, d)
    nat = x[:, :, :h + hk]
    if pairs:
        nat = nat.reshape(b, t, h + hk, d // 2, 2).transpose(-1, -2).reshape(b, t, h + hk, d)
    f = nat.float()
    rot = torch.cat([-f[..., d // 2:], f[..., :d // 2]], -1)
    want = (f * cos[:t, None] + rot * sin[:t, None]).half()
    assert torch.equal(q, want[:, :, :h])
    assert torch.equal(kc[:, :, :t], want[:, :, h:].transpose(1, 2)) and torch.equal(vc[:, :, :t], x[:, :, h + hk:].transpose(1, 2))
    assert torch.equal(kc[:, :, t:], k_old[:, :, t:]) and torch.equal(vc[:, :, t:], v_old[:, :, t:])
    o = ops.attention_tokens(q, kc, vc, t, True)
    same = ops.flash_attn(q.transpose(1, 2).contiguous(), kc[:, :, :t].contiguous(), vc[:, :, :t].contiguous(), causal=True)
    assert torch.equal(o, same.transpose(1, 2))


@pytest.mark.parametrize("rows,inter", [(1, 1), (3, 7), (5, 64), (130, 1026)])
def test_silu_mul_pairs(rows, inter):
    gu = rand(rows, 2 * inter)
    gate, up = gu.view(rows, inter, 2).unbind(-1)
    want = torch.nn.functional.silu(gate) * up
    assert (ops.silu_mul(gu, pairs=True).float() - want.float()).abs().max() <= 2e-3 * want.float().abs().max() + 1e-6


@pytest.mark.parametrize("hidden", [8, 2048, 2056, 8192, 12296, 32768])
def test_rmsnorm_widths(hidden):
    x, r, w = rand(3, hidden), rand(3, hidden, seed=1), rand(hidden, seed=2)
    y, s = ops.add_rmsnorm(x, w, 1e-5, r)
    f = (x + r).float()
    want = (f * torch.rsqrt(f.pow(2).mean(-1, keepdim=True) + 1e-5)).half() * w
    assert torch.equal(s, x + r)
    assert (y.float() - want.float()).abs().max() <= 2e-3 * want.float().abs().max()


def test_prompt_ids_are_table_indices():
    """Negative ids count from the end, as torch indexing has them; an id outside the table is reported, nothing faults."""
    g = torch.Generator(device="cuda").manual_seed(4)
    embed = torch.randn(300, 256, generator=g, device="cuda", dtype=torch.float16)
    w = torch.ones(256, device="cuda", dtype=torch.float16)
    ids = torch.tensor([0, 299, -1, -300, 17], device="cuda")
    assert torch.equal(ops.embed_rmsnorm(ids, embed, w, 1e-5, prompt=True)[1], embed[ids])
    dev = torch.device("cuda", 0)
    assert _capi.device_status(dev) == 0
    try:
        for bad in (300, -301, 1 << 40):
            ops.embed_rmsnorm(torch.tensor([5, bad], device="cuda"), embed, w, 1e-5, prompt=True)
            torch.cuda.synchronize()
            assert _capi.device_status(dev) == 0x702
            _capi.device_status_reset(dev)
    finally:
        _capi.device_status_reset(dev)
        torch.cuda.synchronize()
