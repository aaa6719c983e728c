"""The GPU quantiser at the values where its reciprocal shortcut must hand over to the exact division, bit for bit against
the torch formulation (kernelforge.quantize on a CPU tensor)."""

import pytest
import torch

from kernelforge import quantize as kq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("n,k", [(1, 128), (3, 192), (129, 1152), (1000, 256)])
def test_bits_at_half_integers_and_extremes(n, k, group, dtype):
    if k % group:
        pytest.skip("K is not a multiple of the group")
    g = torch.Generator().manual_seed(n + k + group)
    w = torch.randn(n, k, generator=g) * 0.02
    ties = w[:, ::3].sign() * (torch.randint(0, 15, w[:, ::3].shape, generator=g) * 0.5)   # multiples of half a step
    w[:, ::3] = ties * 0.015625
    w[:, 5::7] = 0.109375                       # 7 steps of 2^-6: the scale is exactly 2^-6
    w[0, :group] = 0.0                          # an all-zero group
    if n > 1:
        w[1] = torch.randn(k, generator=g) * 1e-6   # below the smallest scale
    if n > 2:
        w[2] = torch.randn(k, generator=g) * (1e4 if dtype == torch.float16 else 3e5)
    w = w.to(dtype)
    want, got = kq.quantize_weight(w, group), kq.quantize_weight(w.cuda(), group)
    assert torch.equal(got.packed.cpu(), want.packed)
    assert torch.equal(got.scales.cpu().view(torch.int16), want.scales.view(torch.int16))


def test_nan_and_infinity_take_the_definition():
    """Not meaningful as weights, but the words stay what rint / clamp give: NaN and -inf the smallest code, in the lane only."""
    w = torch.randn(2, 256, generator=torch.Generator().manual_seed(0)) * 0.02
    clean = kq.quantize_weight(w.cuda(), 128)
    bad = w.clone()
    bad[0, 9] = float("nan")
    got = kq.quantize_weight(bad.cuda(), 128)
    q, q0 = kq.unpack_int4(got.packed).cpu(), kq.unpack_int4(clean.packed).cpu()
    assert q[0, 9] == -8 and torch.equal(q[1], q0[1]) and torch.equal(q[0, 16:], q0[0, 16:])
