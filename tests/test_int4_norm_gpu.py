"""RMSNorm fused with the INT4 linear behind it, against the two separate kernels: row counts around the 16-row blocks, around
two blocks per SM and where a CTA owns three, four and five blocks, in a full second wave and in one that is left to the other kernel; the smallest and largest share of K per warp; both group
sizes; the residual epilogue of the linears without a norm."""

import pytest
import torch

from kernelforge import ops, quantize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k,group", [
    (2, 128, 128), (16, 64, 64), (18, 256, 64), (2560, 2048, 128), (4736, 2048, 128), (4738, 2048, 128), (7106, 1024, 64),
    (9474, 2048, 64), (11264, 2048, 128), (14000, 1024, 128), (22016, 512, 128), (1000, 4096, 128), (640, 3072, 64), (48, 4096, 64), (5000, 4096, 128),
])
def test_norm_linear(m, n, k, group):
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").half()
    qw = quantize.quantize_weight(rn(n, k) * 0.05, group)
    x, w, res = rn(m, k) * 3, 1 + 0.1 * rn(k), rn(m, n)
    wd = quantize.dequantize(qw, torch.float32)
    want = ops.add_rmsnorm(x, w, 1e-5)[0].float() @ wd.T
    tol = 2e-3 * want.abs().max().item()
    got = ops.int4_gemv_fused(x, qw.packed, qw.scales, group, ops.XFORM_RMSNORM, w, 1e-5)
    assert (got.float() - want).abs().max().item() <= tol
    got = ops.int4_gemv_silu_pair(x, qw.packed, qw.scales, group, w, 1e-5)
    act = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    assert (got.float() - act).abs().max().item() <= 4e-3 * max(act.abs().max().item(), want.abs().max().item())
    got = ops.int4_gemv_fused(x, qw.packed, qw.scales, group, residual=res)
    want = x.float() @ wd.T + res.float()
    assert (got.float() - want).abs().max().item() <= 2e-3 * want.abs().max().item()


@pytest.mark.parametrize("b", [1, 2])
def test_norm_rope_kv(b):
    h, hk, d, k, lmax, pos = 32, 4, 64, 2048, 24, 9
    g = torch.Generator(device="cuda").manual_seed(b)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").half()
    qw = quantize.quantize_weight(rn((h + 2 * hk) * d, k) * 0.05, 128)
    x, w = rn(b, k), 1 + 0.1 * rn(k)
    ang = torch.outer(torch.arange(lmax, device="cuda").float(), 1e4 ** (-torch.arange(0, d, 2, device="cuda").float() / d))
    cos, sin = (f(torch.cat([ang, ang], -1)).contiguous() for f in (torch.cos, torch.sin))
    at = torch.tensor([pos], device="cuda")
    caches = [torch.zeros(b, hk, lmax, d, dtype=torch.float16, device="cuda") for _ in range(4)]
    got = ops.int4_gemv_rope_kv(x, qw.packed, qw.scales, 128, cos, sin, at, caches[0], caches[1], h, w, 1e-5)
    want = ops.int4_gemv_rope_kv(ops.add_rmsnorm(x, w, 1e-5)[0], qw.packed, qw.scales, 128, cos, sin, at, caches[2], caches[3], h)
    for a, c in ((got, want), (caches[0], caches[2]), (caches[1], caches[3])):
        assert (a.float() - c.float()).abs().max().item() <= 2e-3 * c.float().abs().max().item()
    assert not caches[0][:, :, :pos].any() and not caches[1][:, :, pos + 1:].any()


@pytest.mark.parametrize("mean", [0.0, 4.0, -4.0])
@pytest.mark.parametrize("m,n,k,group", [(1, 7106, 1024, 64), (2, 9474, 2048, 64), (1, 11264, 2048, 128), (2, 11000, 2048, 128)])
def test_nibbles_multiplied_as_they_are(m, n, k, group, mean):
    """Several row blocks per CTA take nibbles without their offset of 8, which is made up for by the sum of the activations: also
    where that sum is large because they have one sign."""
    g = torch.Generator(device="cuda").manual_seed(n)
    qw = quantize.quantize_weight((torch.randn(n, k, generator=g, device="cuda") * 0.05).half(), group)
    x, w = (torch.randn(m, k, generator=g, device="cuda") + mean).half(), torch.ones(k, device="cuda").half()
    got = ops.int4_gemv_fused(x, qw.packed, qw.scales, group, ops.XFORM_RMSNORM, w, 1e-5).double()
    h, wd = ops.add_rmsnorm(x, w, 1e-5)[0].double(), quantize.dequantize(qw, torch.float32).double()
    ref = h @ wd.T
    # FP32 sums of nibble * activation, nibbles up to 15 with an offset of 8: at most 2 * 2^-24 of the sum of their magnitudes for each
    # of the additions that a sum goes through (k / 16 in the tensor core, 32 around it); the norm's own rounding may differ by one
    # step of fp16 in an activation here and there; one rounding to fp16
    terms = h.abs() @ (wd.abs() + 8 * qw.scales.double().repeat_interleave(group, 1)).T
    bound = 2 * (k / 16 + 32) * 2.0 ** -24 * terms + 2.0 ** -10 * (h.abs() @ wd.abs().T) / 16 + ref.abs() * 2.0 ** -11
    assert ((got - ref).abs() <= bound).all()
    assert (got - ref).mean().abs().item() <= 0.1 * 2.0 ** -11 * ref.abs().max().item()     # unbiased


@pytest.mark.parametrize("at", [[0], [3], [517], [1022], [64, 700], [1, 2, 3]])
@pytest.mark.parametrize("m,n,k,group", [(1, 2048, 1024, 128), (1, 7106, 1024, 64), (2, 7107, 2048, 64), (2, 9474, 2048, 128), (1, 11264, 2048, 128), (2, 11264, 1024, 64)])
def test_activations_that_overflow(m, n, k, group, at):
    """A normalised activation past the largest fp16 number: results are what the definition gives, infinite with the sign of the product and
    NaN where the nibble is zero or two infinities differ in sign.  The other batch row stays as it is."""
    g = torch.Generator(device="cuda").manual_seed(n + k)
    qw = quantize.quantize_weight((torch.randn(n, k, generator=g, device="cuda") * 0.05).half(), group)
    x, w = torch.randn(m, k, generator=g, device="cuda").half(), torch.ones(k, device="cuda").half()
    for i, j in enumerate(at):
        x[0, j], w[j] = (-1.0) ** i * 20.0, 60000.0
    x[1:, at] = 0.0
    h, wd = ops.add_rmsnorm(x, w, 1e-5)[0].double(), quantize.dequantize(qw, torch.float32).double()
    assert h[0, at].isinf().all() and h.isinf().sum() == len(at)
    want = torch.stack([(row * wd).sum(1) for row in h])
    got = ops.int4_gemv_fused(x, qw.packed, qw.scales, group, ops.XFORM_RMSNORM, w, 1e-5).double()
    assert not want[0].isfinite().any() and want[1:].isfinite().all()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[got.isinf()], want[want.isinf()])
    if m > 1:
        assert (got[1] - want[1]).abs().max().item() <= 2e-3 * want[1].abs().max().item()
