"""Calls that the native host path (csrc/host.cpp) has to take, decline or refuse as the Python operators do."""

import pytest
import torch

from kernelforge import ops
from kernelforge import quantize as kq

pytestmark = pytest.mark.gpu


def weight(n, k, seed=1, group=128):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return kq.quantize_weight(torch.randn(n, k, generator=g, device="cuda", dtype=torch.float16) * 0.02, group)


def test_a_result_that_does_not_fit_raises_torchs_out_of_memory_error():
    """The 256 GB result is refused by the allocator, before any launch."""
    packed = torch.zeros(1 << 20, 8, dtype=torch.int32, device="cuda")
    scales = torch.ones(1 << 20, 1, dtype=torch.float16, device="cuda")
    x = torch.zeros(1 << 17, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        ops.int4_linear(x, packed, scales, 64)
    torch.cuda.empty_cache()
    assert not ops.int4_linear(x[:3], packed, scales, 64).any()    # and the next call works


@pytest.mark.parametrize("call", ["flash_attn", "flash_attn_kv_view", "flash_attn_decode"])
def test_a_scale_that_is_not_a_number_is_refused(call):
    q, kv = torch.zeros(1, 2, 1, 64, dtype=torch.float16, device="cuda"), torch.zeros(1, 2, 70, 64, dtype=torch.float16, device="cuda")
    lengths = (torch.ones(1, dtype=torch.int32, device="cuda"),) if call == "flash_attn_decode" else ()
    with pytest.raises(ValueError, match="scale must be positive"):
        getattr(ops, call)(q, kv, kv, *lengths, scale=float("nan"))


@pytest.mark.parametrize("m", [1, 5, 40])
def test_group_size_may_be_any_number_equal_to_it(m):
    qw = weight(256, 512)
    x = torch.randn(m, 512, device="cuda", dtype=torch.float16)
    got = ops.int4_matmul(x, qw.packed, qw.scales, 128.0)
    assert got is not None and torch.equal(got, ops.int4_matmul(x, qw.packed, qw.scales, 128))


def test_wrappers_of_torch_func_are_never_read_as_memory():
    """The operands of vmap, grad and jvp look like plain tensors and have no memory: a call raises, or (where torch can take it
    apart) gives what the calls one by one give.  It does not crash."""
    qw = weight(256, 512)
    x = torch.randn(2, 4, 512, device="cuda", dtype=torch.float16)
    q, kv = torch.randn(2, 1, 2, 3, 64, device="cuda", dtype=torch.float16), torch.randn(2, 1, 2, 70, 64, device="cuda", dtype=torch.float16)
    linear = lambda t: ops.int4_linear(t, qw.packed, qw.scales)
    attend = lambda t: ops.flash_attn(t, kv[0], kv[0])
    one_by_one = torch.stack([ops.flash_attn(q[i], kv[i], kv[i]) for i in range(2)])
    calls = [(lambda: torch.func.vmap(linear)(x), linear(x)), (lambda: torch.func.jvp(linear, (x[0],), (x[1],))[0], linear(x[0])),
             (lambda: torch.func.grad(lambda t: linear(t).float().sum())(x[0]), torch.zeros_like(x[0])),
             (lambda: torch.func.vmap(ops.flash_attn)(q, kv, kv), one_by_one), (lambda: torch.func.vmap(ops.flash_attn_kv_view)(q, kv, kv), one_by_one),
             (lambda: torch.func.jvp(attend, (q[0],), (q[1],))[0], attend(q[0])),
             (lambda: torch.func.vmap(lambda w: kq.quantize_weight(w).packed)(x), torch.stack([kq.quantize_weight(w).packed for w in x]))]
    raised = 0
    for call, want in calls:
        try:
            got = call()
        except (RuntimeError, ValueError):
            raised += 1
        else:
            assert torch.equal(got, want)
    assert raised >= 3
    assert torch.isfinite(linear(x)).all()


@pytest.mark.parametrize("prepacked", [False, True])
@pytest.mark.parametrize("m", [1, 4, 40])
def test_a_bias_that_is_trained_batched_or_dual_is_added_by_torch(m, prepacked):
    """The product has no backward, its bias is an ordinary addend: gradients, vmap and forward mode over it work."""
    n, k = 256, 512
    qw = weight(n, k)
    if prepacked:
        ops.prepack_weight_(qw.packed)
    x = torch.randn(m, k, device="cuda", dtype=torch.float16)
    y = ops.int4_linear(x, qw.packed, qw.scales)
    bias = torch.randn(n, device="cuda", dtype=torch.float16)
    linear = lambda b: ops.int4_linear(x, qw.packed, qw.scales, 128, b)
    assert torch.equal(linear(bias), y + bias)
    trained = torch.nn.Parameter(bias.clone())
    out = linear(trained)
    out.backward(torch.ones_like(out))
    assert torch.equal(out, y + bias) and torch.equal(trained.grad, torch.full_like(bias, m))
    with torch.no_grad():
        assert not linear(trained).requires_grad
    several = torch.randn(3, n, device="cuda", dtype=torch.float16)
    assert torch.equal(torch.func.vmap(linear)(several), y + several[:, None])
    if prepacked:
        return   # (its entry allocates in Python: a transform of torch.func that wraps every new tensor is refused)
    value, tangent = torch.func.jvp(linear, (bias,), (several[0],))
    assert torch.equal(value, y + bias) and torch.equal(tangent, several[0].expand(m, n))


def test_lengths_may_be_a_strided_view():
    q, kv = (torch.randn(3, 4, n, 64, device="cuda", dtype=torch.float16) for n in (1, 900))
    table = torch.tensor([[900, 1], [7, 2], [450, 3]], dtype=torch.int32, device="cuda")
    lengths = table[:, 0]
    want = ops.flash_attn_decode(q, kv, kv, lengths.contiguous())
    assert torch.equal(ops.flash_attn_decode(q, kv, kv, lengths), want)
    part = lambda n: ops.flash_attn_merge_partials(ops.flash_attn_decode_partial(q, kv, kv, n), q, 4, 900)
    assert torch.equal(part(lengths), part(lengths.contiguous()))


def test_both_decode_calls_are_native(monkeypatch):
    """A plain call stays off the general Python route (16 us of host time instead of 4)."""
    q, kv = torch.randn(2, 4, 1, 64, device="cuda", dtype=torch.float16), torch.randn(2, 4, 200, 64, device="cuda", dtype=torch.float16)
    lengths = torch.tensor([200, 7], dtype=torch.int32, device="cuda")
    view = torch.randn(2, 4, 264, 64, device="cuda", dtype=torch.float16)[:, :, 64:]
    own = q.as_subclass(type("Own", (torch.Tensor,), {}))
    want = [ops.flash_attn_decode(q, c, c, lengths) for c in (kv, view)]
    assert torch.equal(ops.flash_attn_decode_step(own, kv, kv, lengths).as_subclass(torch.Tensor), want[0])
    monkeypatch.setattr(ops, "_decode_general", None)
    for call in (ops.flash_attn_decode, ops.flash_attn_decode_step):
        assert all(torch.equal(call(q, c, c, lengths), w) for c, w in zip((kv, view), want))
