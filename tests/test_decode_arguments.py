"""What decode attention refuses before anything is launched: lengths that are not on the device of the queries, or not lengths."""

import pytest
import torch

from kernelforge import ops


def on(index, t):
    """A host tensor that says it lives on a GPU: enough for checks, which is all that may look at it."""
    kind = type(f"Cuda{index}", (torch.Tensor,), {"is_cuda": True, "device": torch.device("cuda", index)})
    return t.as_subclass(kind)


def operands(b=2):
    return [on(0, torch.zeros(b, 4, n, 64, dtype=torch.float16)) for n in (1, 70, 70)]


@pytest.mark.parametrize("call", ["flash_attn_decode", "flash_attn_decode_step", "flash_attn_decode_partial"])
def test_lengths_on_another_gpu(call):
    with pytest.raises(ValueError, match="one CUDA device"):
        getattr(ops, call)(*operands(), on(1, torch.ones(2, dtype=torch.int32)))


@pytest.mark.parametrize("call", ["flash_attn_decode", "flash_attn_decode_step", "flash_attn_decode_partial"])
@pytest.mark.parametrize("lengths", [torch.ones(2, dtype=torch.int32), on(0, torch.ones(2, dtype=torch.int64)), on(0, torch.ones(1, dtype=torch.int32))])
def test_lengths_that_are_none(call, lengths):
    with pytest.raises(TypeError, match="kv_len must be"):
        getattr(ops, call)(*operands(), lengths)


@pytest.mark.parametrize("call", ["flash_attn_decode", "flash_attn_decode_step"])
def test_caches_that_no_kernel_reads_in_place(call):
    q, k, v = operands()
    lengths = on(0, torch.ones(2, dtype=torch.int32))
    with pytest.raises(ValueError, match="share strides"):
        getattr(ops, call)(q, k, on(0, torch.zeros(2, 4, 140, 64, dtype=torch.float16)[:, :, ::2]), lengths)
    odd = [on(0, torch.zeros(2, 4, 70, 68, dtype=torch.float16)[..., :64]) for _ in "kv"]
    with pytest.raises(ValueError, match="multiples of 8"):
        getattr(ops, call)(q, *odd, lengths)


def test_a_step_takes_lengths_as_they_lie():
    with pytest.raises(ValueError, match="contiguous kv_len"):
        ops.flash_attn_decode_step(*operands(), on(0, torch.ones(4, dtype=torch.int32)[::2]))
