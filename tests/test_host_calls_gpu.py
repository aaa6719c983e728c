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
