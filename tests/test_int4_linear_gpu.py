"""ops.int4_linear (the dispatcher kfb_int4_linear and the kernels it chooses) against the FP32 oracle."""

import numpy as np
import pytest
import torch

from helpers import assert_int4_close, int4_case
from kernelforge import ops

pytestmark = pytest.mark.gpu


def check(m, n, k, group, dtype, with_bias):
    _, x, packed, scales, ref = int4_case(m, n, k, group, seed=m + n + k)
    xs = torch.from_numpy(x).cuda().to(dtype)
    if dtype == torch.bfloat16:   # the oracle sees the rounded activations
        from oracle import kf_oracle as ko
        ref = xs.float().cpu().numpy() @ ko.dequantize(packed, scales, group, np.float32).T
    bias = torch.from_numpy(np.random.default_rng(1).standard_normal(n).astype(np.float32) * 0.1).to(dtype) if with_bias else None
    out = ops.int4_linear(xs, torch.from_numpy(packed).cuda(), torch.from_numpy(scales).cuda(), group, None if bias is None else bias.cuda())
    assert out.shape == (m, n) and out.dtype == dtype
    if bias is not None:
        ref = ref + bias.float().numpy()
    if dtype == torch.float16:
        assert_int4_close(out, ref, f"m{m} n{n} k{k} g{group} bias{with_bias}")
    else:   # bf16 outputs: 8x the fp16 bound
        err = np.abs(out.float().cpu().numpy() - ref).max()
        assert err <= 1.6e-2 * np.abs(ref).max(), f"m{m} n{n} k{k} g{group}: {err}"


# (M, N, K): one row, ragged N (last row block), one scale group, one group more than the warps share evenly, a long K on
# few rows (16 shares of K), more row blocks than one wave of CTAs holds (two blocks per warp at 9 <= M <= 16)
SMALL = [(1, 33, 128), (2, 16, 128), (8, 1, 256), (7, 129, 1152), (8, 1536, 8960), (9, 40, 4096), (16, 7121, 1536), (16, 8960, 640),
         (17, 100, 1024), (32, 1536, 4224), (32, 2050, 2048)]


@pytest.mark.parametrize("dtype,group", [(torch.float16, 128), (torch.float16, 64), (torch.bfloat16, 128), (torch.bfloat16, 64)])
@pytest.mark.parametrize("m,n,k", SMALL)
def test_small_batches(m, n, k, group, dtype):
    check(m, n, k, group, dtype, False)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(1, 77, 256), (5, 1001, 256), (16, 192, 512), (33, 136, 256), (200, 72, 256), (64, 256, 4096)])
def test_bias_in_the_epilogue(m, n, k, dtype):
    check(m, n, k, 128, dtype, True)
