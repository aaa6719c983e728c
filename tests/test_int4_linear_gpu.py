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


# (M, N, K): tiles with remainders in every direction, one and several batch tiles, odd N (2-byte stores), a last half K
# block of 64 (group 64), split K, two accumulators in flight (tiles of <= 128 batch rows) and one
LARGE = [(33, 64, 128), (33, 257, 1024), (64, 1536, 4224), (96, 511, 640), (129, 130, 256), (257, 300, 2048), (300, 4096, 256),
         (520, 1025, 704), (700, 2304, 1088), (2100, 512, 384)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", LARGE)
def test_gemm_tiles(m, n, k, dtype):
    check(m, n, k, 64, dtype, m % 2 == 0)
    if k % 128 == 0:
        check(m, n, k, 128, dtype, m % 2 == 1)


@pytest.mark.parametrize("m,n,k", [(1, 64, 256), (1, 11264, 256), (5, 36, 256), (31, 260, 512), (33, 132, 256), (70, 300, 4096), (300, 1028, 512)])
def test_silu_pairs_epilogue(m, n, k):
    _, x, packed, scales, _ = int4_case(m, n, k, 128, seed=n)
    args = tuple(torch.from_numpy(a).cuda() for a in (x, packed, scales))
    got = ops.int4_linear_silu_pairs(*args, 128)
    gate, up = ops.int4_linear(*args, 128).view(m, n // 2, 2).unbind(-1)
    want = torch.nn.functional.silu(gate) * up
    assert got.shape == want.shape
    assert (got.float() - want.float()).abs().max() <= 3e-3 * want.float().abs().max()


@pytest.mark.parametrize("m,n,k", [(1, 512, 1024), (2, 512, 1024), (8, 512, 1024), (32, 1536, 1024)])
def test_result_buffer_of_two_byte_alignment(m, n, k):
    """A caller of the C ABI may hand over any element of an fp16 buffer: the 4-byte stores look at the address first."""
    from kernelforge import _capi
    _, x, packed, scales, ref = int4_case(m, n, k, 128, seed=m)
    x, packed, scales = (torch.from_numpy(t).cuda() for t in (x, packed, scales))
    buf = torch.full((m * n + 2,), 7.0, dtype=torch.float16, device="cuda")
    _capi.check(_capi.lib().kfb_int4_linear(x.data_ptr(), packed.data_ptr(), scales.data_ptr(), None, buf.data_ptr() + 2, m, n, k, 128, 0, None, 0,
                                            _capi.stream_ptr(x.device)))
    assert_int4_close(buf[1:-1].view(m, n), ref)
    assert buf[0] == 7.0 and buf[-1] == 7.0
    assert torch.equal(buf[1:-1].view(m, n), ops.int4_linear(x, packed, scales, 128))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(17, 768, 640), (17, 769, 640), (24, 800, 128), (25, 1000, 4224), (32, 769, 8064), (32, 2400, 1152)])
def test_blocks_of_64_above_16_rows(m, n, k, dtype):
    """Groups of 128 walked in blocks of 64, from 49 row blocks on: both sides of the line, fewer blocks than warps, a long K."""
    check(m, n, k, 128, dtype, True)
