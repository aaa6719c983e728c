"""The streaming lm_head at the edges of its batches: vocabulary rows and K chunks that do not fill one, every number of batch columns."""

import pytest
import torch

from kernelforge import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("n,k", [(1, 32), (15, 64), (16, 96), (127, 128), (129, 160), (1000, 256), (263, 288), (4100, 2048), (130, 1056)])
def test_ragged_rows_and_chunks(m, n, k):
    g = torch.Generator().manual_seed(n + k + m)
    h, w = torch.randn(m, k, generator=g).half(), (torch.randn(n, k, generator=g) * 0.05).half()
    w[n // 2] = w[-1]     # a tie: the first maximum wins
    best = torch.zeros(m, dtype=torch.int64, device="cuda")
    logits = ops.lm_head_argmax(h.cuda(), w.cuda(), None, best)
    ref = h.double() @ w.double().T
    # products of 16-bit numbers are exact in FP32: k additions at most 2^-24 of the running sum each, and one rounding to fp16
    bound = k * 2.0 ** -24 * (h.double().abs() @ w.double().abs().T) + ref.abs() * 2.0 ** -11 + 2.0 ** -24
    assert ((logits.cpu().double() - ref).abs() <= bound).all()
    first = (logits.cpu() == logits.cpu().max(1, keepdim=True).values).int().argmax(1)
    assert torch.equal(0xFFFFFFFF - (best.cpu() & 0xFFFFFFFF), first.long())
    assert torch.equal(ops.lm_head_argmax(h.cuda(), w.cuda()), logits)
