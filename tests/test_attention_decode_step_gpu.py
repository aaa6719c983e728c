"""Decode attention that reads old cache rows before the kernel in front has finished: the same bits as the plain call, whichever
kernel wrote the last row, with the last row first or last in its tile, empty and partly empty splits, clusters and single CTAs."""

import pytest
import torch

from kernelforge import _capi, ops, quantize

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


# What writes q and the last row: RoPE + cache write on its own, or in the epilogue of the projection, which goes on for two
# microseconds after it has let the attention start.  Clusters; one CTA per group with more tiles than its ring holds (the wait is then
# at the end of the ring) and with fewer; more than eight splits and the merge kernel.
CHAINS = [("rope", 2, 32, 4, 64, 1200), ("rope", 8, 8, 4, 128, 300), ("rope", 40, 8, 4, 64, 600), ("rope", 40, 8, 4, 128, 300),
          ("rope", 1, 8, 2, 64, 16384), ("projection", 1, 32, 4, 64, 1200), ("projection", 2, 32, 4, 64, 300), ("projection", 1, 16, 2, 128, 900)]


@pytest.mark.parametrize("front,b,h,hk,d,cap", CHAINS)
def test_the_kernel_in_front_writes_the_last_row(front, b, h, hk, d, cap):
    """A chain of such kernels and attentions in one CUDA graph of programmatic launches, as in a captured decode step: each attention
    starts while the kernel in front of it is still to write.  Every position checked bit for bit against a call that waits."""
    g = torch.Generator(device="cuda").manual_seed(d)
    rn = lambda *size: torch.randn(*size, generator=g, device="cuda")
    cos, sin = rn(cap, d), rn(cap, d)
    k, v = (torch.zeros(b, hk, cap, d, device="cuda", dtype=torch.float16) for _ in "kv")
    rows = (h + 2 * hk) * d
    if front == "projection":
        qw, one = quantize.quantize_weight((rn(rows, 2048) * 0.03).half(), 128), torch.ones(2048, device="cuda").half()
        write = lambda x, pos: ops.int4_gemv_rope_kv(x, qw.packed, qw.scales, 128, cos, sin, pos, k, v, h, one, 1e-5)
    else:
        write = lambda x, pos: ops.rope_kv_write(x, cos, sin, pos, k, v, h)
    # tiles of 64 rows: the last row alone in its tile, last in it, in the first tile, past the ring, in each of the later splits
    steps = [i for i in range(cap) if i < 4 or (i % 64 in (0, 1, 63) and (i < 1300 or i > cap - 200 or i % 1024 < 2))] + [cap - 1]
    xs = [rn(b, 2048 if front == "projection" else rows).half() for _ in steps]
    poss = [torch.tensor([i], device="cuda") for i in steps]
    lens = [torch.full((b,), i + 1, dtype=torch.int32, device="cuda") for i in steps]

    want = []
    for x, pos, n in zip(xs, poss, lens):
        q = write(x, pos)
        torch.cuda.synchronize()
        want.append(ops.flash_attn_decode(q, k, v, n))
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), _capi.programmatic_launch(True), torch.cuda.graph(graph, stream=side):
        got = [ops.flash_attn_decode_step(write(x, pos), k, v, n) for x, pos, n in zip(xs, poss, lens)]
    for _ in range(3):
        k.zero_(), v.zero_(), [o.fill_(7.0) for o in got]
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert _capi.device_status(torch.device("cuda", 0)) == 0
