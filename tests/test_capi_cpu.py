"""CPU-side checks of the boundary: the C-ABI library loads and exports everything the header declares,
and the package's host logic (CPU-tensor quantiser, validators, custom-op registration) behaves like the
reference's (kernelforge/quantize.py, kernelforge/ops.py:171-302).  No kernel is launched here."""

import ctypes
import re
import glob

import numpy as np
import pytest
import torch

from conftest import ROOT, GOLDEN
from kernelforge import _capi, ops
from kernelforge import quantize as kq


def _declared_functions():
    text = (ROOT / "include" / "kfb200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(kfb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    names = _declared_functions()
    assert len(names) >= 10
    handle = ctypes.CDLL(str(ROOT / "kernel-forge_b200" / "kernelforge" / "libkfb200.so"))
    for name in names:
        assert hasattr(handle, name), f"{name} is declared in include/kfb200.h but not exported"
    assert sorted(_capi.exported_symbols()) == names  # the ctypes table binds exactly the header
    assert _capi.lib().kfb_version() >= 100
    assert _capi.lib().kfb_last_error() is not None


@pytest.mark.parametrize("path", sorted(glob.glob(str(GOLDEN / "quant_*.npz"))), ids=lambda p: p.split("/")[-1])
def test_cpu_tensor_quantizer_matches_reference_bits(path):
    z = np.load(path)
    group = int(z["group"])
    w = torch.from_numpy(z["w"])
    if "_f16" in path:
        w = w.half()
    elif "_bf16" in path:
        w = w.bfloat16()
    qw = kq.quantize_weight(w, group)
    assert np.array_equal(qw.packed.numpy(), z["packed"])
    assert np.array_equal(qw.scales.numpy().view(np.uint16), z["scales"].view(np.uint16))
    assert np.array_equal(kq.unpack_int4(qw.packed).numpy(), z["q"])
    assert np.array_equal(kq.dequantize(qw, torch.float32).numpy(), z["deq32"])
    assert np.array_equal(kq.dequantize(qw, torch.float16).numpy().view(np.uint16), z["deq16"].view(np.uint16))
    assert qw.nbytes == z["packed"].size * 4 + z["scales"].size * 2 and qw.shape == tuple(z["w"].shape)


def test_bit_layout_known_answer():
    q = torch.arange(0, 8, dtype=torch.int8).reshape(1, 8)
    word = kq.pack_int4(q).item() & 0xFFFFFFFF
    assert [(word >> (4 * i)) & 0xF for i in range(8)] == [8, 10, 12, 14, 9, 11, 13, 15]


def test_quantization_error_stats():
    g = torch.Generator().manual_seed(1)
    w = torch.randn(256, 1024, generator=g) * 0.02
    for group in (64, 128):
        qw = kq.quantize_weight(w, group)
        step = qw.scales.float().repeat_interleave(group, dim=1)
        assert ((kq.dequantize(qw, torch.float32) - w).abs() <= 0.5 * step + 1e-8).all()
        stats = kq.quantization_error(w, qw)
        assert stats["rel_fro_err"] < 0.15 and stats["bits_per_weight"] == pytest.approx(4 + 16 / group)


def test_quantizer_rejections():
    with pytest.raises(ValueError, match="not a multiple of group_size"):
        kq.quantize_weight(torch.randn(16, 200), 128)
    with pytest.raises(ValueError, match="group_size"):
        kq.quantize_weight(torch.randn(16, 256), 32)
    with pytest.raises(ValueError, match="2-D"):
        kq.quantize_weight(torch.randn(4, 16, 256), 128)
    with pytest.raises(ValueError, match=r"\[-8, 7\]"):
        kq.pack_int4(torch.full((1, 8), 9, dtype=torch.int8))
    with pytest.raises(ValueError, match="multiple of 8"):
        kq.pack_int4(torch.zeros(2, 12, dtype=torch.int8))


def test_validators_reject_cpu_tensors_like_the_reference():
    q = torch.randn(1, 2, 8, 64, dtype=torch.float16)
    with pytest.raises(ValueError, match="CUDA"):
        ops.flash_attn(q, q, q)
    with pytest.raises(TypeError, match="2-D fp16 CUDA tensor"):
        ops.int4_linear(torch.randn(2, 256).half(), torch.zeros(8, 32, dtype=torch.int32),
                        torch.ones(8, 2, dtype=torch.float16))
    with pytest.raises(ValueError, match="positive"):
        ops._resolve_scale(-1.0, 64)
    assert ops._resolve_scale(None, 64) == pytest.approx(0.125)


def test_custom_ops_registered_with_fakes():
    assert hasattr(torch.ops.kernelforge, "flash_attn") and hasattr(torch.ops.kernelforge, "int4_matmul")
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        q = torch.empty(2, 8, 16, 64, dtype=torch.float16, device="cuda")
        k = torch.empty(2, 2, 48, 64, dtype=torch.float16, device="cuda")
        assert torch.ops.kernelforge.flash_attn(q, k, k, True, 0.125).shape == q.shape
        x = torch.empty(3, 256, dtype=torch.float16, device="cuda")
        p = torch.empty(40, 32, dtype=torch.int32, device="cuda")
        s = torch.empty(40, 2, dtype=torch.float16, device="cuda")
        assert torch.ops.kernelforge.int4_matmul(x, p, s, 128).shape == (3, 40)


def test_prefill_workspace_covers_the_plan_with_and_without_the_causal_mask():
    """The bytes that kfb_flash_attn_ws_bytes reports are enough for the plan a call takes, causal or not (it is not told
    which); without a workspace the call is planned for no splits, not a split plan run unsplit.  Host logic."""
    import random
    lib = _capi.lib()

    def plan(shape, causal, ws):
        tiles, splits = ctypes.c_int(), ctypes.c_int()
        assert lib.kfb_flash_attn_plan(*shape, causal, ws, ctypes.byref(tiles), ctypes.byref(splits)) == 0
        return tiles.value, splits.value

    rng = random.Random(1)
    shapes = [(2, 1, 1, 3907, 3907, 64), (1, 8, 8, 1557, 1557, 128), (1, 12, 2, 509, 4093, 128)]
    for _ in range(3000):
        hk, n = rng.choice((1, 2, 4, 8)), int(2 ** rng.uniform(1, 13))
        shapes.append((rng.choice((1, 2, 3, 8)), hk * rng.choice((1, 2, 6, 8)), hk, n, n + rng.choice((0, 0, 300, 4000)), rng.choice((64, 128))))
    split = 0
    for shape in shapes:
        ws = lib.kfb_flash_attn_ws_bytes(*shape)
        for causal in (0, 1):
            best = plan(shape, causal, 1 << 60)
            assert plan(shape, causal, ws) == best, (shape, causal)
            assert plan(shape, causal, 0)[1] == 1
            split += best[1] > 1
    assert split > 100
    # 3907 queries of one head: with splits two tiles per CTA are best, without them one
    assert plan(shapes[0], 1, 1 << 60)[0] == 2 and plan(shapes[0], 1, 0) == (1, 1)


def test_every_decode_plan_fits_the_array_of_the_allocation_free_entry():
    """kfb_flash_attn_decode_noalloc has 2 MiB for partials: no plan needs more, over groups, keys and head dims.  A workspace is
    asked for only where partials are written, so most plans need none.  Host logic."""
    lib = _capi.lib()
    most, none, some = 0, 0, 0
    for d in (64, 128):
        for b in list(range(1, 80)) + [100, 148, 149, 300]:
            for h, hk in ((1, 1), (16, 1), (17, 1), (40, 1), (8, 2), (32, 4), (34, 2), (64, 8)):
                for nk in (1, 64, 449, 512, 1000, 1025, 2048, 4096, 5000, 16384, 65536, 131072, 1 << 20):
                    need = lib.kfb_flash_attn_ws_bytes(b, h, hk, 1, nk, d)
                    most, none, some = max(most, need), none + (need == 0), some + (need > 0)
    assert 0 < most <= 2 << 20
    assert some > 50 and none > some
    assert lib.kfb_flash_attn_ws_bytes(8, 32, 4, 1, 4608, 64) == 0      # a cluster of four
    assert lib.kfb_flash_attn_ws_bytes(1, 32, 4, 1, 16384, 64) > 0      # more than eight splits


def test_splits_that_write_partials_have_two_tiles_of_keys():
    """A shard's partials are gathered from all ranks and merged by a kernel: no split of less than two tiles, no pairs below 24 tiles and
    no threes below 12, unlike clusters.  Host logic."""
    lib = _capi.lib()
    split = 0
    for d in (64, 128):
        for groups in list(range(1, 76)):
            for tiles in range(1, 80):
                n = ctypes.c_int()
                nbytes = lib.kfb_flash_attn_decode_partial_bytes(groups, 8, 1, tiles * 64, d, ctypes.byref(n))
                assert nbytes == groups * n.value * 16 * (d + 2) * 4
                assert n.value == 1 or (n.value * 2 <= tiles and tiles >= {2: 24, 3: 12}.get(n.value, 8)), (d, groups, tiles, n.value)
                split += n.value > 1
    assert split > 2000


def test_no_kernel_asks_for_non_coherent_loads():
    """Kernels are resident while the one in front still writes (programmatic dependent launch): what they read has to go through
    coherent loads behind pdl_wait.  __ldg and ld.global.nc are taken to be invariant and may be moved above it."""
    found = []
    for src in sorted((ROOT / "kernel-forge_b200" / "csrc").iterdir()):
        code = re.sub(r"//[^\n]*", "", src.read_text())
        found += [f"{src.name}: {hit}" for hit in re.findall(r"__ldg\s*\(|ld\.global\.nc", code)]
    assert not found, found


def test_int4_matmul_routing_table():
    """Which kernel int4_linear / int4_matmul takes by shape (pure host logic, kfb_int4_linear_route), on both sides of each line."""
    gemv, stream, small, gemm = range(4)
    route = _capi.lib().kfb_int4_linear_route
    fp16, bf16 = (_capi.dtype_code(t) for t in (torch.float16, torch.bfloat16))
    for m, n, k, want in ((1, 8191, 2048, gemv), (1, 8192, 2048, small), (1, 75776, 2048, gemv), (8, 75776, 2048, gemv), (9, 75776, 2048, stream),
                          (16, 75776, 2048, stream), (17, 75776, 2048, gemm), (2, 5632, 2048, small), (16, 11264, 2048, small), (17, 11264, 2048, gemm),
                          (32, 2048, 8192, small), (32, 2049, 8192, gemm), (33, 256, 1024, gemm), (24, 1536, 8192, small), (25, 1536, 8192, gemm),
                          (25, 1537, 8192, small), (16, 1536, 12288, small), (17, 1024, 12288, gemm), (32, 1536, 8128, small)):
        assert route(m, n, k, fp16, 0) == want, (m, n, k)
    for m, n, k, want in ((1, 100, 2048, small), (1, 80000, 2048, small), (16, 80000, 1024, small), (17, 1536, 8192, gemm), (17, 1536, 8128, small),
                          (17, 1537, 8192, small), (33, 64, 64, gemm)):
        assert route(m, n, k, bf16, 0) == want, (m, n, k)
    assert route(8, 75776, 2048, fp16, 1) == small      # the streaming kernels have no bias to add
    assert route(0, 64, 64, fp16, 0) < 0
    assert ops.GEMV_MAX_M == 8 and ops.SMALL_BATCH_MAX_M == 32 and ops.PREPACKED_GEMV_MAX_M == 32


def test_decoder_refuses_steps_that_do_not_fit_the_cache():
    """Host-side position check of the end-to-end decoder (the step graph reads the position on the device, so the
    host must make sure a replay is never asked to write past the KV cache).  Nothing is launched: built on CPU."""
    from kernelforge.llama_decode import LlamaInt4Decoder, LlamaShape
    shape = LlamaShape(hidden=128, layers=1, heads=2, kv_heads=1, head_dim=64, intermediate=128, vocab=64)
    dec = LlamaInt4Decoder.random_init(shape, "cpu", batch=1, max_len=8)
    with pytest.raises(ValueError, match="no room"):
        dec.prefill(torch.zeros(1, 8, dtype=torch.long))          # a prompt as long as the cache
    dec._host_pos = 6                                             # as after a 6-token prompt
    with pytest.raises(ValueError, match="do not fit"):
        dec.decode(3)
    dec._host_pos = 8
    with pytest.raises(ValueError, match="full"):
        dec.capture()


@pytest.mark.parametrize("n_rows,k,group", [(2560, 2048, 128), (2048, 2048, 128), (11264, 2048, 128), (2048, 5632, 128),
                                            (32000, 2048, 0), (512, 256, 128), (1024, 256, 64), (320, 256, 0)])
@pytest.mark.parametrize("n_ctas", [148, 132, 7])
def test_persistent_step_schedule_covers_every_row_once(n_rows, k, group, n_ctas):
    """kfb_decode_step_slice (host only): the row slices of the CTAs tile the matrix without gap or overlap, start on the
    16-byte boundaries the bulk copies need (weights and scales), and a ring slot's worth of rows fits its 44 KB."""
    import ctypes
    from kernelforge import _capi
    lib = _capi.lib()
    r0, rows, rpc = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    nxt = 0
    row_w = k // 2 if group else k * 2
    row_s = (k // group) * 2 if group else 0
    for cta in range(n_ctas):
        _capi.check(lib.kfb_decode_step_slice(n_rows, k, group, 0, cta, n_ctas, ctypes.byref(r0), ctypes.byref(rows), ctypes.byref(rpc)))
        assert r0.value == nxt and rows.value >= 0
        nxt += rows.value
        assert (r0.value * row_w) % 16 == 0 and (r0.value * row_s) % 16 == 0
        assert rpc.value >= 1 and rpc.value * (row_w + row_s) <= 45056
        if group:
            assert rows.value % 2 == 0 and rpc.value % 2 == 0      # pairs of rows stay together
            assert (rpc.value * row_s) % 16 == 0
    assert nxt == n_rows


def test_prepack_shape_rules_and_routing_rule():
    """Host-side rules of the private prepacked weight cache: which shapes get a fragment-order copy, and where the
    measured M = 1 exception applies (small N with long K stays on the public-format kernel)."""
    import torch
    from kernelforge import ops
    ok = lambda n, k: ops.prepack_supported(torch.empty(n, k // 8, dtype=torch.int32))
    assert ok(5632, 2048) and ok(16, 64) and ok(1536, 8960) and ok(32000, 2048)
    assert not ok(5630, 2048)        # N % 16
    assert not ok(64, 96)            # K % 64
    assert not ok(64, 12288 + 64)    # a warp's share of K must fit its registers
    assert not ops.prepack_supported(torch.empty(8, dtype=torch.int32))
    assert ops._prepacked_wins(2, 1536, 8960) and ops._prepacked_wins(32, 256, 1536)
    assert ops._prepacked_wins(1, 5632, 2048) and not ops._prepacked_wins(1, 1536, 8960)
    with pytest.raises(ValueError):
        ops.prepack_int4(torch.empty(64, 8, dtype=torch.int32))   # not on a CUDA device: no CPU fallback


def test_private_row_orders_are_permutations_prefill_can_undo():
    """ops.interleave_qkv_for_rope / interleave_gate_up only permute rows: the projection of the permuted matrix, read back
    the way LlamaInt4Decoder.prefill and _mlp read it, equals the projection of the natural matrix (pure torch, on CPU)."""
    import torch
    from kernelforge import ops
    g = torch.Generator().manual_seed(0)
    h, hk, d, k, inter, b, t = 4, 2, 64, 96, 40, 2, 3
    wq, wk, wv = (torch.randn(n, k, generator=g, dtype=torch.float64) for n in (h * d, hk * d, hk * d))
    x = torch.randn(b, t, k, generator=g, dtype=torch.float64)
    nat = x @ torch.cat([wq, wk, wv], 0).T
    qkv = x @ ops.interleave_qkv_for_rope(wq, wk, wv, d).T
    nq, nkv = h * d, hk * d
    unpair = lambda z, heads: z.reshape(b, t, heads, d // 2, 2).transpose(-1, -2).reshape(b, t, heads * d)
    back = torch.cat([unpair(qkv[..., :nq], h), unpair(qkv[..., nq:nq + nkv], hk), qkv[..., nq + nkv:]], -1)
    assert torch.equal(back, nat)
    # the pair (2j, 2j + 1) of a q / k head holds features (j, j + D/2): what the rotate-half embedding mixes
    perm = ops.interleave_qkv_for_rope(torch.arange(h * d, dtype=torch.float64)[:, None], torch.zeros(hk * d, 1, dtype=torch.float64),
                                       torch.zeros(hk * d, 1, dtype=torch.float64), d)[:h * d, 0].reshape(h, d // 2, 2)
    assert torch.equal(perm[..., 1] - perm[..., 0], torch.full((h, d // 2), float(d // 2), dtype=torch.float64))
    gate, up = (torch.randn(inter, k, generator=g, dtype=torch.float64) for _ in range(2))
    gu = (x @ ops.interleave_gate_up(gate, up).T).view(b, t, inter, 2)
    assert torch.equal(gu[..., 0], x @ gate.T) and torch.equal(gu[..., 1], x @ up.T)


def test_every_role_of_the_gemm_waits_for_the_cluster_once():
    """int4_gemm_kernel arrives on the cluster barrier before its roles part: each role has to wait for that phase before the
    arrive of the teardown (two arrives in a row are not defined).  Read from the source: no run shows it."""
    code = re.sub(r"//[^\n]*", "", (ROOT / "kernel-forge_b200" / "csrc" / "int4_gemm.cu").read_text())
    code = code[code.index("int4_gemm_kernel("):]
    first = code.index("cluster_arrive();")
    roles, teardown = code[first:code.index("cluster_arrive_relaxed();")], code[code.index("cluster_arrive_relaxed();"):]
    assert roles.count("cluster_arrive") == 1 and teardown.index("cluster_wait();") > 0
    inner = roles[roles.index("if (warp >= kProducerWarp) {"):]
    producer, rest = inner.split("} else if (warp == kMmaWarp) {", 1)
    mma, rest = rest.split("} else {\n      cluster_wait();", 1)       # the filling warps
    dequant, epilogue = rest.split("} else if (warp < kDequantWarps) {", 1)[1].split("} else {\n", 1)
    assert producer.count("cluster_wait();") == 1 and mma.count("cluster_wait();") == 1
    assert dequant.count("cluster_wait();") + epilogue.count("cluster_wait();") == 3   # (dequantise: at its first block, or at the end)


@pytest.mark.parametrize("call", ["flash_attn", "flash_attn_kv_view"])
def test_attention_refuses_tensors_of_different_devices(call):
    """The native path declines them; what stands behind it has to raise, not to return None."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode(allow_non_fake_inputs=True):
        q, k = (torch.empty(1, 2, 16, 64, dtype=torch.float16, device=f"cuda:{i}") for i in (0, 1))
        with pytest.raises(ValueError, match="same CUDA device"):
            getattr(ops, call)(q, k, k)


def test_where_a_decode_step_has_its_norms_in_the_projections():
    """kfb_int4_norm_fits (148 SMs without a GPU) and the decoder's use of it: hidden sizes and widths on both sides of the lines."""
    from kernelforge.llama_decode import LlamaInt4Decoder, LlamaShape
    fits = _capi.lib().kfb_int4_norm_fits
    for m, n, k, group, want in ((1, 11264, 2048, 128, 1), (2, 11840, 2048, 128, 1), (1, 11841, 2048, 128, 0), (1, 16384, 2048, 128, 0),
                                 (1, 22016, 2048, 128, 1), (1, 4736, 4096, 128, 1), (1, 4752, 4096, 128, 0), (3, 256, 2048, 128, 0),
                                 (1, 256, 2048, 96, 0), (1, 256, 100, 64, 0), (0, 256, 2048, 128, 0)):
        assert fits(m, n, k, group) == want, (m, n, k, group)

    def fused(hidden, intermediate):
        shape = LlamaShape(hidden=hidden, layers=1, heads=hidden // 64, kv_heads=1, head_dim=64, intermediate=intermediate, vocab=16)
        return LlamaInt4Decoder.random_init(shape, "cpu", batch=1, max_len=4).fused

    assert fused(1536, 256) and not fused(1408, 256) and not fused(2176, 256)
    assert not fused(1536, 6016)     # 12032 gate and up rows: a second wave of CTAs, nearly empty


def test_decode_attention_waits_for_its_copies_before_it_reuses_their_ring():
    """After an expired wait copies may still be in flight: they get time to land before the ring becomes the scratch of the merge
    and the CTA leaves.  Read from the source: a run would need a wait that expires in mid-copy."""
    code = re.sub(r"//[^\n]*", "", (ROOT / "kernel-forge_b200" / "csrc" / "attn_decode.cu").read_text())
    kernel = code[code.index("attn_decode_kernel("):code.index("attn_decode_merge_kernel(")]
    consumed, merge = kernel.split("float* scratch", 1)
    for wait in ("if (!mbar_wait(&empty[s]", "if (!ok)"):     # the producer's wait and the consumers'
        assert consumed.count(wait) == 1
        expired = consumed[consumed.index(wait):]
        assert "let_copies_land();" in expired[:expired.index("break;")]
    assert consumed.count("break;") == 2      # no other way out of the loops
    helper = code[code.index("void let_copies_land()"):]
    assert "200000ull" in helper[:helper.index("\n}")]


def test_prefill_refuses_ids_that_are_no_indices():
    from kernelforge.llama_decode import LlamaInt4Decoder, LlamaShape
    shape = LlamaShape(hidden=128, layers=1, heads=2, kv_heads=1, head_dim=64, intermediate=128, vocab=64)
    dec = LlamaInt4Decoder.random_init(shape, "cpu", batch=1, max_len=8)
    for ids in (torch.ones(1, 4), torch.ones(1, 4, dtype=torch.int16), torch.tensor([[1, 64]]), torch.tensor([[0, -65]])):
        with pytest.raises(IndexError):
            dec.prefill(ids)
