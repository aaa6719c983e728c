"""bench.py prints one JSON line that survives a reader who keeps only the last 3000 characters of the output.  Host logic."""

import json
import sys

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402


def record(bound, **extra):
    roof = {"bound": bound, "achieved": 1234.56789012, "peak": 6543.21, "unit": "GB/s", "frac": 0.123456789, "traffic": None,
            "peak_source": "measured HBM copy", "note": "x" * 80}
    return dict({"us_per_call": 12.3456789, "gbs": 1234.56789, "tflops": 123.456789, "bytes": 123456789, "roofline": roof,
                 "cpu_baseline": {"value": 1.23456789, "sample": "y" * 150}}, **extra)


def test_the_printed_line_is_short_and_complete():
    also = {"c1_int4_linear_m1_5632x2048": record("hbm")}
    also.update({f"c1_stream_m{m}_{n}x2048": record("hbm") for m, n in ((1, 180224), (1, 720896), (8, 720896))})
    also["c2_flash_attn_causal_b2_h16_n2048_d64"] = record("tensor")
    also["c2_sweep_b2_h16"] = {f"n{n}_d{d}_{c}": {"tflops": 1098.7654, "ms_per_step": 0.1, "frac": 0.6} for n in (512, 1024, 2048, 4096, 8192)
                               for d in (64, 128) for c in ("full", "causal")}
    also["c3_gqa_prefill_b1_hq32_hkv4_n2048_d64_causal"] = record("tensor")
    also.update({f"c3_decode_attn_b{b}_nk{nk}": record("hbm") for b, nk in ((1, 4096), (8, 4096), (64, 4096), (8, 16384))})
    also.update({f"c4_{name}_{n}x{k}_m{m}": record("tensor" if m >= 128 else "hbm", N=n, K=k, M=m)
                 for name, (n, k) in bench.QWEN_SHAPES.items() for m in (1, 16, 128, 1024)})
    also.update({f"c5_decode_e2e_tinyllama_arch_b{b}": record("hbm", tok_per_s=12345.678) for b in (1, 8)})
    also["c5_decode_e2e_tinyllama_arch_b32"] = {"error": "RuntimeError: " + "z" * 300}
    short = bench.brief(also)
    text = json.dumps(short, separators=(",", ":"))
    assert len(text) < 1400 and json.loads(text) == short
    assert short["c1_m1_5632x2048"] == [1230.0, 0.123] and short["c5_dec_e2e_b8"][0] == 12300.0 and "z" in short["c5_dec_e2e_b32"]


def test_rounding_keeps_whole_numbers_and_structure():
    assert bench.digits({"a": [1.23456789, 7, None, "s"], "b": {"c": 123456789}, "d": True}, 3) == {"a": [1.23, 7, None, "s"], "b": {"c": 123456789},
                                                                                                  "d": True}
