"""bench.py's line: everything that the contract asks for, short enough for a reader that keeps the last few
kilobytes of the output, and the launch count of the path that a batch takes."""
import importlib.util
import json
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _full():
    x = 123456.78901234567
    rates = {"tc": x, "dp4a": x, "int32": x, "unit": "encaps+decaps/s"}
    stages = {"enc": dict.fromkeys(("prologue", "sa_product", "final_hash"), x),
              "dec": dict.fromkeys(("w_decode", "prologue", "sa_product", "final_hash"), x)}
    level = {"load": 0.5, "p50_ms": x, "p99_ms": x, "ops_per_s": x}
    return {
        "metric": "KEM encaps+decaps/sec at batch 8192 (int8 TC vs dp4a, bit-exact); p99 latency", "value": x,
        "unit": "encaps+decaps/s", "n_gpus": 8, "steps": 1000, "warmup": 100, "ms_per_step": x, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u8xs8->s32 (tcgen05 kind::i8), u64 Keccak lanes",
        "data": "synthetic (seeded SHAKE256 coins, keypairs generated on the GPU)",
        "config": {"workload": "w" * 90, "scheme": "s" * 20, "l2": "l" * 80, "parallelism": "p" * 40, "form": "tc",
                   "batch_per_gpu": 8192, "global_batch": 65536},
        "bit_exact_roundtrip": True, "gpu_launches": 9000, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0,
                                                                       "reasons": ["sw_power_cap"], "samples": 12, "power_w_max": x},
        "roofline": {"kernel": "k" * 80, "bound": "int", "unit": "Gop/s", "achieved": x, "peak": x, "frac": x,
                     "avg_launch_ms": x, "algorithmic": "a" * 200},
        "stage_run": "r" * 60, "stage_ms": stages, "tensor": {"pad": "t" * 4000},
        "e2e": {"value": x, "unit": "encaps+decaps/s", "h2d_bytes_per_step": 513605632, "d2h_bytes_per_step": 129368064,
                "roundtrip_ok": True, "pcie_gbs": {}},
        "cpu_baseline": {"value": x, "unit": "encaps+decaps/s", "cores": 192, "kind": "port", "sample": "s" * 300},
        "forms": {**rates, "tc_over_dp4a": x, "product_stage_tc_over_dp4a": x, "product_only_tc_over_dp4a": x},
        "frodo976aes_batch8192": rates, "frodo976_shared_key_batch8192": rates, "saber_l3_batch4096": rates,
        "single_request": {k: {"default": {"enc_ms": x, "dec_ms": x}} for k in ("frodo976", "saber_l3")},
        "mixed_16384": {"tc": x, "tc_eager": x, "tc_bit_exact": True},
        "serving": {"pad": "p" * 8000, "service": {"note": "n", **{f: {"peak_ops_per_s": x, "levels": [level], "bit_exact": True}
                                                                    for f in ("tc", "dp4a")}}},
        "frames_16384": {"frames_run": {"ops_per_s": x}, "ring_external_process": {"ops_per_s": x}},
        "peaks_file": "measured"}


def test_headline_is_short_and_whole():
    b, full = _bench(), _full()
    out = b.headline(full)
    text = json.dumps(out)
    assert len(text) < 2900
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches"):
        assert k in out, k
    assert out["value"] == 123457.0 and out["e2e"]["h2d_bytes_per_step"] == 513605632
    # without the secondary sections
    for k in ("forms", "serving", "frames_16384", "cpu_baseline", "e2e", "mixed_16384"):
        full.pop(k)
    assert json.loads(json.dumps(b.headline(full)))["metric"]


def test_launches():
    b = _bench()
    assert b.launches_per_step(True, 8192) == 9 and b.launches_per_step(True, 1024) == 7
    assert b.launches_per_step(True, 1025) == 9 and b.launches_per_step(False, 8192) == 7
