"""The bench line (CPU only): it holds the contract's keys and every leg's
figures, and stays short enough to be kept whole in a log's last 3000
characters."""
import json

import bench

X = 1234.5678901234567  # a float of full length wherever a measurement stands


def _full():
    timed = {"ms": X, "gbs": X, "frac": 0.98765432109876}
    ntt = {f"2^{k}": {d: {**timed, "reference": {"ms": X}} for d in ("evaluate", "interpolate")} for k in (20, 24, 28)}
    ntt["batch_10x2^22"] = {"evaluate_vortex": timed, "interpolate_vortex": timed, "values_equal": True}
    kernels = {"log_n": 26, "reps": 5, "fri_chain_committed": {"ms": X, "layers": 25, "frac_of_probe": 0.9}}
    for name, legs in (("merkle_commit_m31", ("vortex", "vortex_fused_tree")), ("fri_fold_qm31_to_2", ("vortex",)),
                       ("bit_reverse", ("qm31_vortex", "m31_2^28_vortex", "permute_m31_2^28_vortex")),
                       ("stwo_ntt", ("single_2^24_evaluate_vortex", "single_2^24_interpolate_vortex",
                                     "batch16_2^20_evaluate_vortex", "batch16_2^20_interpolate_vortex")),
                       ("zero_pad", ("vortex",)), ("fibonacci_quotient", ("vortex",)), ("twiddle_tables", ("vortex",)),
                       ("stwo_poly_ops", ("eval_at_point_2^26_vortex", "barycentric_2^24_vortex"))):
        kernels[name] = {leg: timed for leg in legs} | {"values_equal": name != "zero_pad"}
    point = {"proofs_per_s": X, "p50_ms": X, "p99_ms": X, "rate": X, "by_log_n": {str(k): timed for k in range(5)}}
    stages = ("trace", "interpolate", "lde_evaluate", "trace_commit", "quotient_commit", "circle_fold_commit",
              "line_folds_commit", "queries", "decommit")
    return {
        "metric": bench.METRIC, "value": X, "unit": "proofs/s", "n_gpus": 8, "steps": 1000, "warmup": 100,
        "ms_per_step": X, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32 (M31)",
        "data": "synthetic (seeded SplitMix64 public inputs)",
        "config": {"workload": "fibonacci_stark log_n=24 blowup=4 queries=80 (2^26-point LDE)", "stream": "x" * 200,
                   "log_n": 24, "blowup_bits": 2, "n_queries": 80, "parallelism": "replicas x8",
                   "in_flight": "4 proofs per GPU (4 slots on 4 streams)",
                   "l2": "per-step working set > L2 (LDE 256 MiB + FRI layers 1024 MiB); no flush needed"},
        "e2e": {"value": X, "unit": "proofs/s", "h2d_bytes_per_step": 8, "d2h_bytes_per_step": 1994344,
                "api": "vx_prove_fib_batch (ProverPipeline::prove_batch) over the timed inputs"},
        "value_one_in_flight": X, "p50_ms": X, "p99_ms": X, "latency_api": "vx_prove_fib", "lde_hbm_gbs": X,
        "roofline": {"bound": "int-alu", "kernel": "trace commitment: leaf_subtree_kernel<LeafM31>", "achieved": X,
                     "peak": X, "unit": "G compressions/s", "frac": X, "frac_of_nominal": X, "traffic": 6.1490e8,
                     "traffic_source": "x" * 300},
        "lde_roofline": {"bound": "hbm", "peak": X, "frac": X, "traffic": 1.81426e9, "traffic_source": "x" * 300},
        "stages_ms": {k: X for k in stages}, "stage_rooflines": {k: timed for k in stages},
        "gpu_launches": 50000, "launches_per_proof": 51,
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 1000},
        "autotune": {"ntt_plan": {str(k): [10, 6] for k in range(13, 29)}},
        "ntt_microbench": ntt, "kernel_microbench": kernels,
        "pow_grind": {"ms": X, "valid": True, "candidates_per_s": 2.78036464e10, "frac_of_probe": X, "note": "x" * 200},
        "batched_commit": {"value": X, "value_one_in_flight": X, "e2e": {"value": X, "contexts_bytes_equal": True}},
        "served": {"plain_capacity_per_s": X, "served_sweep": [point] * 11, "plain_sweep": [point] * 7,
                   "speedup_at_equal_p99": {"a": 1.12579664893, "b": 1.11144573279, "c": None}},
        "cpu_baseline": {"value": X, "unit": "proofs/s", "cores": 16, "kind": "port",
                         "sample": "one full log_n=24 proof (2^26-point LDE, 80 queries)"},
    }


def test_the_line_is_short_and_whole():
    full = _full()
    line = bench.summary_line(full)
    assert len(json.dumps(line, separators=(",", ":"))) < 2900 < len(json.dumps(full)) / 4
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "cpu_baseline"):
        assert k in line
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(line["e2e"])
    assert {"sm_mhz", "sm_max_mhz", "reasons"} <= set(line["clocks"])
    assert abs(line["value"] / full["value"] - 1) < 1e-5
    assert line["kernels"]["ntt_2^24_e"] == [1235.0, 0.988] and "twiddle_tables" in line["kernels"]
    assert line["served"] == {"plain_capacity": 1234.57, "engine_peak": 1234.57,
                              "ratio_at_equal_p99": [1.1258, 1.11145, None]}
    assert line["outputs_equal"] == "10/11"  # the planted false flag shows


def test_the_line_without_the_optional_legs():
    full = _full()
    for k in ("ntt_microbench", "kernel_microbench", "pow_grind", "batched_commit", "served", "cpu_baseline"):
        del full[k]
    line = bench.summary_line(full)
    assert "kernels" not in line and "served" not in line and line["value"]
