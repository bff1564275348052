"""bench.py's line for stdout stays within what a reader of a job's last 3,000
characters gets whole, and parses."""
import json

import bench


def _record(n):
    """A workload's record of 4 KB with the keys the line takes from it."""
    return {"value": 41.22158379764565, "unit": "solves/s", "ms_per_step": 24.259135818481447,
            "e2e": {"value": 26.63723075088289, "unit": "solves/s", "includes": "x" * 500},
            "solve": {"true_rel_resid": 5.1986599952168e-07, "mixed_speedup_vs_plain_fp64_early_exit": 24.22434779},
            "config": {f"key{i}": "x" * 100 for i in range(n)}}


def test_the_line_is_short_and_whole():
    out = {"metric": bench.METRIC, "value": 228.7654321012345, "unit": "Mpts/s", "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 4.58365432101234, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f32", "data": "synthetic",
           "config": {"workload": bench.WORKLOAD, "n_points": 1048576, "expansion_order": 8, "leaf_size": 64,
                      "mac_theta": 0.5, "n_nodes": 37449, "n_p2p_pairs": 4569952, "n_m2l_pairs": 30573626,
                      "p2p_interactions": 4703102028, "l2": "flushed by a 256 MiB write between steps",
                      "parallelism": "replicas x1", "rel_l2_vs_fp64_direct_256_targets": 4.6226838958422785e-07},
           "e2e": {"value": 160.54131741574656, "unit": "Mpts/s", "h2d_bytes_per_step": 4194304,
                   "d2h_bytes_per_step": 4194304, "ms_per_step": 6.531502399999312},
           "gpu_launches": 320, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 2},
           "roofline": {"kernel": "k" * 40, "achieved": 34.937730099849404, "traffic_note": "n" * 80,
                        "peak_source": "p" * 80},
           "stages_ms": {k: 2.637123456789012 for k in ("p2m", "m2m", "m2l", "l2l", "p2p")},
           "p2p_tflops": 54.123456789012345,
           "cpu_baseline": {"value": 0.07309530929679621, "unit": "Mpts/s", "cores": 16, "kind": "port",
                            "sample": "s" * 120}}
    recs = {k: _record(30) for k in ("torus_solve", "sphere_solve", "batch_solve")}
    recs["warm_start"] = {"error": "e" * 400}
    text = json.dumps(bench.headline(out, recs))
    line = json.loads(text)
    assert len(text) <= 2900
    for key in out:
        assert key in line
    assert abs(line["value"] / out["value"] - 1) < 1e-5 and line["n_gpus"] == 1 and line["steps"] == 20
    assert line["workloads"]["torus_solve"]["value"] == 41.2216
    assert bench.headline(out, {}).keys() == out.keys()
