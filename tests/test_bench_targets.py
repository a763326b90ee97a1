"""bench.py's targets block: each benchmark target with the figure a run
measured, and whether it is met (host logic only, no GPU)."""
import sys

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402


def line_with(copy_gbs, gather_perm_ratio, batch_ratio):
    line = {"peak_gbs": 6661.0,
            "kernels": [{"kernel": f"copy_exit_warp_{w}B", "gbs": g} for w, g in ((4, copy_gbs), (64, 7100.0))]}
    subs = {"gather": {"reference_gpu": {"ratio": 1.04, "ratio_by_pattern": {"perm": gather_perm_ratio}},
                       "ceiling": {"this_frac_perm_min": 0.99, "this_frac_perm_mean": 1.0}},
            "batch": {"details": {"batched_vs_per_call": batch_ratio}}}
    return line, subs


def test_targets_met_and_not_met():
    t = bench.targets(*line_with(6900.0, 1.02, 1.91))
    assert t["copy_at_85pct_of_hbm_peak_4_64B"]["met"] is True
    assert t["copy_at_85pct_of_hbm_peak_4_64B"]["slowest_kernel_gbs"] == 6900.0
    assert t["random_gather_1p2x_reference"]["met"] is False
    assert t["random_gather_1p2x_reference"]["frac_of_random_block_ceiling_perm"]["this_frac_perm_min"] == 0.99
    assert t["batched_2x_per_call"] == {"ratio": 1.91, "met": False}
    t = bench.targets(*line_with(6700.0, 1.25, 2.02))
    assert t["copy_at_85pct_of_hbm_peak_4_64B"]["met"] is False  # 6700 < 0.85 * 8000
    assert t["random_gather_1p2x_reference"]["met"] is True
    assert t["batched_2x_per_call"]["met"] is True


def test_targets_skip_what_did_not_run():
    line, _ = line_with(6900.0, 1.0, 2.0)
    t = bench.targets(line, {})
    assert set(t) == {"copy_at_85pct_of_hbm_peak_4_64B"}


def test_result_line_can_be_read_back():
    """The printed line keeps every contract key and stays short however many kernels
    and sub-records were measured."""
    import json
    contract = {"metric": "m", "value": 1.0, "unit": "GB/s", "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 2.0,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
                "config": {"workload": "sweep", "structs_per_width": {str(k): 1 << 20 for k in range(16)}},
                "e2e": {"value": 1.0, "unit": "GB/s", "h2d_bytes_per_step": 5, "d2h_bytes_per_step": 8},
                "gpu_launches": 640, "clocks": {"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": []}}
    kernels = [{"kernel": f"copy_exit_warp_{w}B", "gbs": 7000.0, "launches": 20} for w in range(4, 65, 4)] * 20
    sub = {"value": 2.0, "ms_per_step": 1.0, "bit_exact": True, "kernels": kernels, "details": {"x": kernels}}
    line = dict(contract, peak_gbs=6691.5, kernels=kernels, cpu_baseline={"value": 1.0, "unit": "GB/s", "sample": "s" * 900},
                roofline={"bound": "hbm", "achieved": 1.0, "basis": "b" * 900},
                details={"configs": {n: sub for n in ("gather", "batch", "serve", "layout", "copy12")}})
    line["details"]["targets"] = bench.targets(line, {"batch": {"details": {"batched_vs_per_call": 1.8}}})
    out = json.dumps(bench.summary(line))
    back = json.loads(out)
    assert len(out) <= bench.SUMMARY_LIMIT
    for k, v in contract.items():
        assert back[k] == ({"workload": "sweep"} if k == "config" else v), k
    assert back["targets"]["batched_2x_per_call"] == {"ratio": 1.8, "met": False}
    assert back["configs"]["gather"]["value"] == 2.0
