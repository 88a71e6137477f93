"""bench.py's result line: complete, parseable and short, however long the breakdown is; its kernels and their
traffic are the present ones."""
import json
import sys

from conftest import ROOT


def record():
    """A record of the shape that a default run builds: 20 updates, six forms, a CPU baseline on 16 cores."""
    rows = [0.123456789012345678] * 20
    form = {"method": "dg", "updates": 20, "ms": 1e4 / 3, "krylov": [205] * 20, "rms": rows, "damping": rows,
            "timers_all_unit_updates": {n: {"ms": 1 / 3, "launches": 1000} for n in "abcdefg"}}
    per = {m: {"proxy_seconds_per_update": rows[:16], "krylov": [205], "updates_per_s_at_workload": 1 / 3} for m in ("dg", "hdg")}
    host = {"nproc": 16, "cpu_model": "Intel(R) Xeon(R) Processor", "mem_available_gb": 207.974887424}
    run = {"value": 1 / 7, "processes": 16, "per_method": per, "cell_ratio": 256.0, "wall_s": 27.3, "host": host}
    forms = [f"{m}_{p}" for m in ("dg", "hdg") for p in ("fp64", "mixed", "mixed16", "mixed32")]
    return {"metric": "m" * 80, "value": 2 / 3, "unit": "updates/s", "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 1e3 / 3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "d" * 160, "data": "synthetic",
            "config": {"workload": "w" * 300, "parallelism": "replicas x1", "l2": "l" * 80, "value_definition": "v" * 150},
            "roofline": {"bound": "hbm", "achieved": 5e3 / 3, "peak": 6550.1, "unit": "GB/s", "frac": 5 / 7, "traffic": 1e10 / 3,
                         "traffic_source": "t" * 160, "kernel": "k" * 90, "peak_source": "measured"},
            "gpu_launches": 123456, "with_forcing_floor": {"value": 2 / 3, "forms": forms[:2]},
            "headline_forms": {"dg": "f" * 120, "hdg": "f" * 120}, "speedup_vs_fp64": {f: 4 / 3 for f in forms},
            "rel_error_vs_fp64": {f: 1e-13 / 3 for f in forms}, "krylov_change_vs_fp64": {f: 3 for f in forms},
            "per_method_updates_per_s": {f: 4 / 3 for f in forms}, "breakdown": {f: form for f in forms},
            "clocks": {"sm_mhz": 1642.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]},
            "e2e": {"value": 2 / 3, "unit": "updates/s", "h2d_bytes_per_step": 169869312, "d2h_bytes_per_step": 169869312},
            "cpu_baseline": {"value": 1 / 7, "unit": "updates/s", "cores": 16, "kind": "port", "sample": "s" * 500,
                             "single_thread": {"value": 1 / 9, "unit": "updates/s", "cores": 1, "per_method": per},
                             "all_core": run}}


def test_result_line_is_short_and_complete():
    sys.path.insert(0, str(ROOT))
    import bench

    full = record()
    text = bench.result_line(full)
    line = json.loads(text)
    assert len(text) <= 8000 and "\n" not in text and "breakdown" not in line
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
                "dtype", "data", "config", "roofline", "gpu_launches", "clocks", "e2e", "cpu_baseline"):
        assert key in line, key
    assert abs(line["value"] - full["value"]) < 1e-9 and line["e2e"]["h2d_bytes_per_step"] == 169869312
    assert line["cpu_baseline"]["cores"] == 16 and line["cpu_baseline"]["single_thread"]["cores"] == 1


def test_roofline_names_kernels_that_exist():
    """Each DG form's solve is a kernel of the sources, with DRAM bytes from a committed capture: 1.0 to 1.1 times
    the algorithmic bytes."""
    import re
    import types

    sys.path.insert(0, str(ROOT))
    import bench

    sources = "".join(p.read_text() for p in (ROOT / "dg_hdg_euler_cpp_b200" / "csrc").glob("*.cu*"))
    args = types.SimpleNamespace(k=8, nx=64)
    for form in ("fp64", "mixed", "mixed16", "mixed-af", "mixed16-af"):
        label = bench.solve_kernel(form)
        assert re.search(r"^" + re.escape(label.split("<")[0]) + r"\(", sources, re.M), label
        traffic, source = bench.solve_traffic(args, label)
        assert 1.0 < traffic / bench.algorithmic_bytes("dg", 324, 4096, 36, 8192, 144, form) < 1.1, form
        assert (ROOT / re.search(r"profiles/\S+\.md", source).group()).is_file(), source
