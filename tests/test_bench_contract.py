"""The benchmark's reference arm runs without a GPU: one JSON line on standard output with the keys the contract names."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEYS = {"impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
        "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"}


def _run(*args):
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0", *args],
                       capture_output=True, text=True, cwd=ROOT, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.strip()]
    assert len(lines) == 1, r.stdout          # exactly one line on standard output
    return json.loads(lines[0])


@pytest.mark.parametrize("workload,metric,unit", [("c4", "whisper_large_v3_w4a16_rtfx", "RTFx"), ("c1", "linearq_w4a16_gemm_throughput", "TFLOP/s")])
def test_reference_arm_line(workload, metric, unit):
    d = _run("--workload", workload)
    assert KEYS <= set(d)
    assert d["impl"] == "reference" and d["metric"] == metric and d["unit"] == unit and d["value"] > 0
    cb = d["cpu_baseline"]
    assert cb["kind"] in ("reference", "port") and cb["cores"] >= 1 and cb["sample"] and cb["value"] == d["value"]
    assert d["e2e"] == {"value": d["value"], "unit": unit, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
    assert d["vs_baseline"] is None and d["higher_is_better"] is True and d["config"]["workload"].startswith(workload + ":")


def test_reference_arm_maps_nothing_of_this_library():
    """The arm that the library is compared with imports none of it: no module of the package, none of its shared objects."""
    code = ("import os, runpy, sys\n"
            "sys.argv = ['bench.py', '--impl', 'reference', '--workload', 'c1', '--steps', '1', '--warmup', '0']\n"
            "runpy.run_path('bench.py', run_name='__main__')\n"
            "mapped = {l.split()[-1] for l in open('/proc/self/maps') if 'asrq_b200' in l}\n"
            "named = [m for m in sys.modules if m.split('.')[0] == 'asrq_b200']\n"
            "assert not mapped and not named, (mapped, named)\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def test_ours_arm_refuses_to_run_without_a_gpu():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--steps", "1"], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode != 0 and "no CPU fallback" in (r.stderr + r.stdout)
