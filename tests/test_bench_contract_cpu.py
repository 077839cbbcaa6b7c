"""The reference arm of bench.py needs no GPU: it must run here and print one JSON line with the
keys the harness reads; under a multi-rank launch only rank 0 prints."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(extra_env=None):
    env = dict(os.environ, **(extra_env or {}))
    cmd = [sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--workload", "zipf",
           "--steps", "2", "--warmup", "1"]
    return subprocess.run(cmd, capture_output=True, text=True, env=env, cwd=ROOT, timeout=300)


def test_reference_arm_prints_the_contract_line():
    res = _run()
    assert res.returncode == 0, res.stderr[-2000:]
    line = json.loads(res.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["metric"] == "spmm_gflops" and line["unit"] == "GFLOP/s"
    assert line["higher_is_better"] is True and line["steps"] == 2 and line["warmup"] == 1 and line["n_gpus"] == 1
    assert line["value"] > 0 and line["ms_per_step"] > 0 and line["vs_baseline"] is None
    assert line["config"]["workload"].startswith("zipf") and "model" not in line["config"]
    cb = line["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["value"] == line["value"] and cb["sample"]
    assert line["e2e"] == {"value": line["value"], "unit": "GFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}


def test_reference_arm_other_ranks_stay_silent():
    res = _run({"RANK": "1", "LOCAL_RANK": "1", "WORLD_SIZE": "2"})
    assert res.returncode == 0 and res.stdout.strip() == ""


def test_traffic_figures_are_tied_to_every_file_of_a_kernel():
    """The hash behind a captured figure covers the kernel's source and every header of csrc/ that it includes."""
    import re
    sys.path.insert(0, ROOT)
    import bench
    csrc = os.path.join(ROOT, "liteform_ae_b200", "csrc")

    def includes(name, seen):
        for h in re.findall(r'#include "([^"]+)"', open(os.path.join(csrc, name)).read()):
            if h not in seen and os.path.exists(os.path.join(csrc, h)):
                seen.add(h)
                includes(h, seen)
        return seen
    for files in bench.KERNEL_SOURCES.values():
        assert set(files) == {files[0]} | includes(files[0], set())
