"""The benchmark's reference arm on a CPU: `bench.py --impl reference` runs
the compiled reference's clone engine on a small batch and prints exactly
one JSON line on standard output (the reference library's own printf
lines go to standard error), with the fields its consumers read."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_prints_one_json_line(reflib):
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference",
                        "--steps", "1", "--warmup", "1", "--events", "2"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.strip()]
    assert len(lines) == 1, r.stdout
    d = json.loads(lines[0])
    assert d["impl"] == "reference"
    assert d["metric"] == "events built/s" and d["unit"] == "events/s"
    assert d["higher_is_better"] is True and d["value"] > 0
    assert d["steps"] == 1 and d["warmup"] == 1 and d["n_gpus"] == 1
    assert d["config"]["events_per_step"] == 2
    cb = d["cpu_baseline"]
    assert cb["kind"] == "reference" and cb["cores"] >= 1 and cb["value"] == d["value"]
    assert d["e2e"] == {"value": d["value"], "unit": "events/s", "h2d_bytes_per_step": 0,
                        "d2h_bytes_per_step": 0}
    assert d["gpu_launches"] == 0


def test_reference_arm_under_two_ranks(reflib):
    """Under the launcher with two ranks, rank 0 alone runs and prints the
    line (n_gpus 2, the GPU arm's config at that world size); the other
    rank exits 0 without work."""
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1",
                        "--nproc-per-node", "2", "--master-addr", "127.0.0.1",
                        "--master-port", "29613", os.path.join(ROOT, "bench.py"),
                        "--impl", "reference", "--gpus", "2", "--steps", "1", "--warmup", "1",
                        "--events", "2"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.strip()]
    assert len(lines) == 1, r.stdout
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["n_gpus"] == 2
    assert d["config"]["parallelism"].startswith("dp2")


def test_lines_without_the_reference_build(monkeypatch, capsys):
    """Where the reference sources were not there to be built, both arms still
    print their line: the GPU arm's CPU figures say why they are absent."""
    import argparse

    import bench
    import oracle.oracle
    monkeypatch.setattr(oracle.oracle, "have_ref", lambda flavour="avx2": False)
    for k in ("RANK", "WORLD_SIZE"):
        monkeypatch.delenv(k, raising=False)
    assert bench.cpu_baseline_fit(None, 8) == {"unavailable": bench.NO_REFERENCE}
    assert bench.cpu_baseline_find([]) == {"unavailable": bench.NO_REFERENCE}
    bench.run_reference(argparse.Namespace(events=2, steps=1, warmup=1))
    assert json.loads(capsys.readouterr().out) == {"impl": "reference",
                                                   "unavailable": bench.NO_REFERENCE}
