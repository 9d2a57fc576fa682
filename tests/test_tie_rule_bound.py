"""The tie rule the beam uses (csrc/tie_rule.h, compiled for the host) against
the reference's heaps: fixed graphs in which a neighbour is rejected at a
lowerBound that fell inside its own unit, and over a million kept runs on random
ones (CPU only)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_kept_runs_are_the_references(tmp_path):
    exe = tmp_path / "tiechk"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "hnsw_rabitq_b200", "csrc"),
                           os.path.join(ROOT, "tests", "tie_rule_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe), "1200000"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
