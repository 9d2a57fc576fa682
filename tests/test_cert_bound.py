"""The certified exact scan's error bound (csrc/cert_bound.h, compiled for the
host) against a model of the tensor cores' accumulation, worst cases included
(CPU only)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bound_holds_for_the_model(tmp_path):
    exe = tmp_path / "certchk"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                           os.path.join(ROOT, "hnsw_rabitq_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cert_bound_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
