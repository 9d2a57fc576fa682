"""How the exact scan sizes its workspace when memory is short (host compile of
the rule, CPU only)."""
import os
import subprocess

from hnsw_rabitq_b200 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_one_query_is_enough(tmp_path):
    exe = tmp_path / "batchchk"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "hnsw_rabitq_b200", "csrc"),
                           "-I", os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include"),
                           os.path.join(ROOT, "tests", "bf_batch_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
