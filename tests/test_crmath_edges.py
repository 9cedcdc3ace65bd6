"""Host check of the exp/log evaluations of bpl_crmath.cuh at the edges of
their tables and argument reductions, and of the exactness these rely on."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fast_exp_log_at_table_edges(tmp_path):
    exe = str(tmp_path / "crmath_edges")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "crmath", "crmath_edges.cpp")])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
