"""The slot count from the degrees alone equals that of every packing."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slots_without_packing(tmp_path):
    exe = str(tmp_path / "slots_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", exe, os.path.join(ROOT, "tests", "cpp", "slots_check.cpp"),
                    os.path.join(ROOT, "analogsat_b200", "csrc", "as_problem.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "slots ok" in r.stdout, r.stdout + r.stderr
