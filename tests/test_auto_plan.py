"""The autotuner's candidates against the untuned plans (host code, on the CPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_untuned_plan_is_among_the_candidates(tmp_path):
    exe = str(tmp_path / "auto_plan")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "proteus_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "auto_plan_main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
