"""The device pool's bookkeeping on the CPU: its CUDA calls are fakes
(tests/cpp/pool_main.cpp), so that streams run as far as the test lets them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranges_in_use_by_another_stream(tmp_path):
    from proteus_gb300 import build

    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    csrc = os.path.join(ROOT, "proteus_gb300", "csrc")
    exe = str(tmp_path / "pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + csrc, "-I" + os.path.join(cuda, "include"), "-x", "c++",
                    os.path.join(csrc, "pool.cu"), os.path.join(ROOT, "tests", "cpp", "pool_main.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
