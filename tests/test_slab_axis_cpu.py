"""The ray-box test of axis-parallel caller rays (csrc/slab.h), on the host
(tests/cpp/slab_axis.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_boxes_on_the_way_are_hit(tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    exe = str(tmp_path / "slab_axis")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "petrichor_gb300", "csrc"), "-isystem", cuda,
                    os.path.join(ROOT, "tests", "cpp", "slab_axis.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    cases, hits = (int(x) for x in r.stdout.split()[1:])
    assert cases > 10_000 and hits > 500
