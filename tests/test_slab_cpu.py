"""The traversal's ray-box test with the near planes chosen once per ray (csrc/slab.h)
against the form that orders every axis's two distances, on the host: every combination of
special values (tests/cpp/slab.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_chosen_planes_equal_the_two_sided_form(tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    exe = str(tmp_path / "slab")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "petrichor_gb300", "csrc"), "-isystem", cuda,
                    os.path.join(ROOT, "tests", "cpp", "slab.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    assert int(r.stdout.split()[1]) > 100_000
