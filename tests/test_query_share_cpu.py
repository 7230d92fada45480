"""Short ray queries whose warps take their rays by index (csrc/query_share.h), on the host:
no ray is left without a warp, whatever the grid (tests/cpp/query_share.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_ray_has_a_warp(tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    exe = str(tmp_path / "query_share")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-fsanitize=undefined", "-fno-sanitize-recover",
                    "-I", os.path.join(ROOT, "petrichor_gb300", "csrc"), "-isystem", cuda,
                    os.path.join(ROOT, "tests", "cpp", "query_share.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    assert int(r.stdout.split()[1]) > 10_000
