"""The host side of device calls (csrc/capi.cpp) over a fake CUDA runtime
(tests/cpp/fake_cuda.h): what a call enqueues, on which stream, and which words it uses."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "petrichor_gb300", "csrc")


@pytest.fixture(scope="module")
def host_objects(tmp_path_factory):
    return build_host_objects(tmp_path_factory.mktemp("host"))


def build_host_objects(out, names=("capi", "scheduler", "server", "bvh_builder")):
    """Objects of the host code behind the C ABI, to be linked with the fake runtime."""
    procs, objs = [], []
    for name in names:
        objs.append(str(out / f"{name}.o"))
        procs.append(subprocess.Popen(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-pthread", *includes(), "-c",
                                       os.path.join(CSRC, f"{name}.cpp"), "-o", objs[-1]]))
    assert all(p.wait() == 0 for p in procs)
    return objs


def includes():
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    return ["-I", CSRC, "-I", os.path.join(ROOT, "include"), "-isystem", cuda]


def run_client(objs, source, exe, *args):
    """Builds tests/cpp/`source` with `objs`; the launch functions it does not define stay
    unresolved and are not called."""
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-no-pie", "-fno-pie", "-pthread",
                    *includes(), os.path.join(ROOT, "tests", "cpp", source), *objs,
                    "-Wl,--unresolved-symbols=ignore-all", "-o", exe], check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_a_query_works_on_its_own_stream_alone(host_objects, tmp_path):
    assert run_client(host_objects, "ray_query.cpp", str(tmp_path / "ray_query")).startswith("ok")


def test_a_render_clears_its_wave_buffers_on_its_own_stream(host_objects, tmp_path):
    assert run_client(host_objects, "render_stream.cpp", str(tmp_path / "render_stream")).startswith("ok")


def test_an_upload_needs_no_more_than_the_build_or_the_scene(host_objects, tmp_path):
    """Device memory of an upload: the larger of the build and the scene, and part of an image."""
    assert run_client(host_objects, "upload_peak.cpp", str(tmp_path / "upload_peak")).startswith("ok")


def test_the_autotuner_probes_waves_that_run_as_the_renders(host_objects, tmp_path):
    assert run_client(host_objects, "autotune_probe.cpp", str(tmp_path / "autotune_probe")).startswith("ok")
