"""Which waves count as interiors, on the host (tests/cpp/interior.cpp)."""
from test_host_streams_cpu import build_host_objects, run_client


def test_interior_waves(tmp_path):
    assert run_client(build_host_objects(tmp_path, ["scheduler"]), "interior.cpp", str(tmp_path / "interior")).startswith("ok")
