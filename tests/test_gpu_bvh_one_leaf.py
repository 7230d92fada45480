"""Device builds of so few triangles that the tree is one leaf, which read no counters back from
the device: the host's tree, whatever the pinned memory held that the counters are given."""
import ctypes

import numpy as np
import pytest

from petrichor_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _leave_bits_in_pinned_memory():
    cuda = ctypes.CDLL("libcuda.so.1")
    blocks = []
    for size in (16, 40, 64, 256, 4096) * 4:
        p = ctypes.c_void_p()
        assert cuda.cuMemHostAlloc(ctypes.byref(p), ctypes.c_size_t(size), 0) == 0
        ctypes.memset(p, 0xFF, size)
        blocks.append(p)
    for p in blocks:
        assert cuda.cuMemFreeHost(p) == 0


@pytest.mark.parametrize("triangles", [1, 2, 3, 4, 5])
def test_small_builds(gpu_ctx, triangles):
    torch.zeros(1, device="cuda")
    rng = np.random.default_rng(triangles)
    pos = rng.uniform(-1, 1, (3 * triangles, 3)).astype(np.float32)
    idx = np.arange(3 * triangles, dtype=np.int32).reshape(-1, 3)
    want = capi.bvh_build(pos, idx)
    for _ in range(8):
        _leave_bits_in_pinned_memory()
        got = gpu_ctx.bvh_build_device(pos, idx)
        for a, b in zip(want[:4], got[:4]):
            assert np.array_equal(np.asarray(a), np.asarray(b))
