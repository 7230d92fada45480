"""Device BVH builds whose node ranges lie at the edges of the block sorts' size classes (128,
1024 and 8192 elements, csrc/bvh_gpu.cu BlockSortKernel): the host build's tree, node for node
and primitive for primitive, for random, sorted, reversed, organ-pipe, few-valued and equal
keys and for std::sort's worst case, inside one block and above it."""
import os
import subprocess

import numpy as np
import pytest

from petrichor_gb300 import capi

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _triangles(x):
    """One triangle per key, its centroid's x exactly 3 key / 3; y and z of the centroids equal."""
    n = len(x)
    x = 3.0 * np.asarray(x, np.float64)
    P = np.stack([np.stack([x, np.zeros(n), np.zeros(n)], 1), np.stack([x, np.ones(n), np.zeros(n)], 1),
                  np.stack([x, np.zeros(n), np.ones(n)], 1)], 1).reshape(-1, 3).astype(np.float32)
    return P, np.arange(3 * n, dtype=np.int32).reshape(n, 3)


def _same(ctx, P, I):
    dev, host = ctx.bvh_build_device(P, I), capi.bvh_build(P, I)
    assert np.array_equal(dev[0].view(np.uint32), host[0].view(np.uint32))
    assert np.array_equal(dev[1], host[1]) and np.array_equal(dev[2], host[2]) and dev[3] == host[3]
    return dev[4]


KEYS = {
    "random": lambda r, n: r.permutation(n),
    "sorted": lambda r, n: np.arange(n),
    "reversed": lambda r, n: np.arange(n)[::-1],
    "organ": lambda r, n: np.minimum(np.arange(n), n - 1 - np.arange(n)),
    "few": lambda r, n: r.integers(0, 7, n),
    "equal": lambda r, n: np.where(np.arange(n) < n // 2, 5, 5 + (np.arange(n) % 997 == 0)),
}


@pytest.mark.parametrize("n", [31, 127, 128, 129, 1023, 1024, 1025, 8191, 8192, 8193, 30000])
@pytest.mark.parametrize("kind", sorted(KEYS))
def test_size_classes(gpu_ctx, kind, n):
    _same(gpu_ctx, *_triangles(KEYS[kind](np.random.default_rng(n), n)))


@pytest.mark.parametrize("n", [120, 1000, 8000, 12000])
def test_depth_budget_runs_out(gpu_ctx, tmp_path, n):
    exe = str(tmp_path / "antiqsort")
    subprocess.run(["g++", "-std=c++17", "-O2", os.path.join(ROOT, "tests", "cpp", "antiqsort.cpp"), "-o", exe],
                   check=True)
    keys = subprocess.run([exe, str(n)], capture_output=True, text=True, check=True).stdout.split()
    stats = _same(gpu_ctx, *_triangles(np.array(keys, np.int64)))
    assert stats.heapsorts > 0


def test_more_positions_than_one_block_scans(gpu_ctx):
    """1.1M triangles: the partition rounds' prefix sums have more spans than ScanTopKernel's
    block has threads."""
    _same(gpu_ctx, *_triangles(np.random.default_rng(2).integers(0, 1 << 20, 1_100_000)))
