"""Leaf construction around the sizes where its scans and its sizing change: tiles of 4,096 values, four tiles scanned
by one block, blocks of 256 keys, and 2^18 keys."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
ryo = pytest.importorskip("ryoanji_b200")

pytestmark = pytest.mark.gpu


def cornerstone(keys, bucket):
    """leaves of at most @p bucket keys by splitting nodes level by level (keys sorted, below 8^21)"""
    done, start, size = [], np.zeros(1, np.uint64), 8 ** 21
    while len(start):
        count = np.searchsorted(keys, start + np.uint64(size)) - np.searchsorted(keys, start)
        split = (count > bucket) & (size > 1)
        done.append(np.stack([start[~split], count[~split].astype(np.uint64)], 1))
        size //= 8
        start = (start[split][:, None] + np.arange(8, dtype=np.uint64) * np.uint64(size)).ravel()
    leaves = np.concatenate(done)
    return leaves[np.argsort(leaves[:, 0])]


@pytest.mark.parametrize("n", [2, 256, 257, 4094, 4095, 4096, 16382, 16383, 16384, 20481, 262143, 262144, 262145])
@pytest.mark.parametrize("bucket", [1, 64])
def test_leaves_at_scan_edges(n, bucket):
    rng = np.random.default_rng(n + bucket)
    keys = rng.integers(0, 8 ** 21, n, dtype=np.uint64)
    keys[: n // 3] >>= np.uint64(20)  # a crowded corner: deep leaves and empty ones beside them
    keys = np.unique(keys)
    leaves, counts = ryo.compute_octree(torch.from_numpy(keys.view(np.int64)).cuda(), bucket)
    want = cornerstone(keys, bucket)
    assert np.array_equal(leaves.cpu().numpy().view(np.uint64), np.append(want[:, 0], np.uint64(8 ** 21)))
    assert np.array_equal(counts.cpu().numpy().astype(np.uint64), want[:, 1])
