"""Small sorts run in one cluster of blocks: edges of its blocks, of its keys per thread, and of the general sort."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
ryo = pytest.importorskip("ryoanji_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distinct", [3, 300, 0])
@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 5121, 8191, 8192, 8193, 14337, 16384, 16385, 20481, 32768,
                               32769, 57345, 65535, 65536, 65537])
def test_small_sort_is_exact_and_stable(n, distinct):
    rng = np.random.default_rng(n + distinct)
    keys = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if distinct:  # equal keys keep their order; the largest key is also what pads the last block
        keys = np.concatenate([rng.integers(0, 1 << 64, distinct - 1, dtype=np.uint64),
                               np.array([2**64 - 1], np.uint64)])[rng.integers(0, distinct, n)]
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    order = np.argsort(keys, kind="stable")
    k = torch.from_numpy(keys.view(np.int64)).cuda()
    v = torch.from_numpy(vals.view(np.int32)).cuda()
    ryo.sort_by_key(k, v)
    assert np.array_equal(k.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[order])
