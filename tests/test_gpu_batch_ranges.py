"""Per-system value ranges of a batched solve: systems that start and end inside, at and across the bodies of a warp."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
ryo = pytest.importorskip("ryoanji_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[256], [255, 1, 257, 3], [1] * 300, [1, 511, 512, 513, 2, 31, 33, 5000, 7]],
                         ids=["one", "edges", "singles", "mixed"])
@pytest.mark.parametrize("multipole", ["quadrupole", "mdq"])
def test_batch_ranges_equal_single_solves(sizes, multipole):
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes)
    pos = rng.normal(size=(3, n)).astype(np.float32) * rng.uniform(0.1, 10.0, n).astype(np.float32)
    m = rng.uniform(0.5, 1.5, n).astype(np.float32)
    h = rng.uniform(0.01, 0.02, n).astype(np.float32)
    first = np.concatenate([[0], np.cumsum(sizes)])
    for s in range(0, len(sizes), 2):  # every other system has one softening and one mass
        m[first[s]:first[s + 1]] = 1.25
        h[first[s]:first[s + 1]] = 0.015625
    params = ryo.SolveParams(theta=0.5, bucket_size=16, group_size=64, multipole=multipole)
    dev = [torch.from_numpy(a.copy()).cuda() for a in (*pos, m, h)]
    out = [torch.empty(n, device="cuda") for _ in range(4)]
    res = ryo.solve_batch([ryo.BatchSystem(k) for k in sizes], *dev, *out, params)
    for s in list(range(len(sizes)))[:20]:
        sl = slice(int(first[s]), int(first[s + 1]))
        one = [torch.from_numpy(a[sl].copy()).cuda() for a in (*pos, m, h)]
        o = [torch.empty(sizes[s], device="cuda") for _ in range(4)]
        r = ryo.solve(*one, *o, params=params)
        assert r.box == pytest.approx(res.boxes[s], rel=0, abs=0)
        assert torch.equal(dev[0][sl], one[0])
        # a group's sums move by a few float ulps of the field where its list is cut elsewhere
        scale = float(torch.sqrt(o[1] ** 2 + o[2] ** 2 + o[3] ** 2).max()) + 1e-30
        for a, b in zip(out[1:], o[1:]):
            assert float((a[sl] - b).abs().max()) <= 1e-6 * scale
        assert float((out[0][sl] - o[0]).abs().max()) <= 1e-6 * float(o[0].abs().max()) + 1e-30
