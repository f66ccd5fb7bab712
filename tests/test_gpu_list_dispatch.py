"""Traversals on either side of the group counts at which interaction lists end agree: the same bodies and tree, groups
of one body, and one group of two or none. Counts per group are equal, results to the rounding of their sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tree(kind, n, shells, special=None):
    import ryoanji_b200 as ryo
    ct = torch.float32 if kind == "f32" else torch.float64
    rt = torch.float64 if kind == "f64" else torch.float32
    rng = np.random.default_rng(n)
    p = np.concatenate([rng.normal(0, 0.02, (n // 4, 3)), rng.uniform(-1, 1, (n - n // 4, 3))])
    x, y, z = (torch.from_numpy(np.ascontiguousarray(v)).cuda().to(ct) for v in p.T)
    m = torch.from_numpy(rng.uniform(0.5, 1.5, n) / n).cuda().to(rt)
    h = torch.full((n,), 1e-3, device="cuda", dtype=rt)
    if special:
        {"m": m, "h": h}[special[0]][n // 3] = special[1]
    tb, box = ryo.TreeBuilder(32), ryo.Box.cube(-1.0, 1.0)
    nn = tb.update(x, y, z, box)
    centers = torch.zeros(nn, 4, device="cuda", dtype=ct)
    mp = torch.zeros(nn, 8, device="cuda", dtype=rt)
    ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
    ryo.upsweep_centers(tb.maxTreeLevel, tb.levelRange, tb.childOffsets(), centers)
    ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
    for level in range(tb.maxTreeLevel - 1, -1, -1):
        ryo.upsweep_multipoles(tb.levelRange[level], tb.levelRange[level + 1], tb.childOffsets(), centers, mp)
    ryo.set_mac(tb.nodeKeys(), centers, 2.0, box)

    def run(groups):
        out = torch.zeros(4, n, device="cuda", dtype=rt)
        pot, m2p, p2p = ryo.traverse(groups, 1, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(), tb.internalToLeaf(),
                                     tb.layout(), centers, mp, 1.0, shells, box.lengths, *out, group_counts=True)
        return out.double(), pot, m2p, p2p, ryo.read_bh_stats()[4]
    return run


@pytest.mark.parametrize("kind,shells,last", [("f32", 0, 16384), ("f32", 1, 2560), ("f64", 0, 49152), ("f64", 1, 24576),
                                              ("mixed", 0, 49152), ("mixed", 1, 24576)])
def test_both_sides_agree(kind, shells, last):
    n = last + 1
    run = _tree(kind, n, shells)
    ones = torch.arange(n + 1, device="cuda", dtype=torch.int32)  # one group too many for lists
    pair = torch.cat([ones[:n - 1], ones[n:]])                    # the last two bodies as one group
    fused, lists = run(ones), run(pair)
    for k in (2, 3):
        assert torch.equal(fused[k][:n - 2], lists[k][:n - 2])
    a, b = fused[0][:, :n - 2], lists[0][:, :n - 2]
    scale = a[1:].norm(dim=0).clamp_min(0.1)  # images cancel; the box's mass is 1, its side 2
    err = ((a - b)[1:].norm(dim=0) / scale).cpu().numpy()
    bound = (5e-6, 5e-5) if kind == "f32" else (2e-6, 2e-5) if kind == "mixed" else (1e-12, 1e-10)
    assert np.percentile(err, 99) < bound[0] and err.max() < bound[1]
    assert torch.allclose(a[0], b[0], rtol=10 * bound[0], atol=float(a[0].abs().max()) * bound[0])
    assert abs(fused[4] - lists[4]) <= 64  # the pair may walk deeper than either of its bodies


# (a mass of NaN or infinity makes every body's sums NaN or infinite; a softening only its own pairs')
@pytest.mark.parametrize("special", [("m", np.nan), ("m", np.inf), ("h", np.nan), ("h", np.inf), ("h", -1e-3)])
@pytest.mark.parametrize("kind,shells,last", [("f32", 0, 16384), ("f32", 1, 2560), ("f64", 0, 49152),
                                              ("mixed", 1, 24576)])
def test_special_values(kind, shells, last, special):
    n = last + 1
    run = _tree(kind, n, shells, special)
    ones = torch.arange(n + 1, device="cuda", dtype=torch.int32)
    fused, lists = run(ones), run(torch.cat([ones[:n - 1], ones[n:]]))
    a, b = fused[0][:, :n - 2], lists[0][:, :n - 2]
    assert torch.equal(a.isnan(), b.isnan())
    inf = a.isinf()
    assert torch.equal(inf, b.isinf()) and torch.equal(a[inf], b[inf])
    ok = a.isfinite()
    if ok.any():
        assert float((a - b)[ok].abs().max()) <= 1e-5 * float(a[ok].abs().max())
