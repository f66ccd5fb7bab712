"""Traversals whose interaction lists find too little free memory take what there is, in more launches, with the same
bits; and a call that fails for lack of memory leaves no error behind."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fill(leave):
    """takes the device's free memory but @p leave bytes"""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")


def _solve(ryo, bodies, work, out, params, ctx):
    for w, b in zip(work, bodies):
        w.copy_(b)
    return ryo.solve(*work, *out, params, ctx=ctx)


# divided walks, whole walks
@pytest.mark.parametrize("n,group,leave", [(1 << 18, 64, 256 << 20), (200003, 16, 256 << 20)])
def test_solve_with_little_memory(n, group, leave):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = ds.plummer(n, seed=n, velocities=False)
    params = ryo.SolveParams(theta=0.5, group_size=group)
    bodies = [torch.from_numpy(a).cuda() for a in (p.x, p.y, p.z, p.m, p.h)]
    work, out = [b.clone() for b in bodies], torch.empty(4, n, device="cuda")
    first = ryo.Context()
    r = _solve(ryo, bodies, work, out, params, first)
    base = out.clone()
    del first
    ctx = ryo.Context()
    hog = _fill(leave)
    try:
        for _ in range(2):
            out.fill_(float("nan"))
            s = _solve(ryo, bodies, work, out, params, ctx)
            assert torch.equal(out, base)
            assert (s.sum_p2p, s.max_p2p, s.sum_m2p, s.max_m2p, s.max_stack, s.retries) == (
                r.sum_p2p, r.max_p2p, r.sum_m2p, r.max_m2p, r.max_stack, r.retries)
    finally:
        del hog
        torch.cuda.empty_cache()
    out.fill_(float("nan"))
    _solve(ryo, bodies, work, out, params, ctx)
    assert torch.equal(out, base)


@pytest.mark.parametrize("real", [torch.float64, torch.float32])
def test_double_traversal_with_little_memory(real):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    n = 250007
    p = ds.plummer(n, seed=3, velocities=False)
    x, y, z = (torch.from_numpy(a.astype(np.float64)).cuda() for a in (p.x, p.y, p.z))
    m, h = torch.from_numpy(p.m).cuda().to(real), torch.from_numpy(p.h).cuda().to(real)
    tb, box = ryo.TreeBuilder(64), ryo.Box.cube(-50.0, 50.0)
    nn = tb.update(x, y, z, box)
    centers = torch.zeros(nn, 4, device="cuda", dtype=torch.float64)
    mp = torch.zeros(nn, 8, device="cuda", dtype=real)
    ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
    ryo.upsweep_centers(tb.maxTreeLevel, tb.levelRange, tb.childOffsets(), centers)
    ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
    for level in range(tb.maxTreeLevel - 1, -1, -1):
        ryo.upsweep_multipoles(tb.levelRange[level], tb.levelRange[level + 1], tb.childOffsets(), centers, mp)
    ryo.set_mac(tb.nodeKeys(), centers, 2.0, box)
    groups = ryo.compute_fixed_groups(0, n, 64)
    out = torch.zeros(4, n, device="cuda", dtype=real)

    def run(ctx):
        out.zero_()
        ryo.traverse(groups, 1, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(), tb.internalToLeaf(), tb.layout(),
                     centers, mp, 1.0, 0, box.lengths, *out, ctx=ctx)
        return out.clone(), ryo.read_bh_stats(ctx)
    first = ryo.Context()
    base, stats = run(first)
    del first
    ctx = ryo.Context()
    hog = _fill(256 << 20)
    try:
        got, s = run(ctx)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert torch.equal(got, base) and s == stats

def test_failed_allocation_leaves_no_error():
    import ryoanji_b200 as ryo
    n = 1 << 22
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    bodies = [torch.rand(n, generator=gen, device="cuda") for _ in range(4)] + [torch.full((n,), 1e-4, device="cuda")]
    work, out = [b.clone() for b in bodies], torch.empty(4, n, device="cuda")
    ctx = ryo.Context()
    hog = _fill(96 << 20)  # the sort alone of four million bodies takes more
    try:
        with pytest.raises(ryo.RyoError) as e:
            _solve(ryo, bodies, work, out, ryo.SolveParams(), ctx)
        assert e.value.status == 3
    finally:
        del hog
        torch.cuda.empty_cache()
    _solve(ryo, bodies, work, out, ryo.SolveParams(), ctx)
    assert torch.isfinite(out).all()
