"""The stack depth that a traversal reports is the one a caller's stack capacity is compared with: that capacity fits
without a split, one entry less does not. Any capacity that fits gives the default's results, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _solve(p, params, ctx):
    import ryoanji_b200 as ryo
    out = [torch.empty(p.n, device="cuda") for _ in range(4)]
    return ryo.solve(*(dev(a) for a in (p.x, p.y, p.z, p.m, p.h)), *out, params, ctx=ctx)


def _tight(run):
    """run(capacity) gives (depth, retries, interaction counts)"""
    depth, retries, counts = run(0)
    assert depth > 1 and retries == 0
    assert run(depth) == (depth, 0, counts)
    try:
        assert run(depth - 1)[1] > 0
    except Exception as e:  # one target alone may be as deep
        assert getattr(e, "status", None) == 4


# walks in eight parts (by children of the root, by replicas), whole walks, and a large solve's queued groups
@pytest.mark.parametrize("kind,n,group", [("plummer", 1000, 64), ("plummer", 4097, 64), ("plummer", 60001, 64),
                                          ("periodic", 20011, 64), ("gauss", 100003, 64), ("plummer", 500009, 64),
                                          ("plummer", 100003, 8), ("plummer", 3200007, 64)])
def test_depth_is_the_capacity_that_fits(kind, n, group):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = (ds.plummer(n, seed=n, velocities=False) if kind == "plummer" else
         ds.periodic_box(n, seed=n, eps=0.002) if kind == "periodic" else ds.gaussian(n, seed=n, sigma=0.3))
    box = ryo.Box(*p.box, boundary=(ryo.BOUNDARY_PERIODIC,) * 3) if kind == "periodic" else None
    ctx = ryo.Context()

    def run(capacity):
        r = _solve(p, ryo.SolveParams(theta=0.5, bucket_size=32, group_size=group, box=box, stack_capacity=capacity),
                   ctx)
        assert ryo.read_bh_stats(ctx)[4] == r.max_stack
        return r.max_stack, r.retries, (r.sum_p2p, r.max_p2p, r.sum_m2p, r.max_m2p)
    _tight(run)


# as above, from a single leaf on, and with signed expansions
@pytest.mark.parametrize("kind,n,mdq", [("plummer", 40, False), ("plummer", 1000, False), ("plummer", 60001, False),
                                        ("periodic", 20011, False), ("gauss", 100003, True), ("plummer", 500009, False),
                                        ("plummer", 3200007, False)])
def test_capacities_that_fit_give_the_same_bits(kind, n, mdq):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = (ds.plummer(n, seed=n, velocities=False) if kind == "plummer" else
         ds.periodic_box(n, seed=n, eps=0.002) if kind == "periodic" else ds.gaussian(n, seed=n, sigma=0.3))
    box = ryo.Box(*p.box, boundary=(ryo.BOUNDARY_PERIODIC,) * 3) if kind == "periodic" else None
    ctx = ryo.Context()

    def run(capacity):
        out = torch.empty(4, n, device="cuda")
        r = ryo.solve(*(dev(a) for a in (p.x, p.y, p.z, p.m, p.h)), *out,
                      ryo.SolveParams(theta=0.5, box=box, multipole="mdq" if mdq else "quadrupole",
                                      stack_capacity=capacity), ctx=ctx)
        return r, out
    r, base = run(0)
    for capacity in (max(r.max_stack, 1), 512, 1024, 5000):
        q, out = run(capacity)
        assert torch.equal(out, base) and q.max_stack == r.max_stack and q.retries == 0


@pytest.mark.parametrize("capacity", [20, 40])
def test_capacity_that_most_groups_pass(capacity):
    """groups split until they fit; the expansions' error at theta 0.5 stays"""
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    n = 20011
    p = ds.plummer(n, seed=n, velocities=False)
    t, out = [dev(a) for a in (p.x, p.y, p.z, p.m, p.h)], torch.full((4, n), float("nan"), device="cuda")
    ctx = ryo.Context()
    try:
        ryo.solve(*t, *out, ryo.SolveParams(theta=0.5, bucket_size=32, stack_capacity=capacity), ctx=ctx)
    except ryo.RyoError as e:
        assert e.status == 4  # a target of its own passes the capacity too, and gets zeros
    assert ryo.read_bh_stats(ctx)[4] <= capacity and ryo.read_traversal_retries(ctx) > 50
    a = torch.stack(ryo.direct_targets_f64(torch.arange(n, device="cuda"), *t)[1:])
    done = out[0] != 0
    assert done.any()
    err = ((out[1:].double() - a).norm(dim=0) / a.norm(dim=0))[done].cpu().numpy()
    assert np.percentile(err, 99) < 1e-3 and np.median(err) < 2e-4


@pytest.mark.parametrize("real", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [3000, 60001])
def test_depth_of_double_traversals(real, n):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = ds.plummer(n, seed=n, velocities=False)
    x, y, z = (dev(a.astype(np.float64)) for a in (p.x, p.y, p.z))
    tb, box = ryo.TreeBuilder(32), ryo.Box.cube(-50.0, 50.0)
    nn = tb.update(x, y, z, box)
    m, h = dev(p.m).to(real), dev(p.h).to(real)
    centers = torch.zeros(nn, 4, device="cuda", dtype=torch.float64)
    mp = torch.zeros(nn, 8, device="cuda", dtype=real)
    ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
    ryo.upsweep_centers(tb.maxTreeLevel, tb.levelRange, tb.childOffsets(), centers)
    ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
    for level in range(tb.maxTreeLevel - 1, -1, -1):
        ryo.upsweep_multipoles(tb.levelRange[level], tb.levelRange[level + 1], tb.childOffsets(), centers, mp)
    ryo.set_mac(tb.nodeKeys(), centers, 2.0, box)
    groups = ryo.compute_fixed_groups(0, n, 64)

    def run(capacity):
        out = [torch.zeros(n, device="cuda", dtype=real) for _ in range(4)]
        ryo.traverse(groups, 1, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(), tb.internalToLeaf(), tb.layout(),
                     centers, mp, 1.0, 0, box.lengths, *out, stack_capacity=capacity)
        s = ryo.read_bh_stats()
        results.append(out)
        return s[4], ryo.read_traversal_retries(), s[:4]
    results = []
    _tight(run)
    run(512)
    for k in (1, -1):  # the depth's own capacity, and the default's size given
        assert all(torch.equal(a, b) for a, b in zip(results[0], results[k]))


def test_depth_of_a_batch():
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    sets = [ds.plummer(3001, seed=1, velocities=False), ds.periodic_box(2000, seed=2, eps=0.002),
            ds.plummer(70, seed=3, velocities=False), ds.periodic_box(9000, seed=4, eps=0.002)]
    bodies = [torch.cat([dev(getattr(p, k)) for p in sets]) for k in ("x", "y", "z", "m", "h")]
    systems = [ryo.BatchSystem(p.n, ryo.Box(*p.box, boundary=(ryo.BOUNDARY_PERIODIC,) * 3) if i % 2 else None, 2)
               for i, p in enumerate(sets)]

    def run(capacity):
        out = torch.empty(4, bodies[0].numel(), device="cuda")
        r = ryo.solve_batch(systems, *(b.clone() for b in bodies), *out,
                            params=ryo.SolveParams(theta=0.5, bucket_size=32, stack_capacity=capacity)).stats
        return r.max_stack, r.retries, (r.sum_p2p, r.max_p2p, r.sum_m2p, r.max_m2p)
    _tight(run)
