"""The sums of interaction lists lose nothing between a group's items: every term of the field below is exact in float
arithmetic, and an item holds its large terms before its small ones, so that its compensated sum is exact as well. The
result is then the exact sum rounded to float once: half a unit in the last place."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cells_of_64(rng):
    """64 bodies in every cell of an 8 x 8 x 8 grid on [-1/4, 1/4]^3, at multiples of 2^-12; all leaves are cells"""
    at = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 1, 3) * 256
    steps = at + rng.integers(0, 256, (512, 64, 3)) - 1024
    return (steps.reshape(-1, 3) * 2.0 ** -12).astype(np.float32)


def test_items_are_added_without_rounding():
    import ryoanji_b200 as ryo
    rng = np.random.default_rng(12)
    x, y, z = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in _cells_of_64(rng).T)
    n = x.numel()
    # (h + h)^2 = 1 is beyond every distance: a source's pull is m times the difference of the positions
    m, h = torch.ones(n, device="cuda"), torch.full((n,), 0.5, device="cuda")
    out = [torch.empty(n, device="cuda") for _ in range(4)]
    params = ryo.SolveParams(theta=0.01, bucket_size=64, box=ryo.Box.cube(-0.25, 0.25))
    ctx = ryo.Context()
    r = ryo.solve(x, y, z, m, h, *out, params, ctx=ctx)  # sorts the bodies: 512 leaves, a group each
    assert r.num_leaves == 512 and r.num_groups == 512 and r.sum_p2p == n * n and r.sum_m2p == 0
    # the walk lists the halves of an octant's 64 leaves as an item each, in this order: large masses in the first
    # half of each, whose signs make the octants cancel, small masses in the second
    leaf = np.arange(n) // 64
    heavy = leaf // 16 % 2 == 0
    sign = np.where(leaf // 64 % 2 == 0, 1.0, -1.0)
    mass = np.where(heavy, sign, 2.0 ** -14).astype(np.float32)
    m.copy_(torch.from_numpy(mass))
    r = ryo.solve(x, y, z, m, h, *out, params, ctx=ctx)
    assert r.sum_p2p == n * n
    assert np.array_equal(m.cpu().numpy(), mass)
    M = mass.astype(np.float64)
    for a, v in zip(out[1:], (x, y, z)):
        v = v.double().cpu().numpy()
        exact = (M * v).sum() - M.sum() * v  # all terms and sums are multiples of 2^-26: exact in float64
        a = a.double().cpu().numpy()
        ulp = np.spacing(np.abs(a).astype(np.float32)).astype(np.float64)
        assert np.abs(a - exact).max() > 0  # not every result fits into a float
        assert (np.abs(a - exact) / ulp).max() <= 0.5


def test_host_launches_add_in_the_order_of_the_device_solve():
    """pageable outputs: eight launches of 375 groups each, whose items are added by a block per group; the device
    solve's 3,000 groups by a warp each. The heavy octants' sums, of some hundreds, nearly cancel in the results, and two
    octants' masses are so small that the others' sums leave out some of their bits in float64."""
    import ryoanji_b200 as ryo
    rng = np.random.default_rng(5)
    n = 24000
    pos = rng.uniform(-0.25, 0.25, (n, 3)).astype(np.float32)
    m = np.where((pos > 0).sum(1) % 2 == 0, 1.0, -1.0) * rng.uniform(0.5, 1.0, n)
    light = (pos[:, 0] > 0) & (pos[:, 1] > 0)
    heavy = np.concatenate([np.ones((n, 1)), pos], 1)[~light].astype(np.float64)
    basis = np.linalg.qr(heavy)[0]
    m[~light] -= basis @ (basis.T @ m[~light])  # the heavy bodies have neither a total mass nor a dipole
    m[light] *= 2.0 ** -30
    m = m.astype(np.float32)
    bodies = [torch.from_numpy(np.ascontiguousarray(v)) for v in (*pos.T, m, np.full(n, 0.5, np.float32))]
    params = ryo.SolveParams(theta=0.01, bucket_size=32, group_size=8, box=ryo.Box.cube(-0.25, 0.25))
    ctx = ryo.Context()
    host = [torch.empty(n) for _ in range(4)]
    ryo.solve_host(*bodies, *host, params=params, ctx=ctx)
    dev = [torch.empty(n, device="cuda") for _ in range(4)]
    r = ryo.solve(*(v.cuda() for v in bodies), *dev, params, ctx=ctx)
    assert r.num_groups == 3000
    assert max(v.abs().median() for v in host[1:]) < 1e-2  # the parts' sums do cancel
    for a, b in zip(host, dev):
        assert torch.equal(a, b.cpu())


def test_host_solve_of_a_clustered_set_equals_the_device_solve():
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    n = 300007
    p = ds.plummer(n, seed=9, velocities=False)
    bodies = [torch.from_numpy(a) for a in (p.x, p.y, p.z, p.m, p.h)]
    ctx = ryo.Context()
    host = [torch.empty(n) for _ in range(4)]
    rh = ryo.solve_host(*bodies, *host, params=ryo.SolveParams(theta=0.5), ctx=ctx)
    dev = [torch.empty(n, device="cuda") for _ in range(4)]
    rd = ryo.solve(*(v.cuda() for v in bodies), *dev, ryo.SolveParams(theta=0.5), ctx=ctx)
    assert 2369 <= rd.num_groups <= 6000 and rh.max_stack == rd.max_stack
    for a, b in zip(host, dev):
        assert torch.equal(a, b.cpu())
