"""Traversals through interaction lists (solves of up to 49,152 target groups, and the longest groups of larger ones).

Interaction counts are compared bit for bit with the oracle's statement of the rule on the same tree, forces with its
double-precision evaluation of the same lists (the tolerances of the other traversal tests). Where the oracle would take
too long, forces are compared with FP64 direct sums.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.cpu().numpy()


def _solve(p, params, ctx):
    import ryoanji_b200 as ryo
    t = [dev(a) for a in (p.x, p.y, p.z, p.m, p.h)]
    out = [torch.empty(p.n, device="cuda") for _ in range(4)]
    return ryo.solve(*t, *out, params, ctx=ctx), t, out


def _set(kind, n):
    from ryoanji_b200 import datasets as ds
    if kind == "plummer":
        return ds.plummer(n, seed=n, velocities=False)
    if kind == "periodic":
        return ds.periodic_box(n, seed=n, eps=0.002)
    p = ds.gaussian(n, seed=n, sigma=0.3)  # per-body masses; per-body softenings too
    p.h = np.random.default_rng(n).uniform(1e-4, 2e-2, n).astype(np.float32)
    return p


# single bodies and groups, one body more than a group, a tree of one leaf, walks split in eight parts with empty parts,
# partial batches, whole and ragged last groups, and (at bucket 1) leaves by the thousand
@pytest.mark.parametrize("kind", ["plummer", "gauss", "periodic"])
@pytest.mark.parametrize("n,bucket", [(1, 64), (2, 64), (64, 64), (65, 64), (66, 8), (129, 8), (1000, 1), (4097, 32),
                                      (20011, 64)])
def test_lists_against_oracle(oracle, kind, n, bucket):
    import ryoanji_b200 as ryo
    p = _set(kind, n)
    box = ryo.Box(*p.box, boundary=(ryo.BOUNDARY_PERIODIC,) * 3) if kind == "periodic" else None
    ctx = ryo.Context()
    off = ryo.EwaldSettings(numReplicaShells=0, lCut=0.0, hCut=0.0, alpha_scale=0.0)
    res, t, out = _solve(p, ryo.SolveParams(theta=0.5, bucket_size=bucket, box=box, ewald=off), ctx)
    again = _solve(p, ryo.SolveParams(theta=0.5, bucket_size=bucket, box=box, ewald=off), ctx)[2]
    assert all(torch.equal(a, b) for a, b in zip(out, again))  # the lists' pieces are added in a fixed order
    arr = ryo.solve_arrays(ctx)
    g = host(arr["groups"]).view(np.uint32)
    x, y, z, m, h = (host(a) for a in t)
    L = [p.box[1] - p.box[0]] * 3 if kind == "periodic" else [0.0] * 3
    tree = {k: host(arr[k]) for k in ("childOffsets", "internalToLeaf", "centers", "multipoles")}
    alone = arr["numNodes"] == 1
    if alone:  # the oracle tests eight siblings: the single leaf and seven cells without extent, which it counts
        tree = {k: np.concatenate([v, np.zeros((7,) + v.shape[1:], v.dtype)]) for k, v in tree.items()}
    m2p, p2p, acc = oracle.traverse_rule(g[:-1], g[1:], x, y, z, h, m, tree, host(arr["layout"]).view(np.uint32),
                                         np.ascontiguousarray(tree["centers"]),
                                         np.ascontiguousarray(tree["multipoles"]), init_node=0 if alone else 1,
                                         numShells=1 if kind == "periodic" else 0, boxL=L, evaluate=True)
    if alone:
        m2p -= np.uint32(7 * (27 if kind == "periodic" else 1))
    assert np.array_equal(host(arr["groupM2P"]).view(np.uint32), m2p)
    assert np.array_equal(host(arr["groupP2P"]).view(np.uint32), p2p)
    sizes = np.diff(g).astype(np.int64)
    assert res.sum_p2p == int((p2p.astype(np.int64) * sizes).sum()) and res.max_p2p == int(p2p.max())
    assert res.sum_m2p == int((m2p.astype(np.int64) * sizes).sum()) and res.max_m2p == int(m2p.max())
    a = np.stack([host(v) for v in out[1:]], 1)
    # the images of a periodic body pull it with G M / L^2 = 1 each and cancel, wholly for a single body
    scale = np.maximum(np.linalg.norm(acc[:, 1:4], axis=1), 1.0 if kind == "periodic" else 1e-30)
    err = np.linalg.norm(a - acc[:, 1:4], axis=1) / scale
    assert np.percentile(err, 99) < 5e-6 and err.max() < 5e-5
    phi = m * acc[:, 0]
    assert np.allclose(host(out[0]), phi, rtol=1e-5, atol=1e-6 * np.abs(phi).max())


def test_list_pool_runs_out():
    """an opening angle so strict that the lists' pieces outnumber the pool: the groups without room walk again"""
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    n = 1 << 16
    p = ds.plummer(n, seed=3, velocities=False)
    ctx = ryo.Context()
    res, t, out = _solve(p, ryo.SolveParams(theta=0.02, bucket_size=16), ctx)
    arr = ryo.solve_arrays(ctx)
    cost = host(arr["groupP2P"]).astype(np.int64) + 2 * host(arr["groupM2P"]).astype(np.int64)
    assert (cost // 1024).sum() > 6 * 8 * len(cost) + 4096  # pieces hold at most 1,024 interactions and a segment
    assert res.sum_p2p == int((host(arr["groupP2P"]).astype(np.int64) * 64).sum())
    rp, rx, ry, rz = ryo.direct_targets_f64(torch.arange(0, n, 37, device="cuda"), *t)
    a = torch.stack(out[1:])[:, ::37].double()
    r = torch.stack([rx, ry, rz])
    err = ((a - r).norm(dim=0) / r.norm(dim=0)).cpu().numpy()
    assert np.percentile(err, 99) < 1e-5 and err.max() < 1e-4


def test_long_groups_of_a_large_solve():
    """more than 49,152 groups: the longest ones leave the fused kernel and go through lists"""
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    n = 3200007
    p = ds.plummer(n, seed=4, velocities=False)
    ctx = ryo.Context()
    res, t, out = _solve(p, ryo.SolveParams(theta=0.5), ctx)
    arr = ryo.solve_arrays(ctx)
    assert res.num_groups > 49152
    g = host(arr["groups"]).view(np.uint32).astype(np.int64)
    p2p, m2p = host(arr["groupP2P"]).astype(np.int64), host(arr["groupM2P"]).astype(np.int64)
    sizes = np.diff(g)
    assert res.sum_p2p == int((p2p * sizes).sum()) and res.sum_m2p == int((m2p * sizes).sum())
    heavy = np.flatnonzero(p2p + 2 * m2p > 32768)
    assert 1 <= len(heavy) < len(p2p)
    pick = np.concatenate([np.arange(g[k], g[k + 1]) for k in heavy[:16]] + [np.arange(0, n, 9973)])
    rp, rx, ry, rz = ryo.direct_targets_f64(torch.from_numpy(pick).cuda(), *t)
    a = torch.stack(out[1:])[:, torch.from_numpy(pick).cuda()].double()
    r = torch.stack([rx, ry, rz])
    err = ((a - r).norm(dim=0) / r.norm(dim=0)).cpu().numpy()
    assert np.percentile(err, 99) < 1e-3 and np.median(err) < 2e-4  # the expansions' error at theta 0.5


def _double_rule(groups, x, y, z, m, h, tree, layout, centers, mp, shells, L):
    """the traversal's rule and sums in numpy float64: per group (cells, bodies) and per body (-phi, ax, ay, az)"""
    child, leaf = tree["childOffsets"], tree["internalToLeaf"]
    pos, out, cells, bodies = np.stack([x, y, z], 1), np.zeros((len(x), 4)), [], []
    for b, e in zip(groups[:-1], groups[1:]):
        t = pos[b:e]
        lo, hi = t.min(0), t.max(0)
        tc, ts, nM, nP, acc = (hi + lo) * 0.5, (hi - lo) * 0.5, 0, 0, np.zeros((e - b, 4))
        for k in np.ndindex(*(2 * shells + 1,) * 3):
            sh = (np.array(k[::-1]) - shells) * L
            tc = tc + sh
            front, at = np.arange(1, 9), t + sh
            while len(front):
                d = np.maximum(np.abs(tc - centers[front, :3]) - ts, 0.0)
                close = (d * d).sum(1) < centers[front, 3]
                node = child[front] != 0
                count = np.where(node, 1, layout[leaf[front] + 1] - layout[leaf[front]])
                far = front[~close | (~node & (count == 0) & (centers[front, 3] != 0))]
                nM += len(far)
                for c in far:
                    r = at - centers[c, :3]
                    q, i1 = mp[c], 1 / np.sqrt((r * r).sum(1))
                    Q = np.array([[q[1], q[2], q[3]], [q[2], q[4], q[5]], [q[3], q[5], q[6]]])
                    Qr = r @ Q
                    rQr = (r * Qr).sum(1)
                    acc[:, 0] += q[0] * i1 + 0.5 * i1 ** 5 * rQr
                    acc[:, 1:] += i1[:, None] ** 5 * Qr - ((2.5 * rQr * i1 ** 5 + q[0] * i1) * i1 * i1)[:, None] * r
                for c in front[close & ~node & (count > 0)]:
                    s = slice(layout[leaf[c]], layout[leaf[c] + 1])
                    nP += s.stop - s.start
                    d = pos[None, s] - at[:, None]
                    r2 = (d * d).sum(2)
                    w = m[None, s] / np.maximum(r2, (h[b:e, None] + h[None, s]) ** 2) ** 1.5
                    acc[:, 0] += (w * r2).sum(1)
                    acc[:, 1:] += (w[:, :, None] * d).sum(1)
                front = (child[front[close & node]][:, None] + np.arange(8)).ravel()
            tc = tc - sh
        cells.append(nM)
        bodies.append(nP)
        out[b:e] = acc
    return np.array(cells), np.array(bodies), out


# a partial group, whole and ragged groups, softenings beyond and within the pairs' distances, replicas
@pytest.mark.parametrize("kind", ["f64", "mixed"])
@pytest.mark.parametrize("n,bucket,eps,shells", [(70, 8, 0.01, 0), (1000, 16, 1e-6, 0), (2051, 8, 0.2, 0),
                                                 (640, 16, 0.01, 1)])
def test_double_lists_against_numpy(kind, n, bucket, eps, shells):
    import ryoanji_b200 as ryo
    rng = np.random.default_rng(n)
    real = torch.float64 if kind == "f64" else torch.float32
    x, y, z = (dev(rng.uniform(-1, 1, n)) for _ in range(3))
    tb, box = ryo.TreeBuilder(bucket), ryo.Box.cube(-1.0, 1.0)
    nn = tb.update(x, y, z, box)
    m, h = dev(rng.uniform(0.5, 1.5, n) / n).to(real), dev(rng.uniform(0.5, 1.5, n) * eps).to(real)
    centers = torch.zeros(nn, 4, device="cuda", dtype=torch.float64)
    mp = torch.zeros(nn, 8, device="cuda", dtype=real)
    ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
    ryo.upsweep_centers(tb.maxTreeLevel, tb.levelRange, tb.childOffsets(), centers)
    ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
    for level in range(tb.maxTreeLevel - 1, -1, -1):
        ryo.upsweep_multipoles(tb.levelRange[level], tb.levelRange[level + 1], tb.childOffsets(), centers, mp)
    ryo.set_mac(tb.nodeKeys(), centers, 2.0, box)
    groups = ryo.compute_fixed_groups(0, n, 64)
    out = [torch.zeros(n, device="cuda", dtype=real) for _ in range(4)]
    pot, gm, gp = ryo.traverse(groups, 1, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(), tb.internalToLeaf(),
                               tb.layout(), centers, mp, 1.0, shells, box.lengths, *out, group_counts=True)
    X, Y, Z, M, H, C, Q = (host(a).astype(np.float64) for a in (x, y, z, m, h, centers, mp))
    tree = dict(childOffsets=host(tb.childOffsets()), internalToLeaf=host(tb.internalToLeaf()))
    cells, bodies, acc = _double_rule(host(groups), X, Y, Z, M, H, tree, host(tb.layout()), C, Q, shells, 2.0)
    assert np.array_equal(host(gm), cells) and np.array_equal(host(gp), bodies)
    # the single-precision rsqrt enters every term with up to 2 ulp, five times in a quadrupole's
    scale = np.maximum(np.linalg.norm(acc[:, 1:], axis=1), 0.25 * (1 + 26 * shells))
    err = np.linalg.norm(np.stack([host(a) for a in out[1:]], 1) - acc[:, 1:], axis=1) / scale
    assert err.max() < 3e-6
    assert np.allclose(host(out[0]), -M * acc[:, 0], rtol=2e-6)
    assert pot == pytest.approx(-0.5 * float((M * acc[:, 0]).sum()), rel=2e-6)
