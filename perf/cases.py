"""The work that programs give this library, as measurable cases: one-call solves of one system (small, ordinary and
large; open, periodic, with signed masses), solves from and to host memory, batches of systems, the served stream, the
reference's step-by-step flow in its two double type sets, and direct sums.

listed() holds the fixed cases and draw() more of the same ranges; prepare() makes a case's inputs on the GPU from a
seed, run() is one pass through the public API, work() the bytes and operations of a pass, and exact() the result in
64 bits from plain torch (all-pairs sums, so the tree's own expansion error shows in the difference).
"""
import math

import numpy as np
import torch

import ryoanji_b200 as ryo
from ryoanji_b200 import datasets as ds

#: largest number of body pairs exact() sums
MAX_PAIRS = 7.5e10


def listed():
    return [
        # one small cluster per call: a user's inner loop over small systems, bound by latency and launches
        dict(name="plummer_4k", kind="solve", set="plummer", n=4096, bucket=32, theta=0.5, moving=False),
        # one step of a star-cluster simulation: an odd body count, velocities carried along with the bodies
        dict(name="plummer_60k_moving", kind="solve", set="plummer", n=60001, bucket=32, theta=0.5, moving=True),
        # an ordinary sphere with a dense centre and sparse outskirts
        dict(name="plummer_1m", kind="solve", set="plummer", n=1 << 20, bucket=64, theta=0.5, moving=False),
        # the benchmark's cube: the largest system of one call
        dict(name="cube_64m", kind="solve", set="cube", n=1 << 26, bucket=64, theta=0.5, moving=False),
        # charges of both signs with monopole + dipole + quadrupole expansions and a strict opening angle
        dict(name="signed_mdq_100k", kind="solve", set="signed", n=100003, bucket=64, theta=0.2, moving=False),
        # a cosmological box: replica shells and the Ewald correction
        dict(name="periodic_256k", kind="solve", set="periodic", n=1 << 18, bucket=64, theta=0.5, moving=False),
        # a host program's bodies in pinned memory, solved and returned there
        dict(name="host_cube_4m", kind="host", set="cube", n=1 << 22, bucket=64, theta=0.5),
        # an ensemble of independent clusters in one call
        dict(name="ensemble_256", kind="batch", systems=256, lo=10.0, hi=15.0, mix=0, bucket=32, theta=0.5),
        # the served stream: requests of mixed kinds and sizes, leapfrog steps, final states back to the host
        dict(name="served_10", kind="served", requests=10, lo=11.0, hi=16.0, mix=3, steps=4, bucket=64, theta=0.5),
        # the reference's own call sequence with double coordinates, double everything
        dict(name="steps_f64_120k", kind="steps", set="plummer", precision="f64", n=120001, bucket=64, theta=0.5),
        # the same with float masses, multipoles and outputs
        dict(name="steps_mixed_250k", kind="steps", set="cube", precision="mixed", n=250000, bucket=64, theta=0.5),
        # all-pairs sums, the check that users of a tree code run
        dict(name="direct_40k", kind="direct", set="plummer", n=40001),
    ]


def draw(rng):
    def log2n(lo, hi):
        return int(round(2.0 ** rng.uniform(lo, hi)))

    kind = rng.choice(["solve", "solve", "solve", "solve", "host", "batch", "served", "steps", "steps", "direct"])
    bucket = rng.choice([16, 32, 64, 64])
    theta = round(rng.uniform(0.4, 0.7), 3)
    if kind == "solve":
        what = rng.choice(["plummer", "plummer", "cube", "signed", "periodic", "halos"])
        hi = {"plummer": 23.0, "cube": 24.0, "signed": 18.0, "periodic": 20.0, "halos": 21.0}[what]
        return dict(kind=kind, set=what, n=log2n(10.0, hi), bucket=bucket, theta=theta, moving=rng.random() < 0.4)
    if kind == "host":
        return dict(kind=kind, set=rng.choice(["cube", "plummer"]), n=log2n(12.0, 23.0), bucket=bucket, theta=theta)
    if kind == "batch":
        return dict(kind=kind, systems=rng.randint(9, 300), lo=9.0, hi=round(rng.uniform(12.0, 15.0), 2),
                    mix=rng.randint(1, 1000), bucket=bucket, theta=theta)
    if kind == "served":
        return dict(kind=kind, requests=rng.randint(2, 12), lo=10.0, hi=round(rng.uniform(13.0, 16.0), 2),
                    mix=rng.randint(4, 1000), steps=rng.randint(1, 4), bucket=bucket, theta=theta)
    if kind == "steps":
        return dict(kind=kind, set=rng.choice(["cube", "plummer"]), precision=rng.choice(["f64", "mixed"]),
                    n=log2n(11.0, 19.0), bucket=bucket, theta=theta)
    return dict(kind=kind, set=rng.choice(["cube", "plummer"]), n=log2n(8.0, 16.5))


# ------------------------------------------------------------------------------------------------------- inputs

def _rand(n, gen, lo, hi):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _bodies(what, n, seed):
    """x, y, z, vx, vy, vz, m, h of one system (float64 device tensors)"""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    zero = torch.zeros(n, device="cuda", dtype=torch.float64)
    m = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    h = torch.full((n,), 1e-6, device="cuda", dtype=torch.float64)
    if what == "plummer":
        x, y, z, vx, vy, vz = ds.plummer_device(torch.ones(n, device="cuda", dtype=torch.float64), gen)
        return x, y, z, vx, vy, vz, m, torch.full_like(h, 0.005)
    if what == "halos":  # eight clumps of different masses and sizes, per-body masses and softenings
        k = torch.randint(0, 8, (n,), generator=gen, device="cuda")
        centers = torch.rand(8, 3, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
        scale = 0.02 * (1 + k)
        x, y, z = (centers[k, d] + scale * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
                   for d in range(3))
        return x, y, z, zero, zero, zero, m * _rand(n, gen, 0.5, 1.5), 1e-4 * _rand(n, gen, 1.0, 2.0)
    if what == "signed":
        x, y, z = ((0.2 * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)).clamp(-1, 1)
                   for _ in range(3))
        return x, y, z, zero, zero, zero, m * (torch.randint(0, 2, (n,), generator=gen, device="cuda") * 2 - 1), h
    lo, hi = (0.0, 1.0) if what == "periodic" else (-1.0, 1.0)
    x, y, z = (_rand(n, gen, lo, hi) for _ in range(3))
    if what == "periodic":
        x, y, z = (v.clamp_max(float(np.nextafter(np.float32(1), np.float32(0)))) for v in (x, y, z))
    return x, y, z, zero, zero, zero, m, h


def _rows(rows, n, dtype=torch.float32):
    """a (rows, n) block whose rows all start on a 256-byte boundary"""
    return torch.zeros(rows, -(-n // 64) * 64, device="cuda", dtype=dtype)[:, :n]


def _box(what):
    if what in ("cube", "signed"):
        return ryo.Box.cube(-1.0, 1.0)
    if what == "periodic":
        return ryo.Box.cube(0.0, 1.0, ryo.BOUNDARY_PERIODIC)
    return None  # the cube around the bodies


def _params(case, box=None):
    return ryo.SolveParams(theta=case["theta"], bucket_size=case["bucket"], group_size=64, box=box,
                           multipole="mdq" if case.get("set") == "signed" else "quadrupole")


def _systems(case):
    return ds.ensemble_sizes(case["systems"], seed=case["mix"], lo_log2=case["lo"], hi_log2=case["hi"])


def _requests(case, seed):
    reqs = ds.served_requests(case["requests"], seed=case["mix"], lo_log2=case["lo"], hi_log2=case["hi"])
    for k, r in enumerate(reqs):
        r["steps"] = 1 + (r["steps"] - 1) % case["steps"]
        r["seed"] = 1000 * int(seed) + k
    return reqs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        b = _bodies(case["set"], case["n"], seed)
        given = _rows(8, case["n"])
        for row, v in zip(given, (b[0], b[1], b[2], b[6], b[7], b[3], b[4], b[5])):
            row.copy_(v)
        given = given if case["moving"] else given[:5]
        return dict(case=case, given=given, work=_rows(len(given), case["n"]), out=_rows(4, case["n"]),
                    order=torch.zeros(case["n"], device="cuda", dtype=torch.int32),
                    params=_params(case, _box(case["set"])))
    if kind == "host":
        b = _bodies(case["set"], case["n"], seed)
        pin = lambda v: v.float().cpu().pin_memory()  # noqa: E731
        return dict(case=case, bodies=[pin(b[k]) for k in (0, 1, 2, 6, 7)],
                    out=[torch.zeros(case["n"]).pin_memory() for _ in range(4)],
                    order=torch.zeros(case["n"], dtype=torch.int32).pin_memory(),
                    params=_params(case, _box(case["set"])))
    if kind == "batch":
        sizes, radii = _systems(case)
        x, y, z, m, h, *_ = ds.plummer_ensemble(sizes, radii, seed=int(seed))
        n = int(sizes.sum())
        given = _rows(5, n)
        for row, v in zip(given, (x, y, z, m, h)):
            row.copy_(v)
        return dict(case=case, given=given, work=_rows(5, n), out=_rows(4, n),
                    order=torch.zeros(n, device="cuda", dtype=torch.int32),
                    systems=[ryo.BatchSystem(int(k)) for k in sizes], params=_params(case))
    if kind == "served":
        reqs = _requests(case, seed)
        for r in reqs:
            r["bodies"] = [v.cpu().pin_memory() for v in ds.request_bodies(r)]
            r["out"] = torch.zeros(10, r["n"]).pin_memory()
        engine = ryo.Engine(_params(case), reserve_bodies=sum(r["n"] for r in reqs))
        return dict(case=case, requests=reqs, engine=engine)
    if kind == "steps":
        b = _bodies(case["set"], case["n"], seed)
        real = torch.float64 if case["precision"] == "f64" else torch.float32
        given = _rows(3, case["n"], torch.float64)
        for row, v in zip(given, b[:3]):
            row.copy_(v)
        box = ryo.Box.cube(-50.0, 50.0) if case["set"] == "plummer" else ryo.Box.cube(-1.0, 1.0)
        return dict(case=case, given=given, work=_rows(3, case["n"], torch.float64), m=b[6].to(real), h=b[7].to(real),
                    out=_rows(4, case["n"], real), box=box, builder=ryo.TreeBuilder(case["bucket"]), real=real)
    b = _bodies(case["set"], case["n"], seed)
    return dict(case=case, bodies=[b[k].float() for k in (0, 1, 2, 6, 7)], out=_rows(4, case["n"]))


# ------------------------------------------------------------------------------------------------------- passes

def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("solve", "batch"):
        work, out = state["work"], state["out"]
        work.copy_(state["given"])  # the call sorts its inputs in place
        x, y, z, m, h = work[:5]
        if kind == "solve":
            v = tuple(work[5:]) if case["moving"] else None
            r = ryo.solve(x, y, z, m, h, *out, params=state["params"], v=v, order=state["order"])
            energy = r.potential_energy
        else:
            b = ryo.solve_batch(state["systems"], x, y, z, m, h, *out, params=state["params"], order=state["order"])
            r, energy = b.stats, np.array(b.energies, np.float32)
        return dict(bodies=work, field=out, order=state["order"], energy=energy, p2p=r.sum_p2p, m2p=r.sum_m2p)
    if kind == "host":
        r = ryo.solve_host(*state["bodies"], *state["out"], params=state["params"], order=state["order"])
        return dict(field=state["out"], order=state["order"], energy=r.potential_energy, p2p=r.sum_p2p,
                    m2p=r.sum_m2p)
    if kind == "served":
        engine = state["engine"]
        for r in state["requests"]:
            periodic = r["kind"] == "periodic"
            box = ryo.Box.cube(0.0, 1.0, ryo.BOUNDARY_PERIODIC) if periodic else None
            engine.submit(r["tag"], *r["bodies"], box=box, steps=r["steps"], dt=r["dt"], want_output=True,
                          out=r["out"])
        done = {}
        while len(done) < len(state["requests"]):
            engine.step()
            for d in engine.poll():
                done[d["tag"]] = d["state"]
        return dict(states=done)
    if kind == "steps":
        work, out, m, h, box = state["work"], state["out"], state["m"], state["h"], state["box"]
        tb, real = state["builder"], state["real"]
        work.copy_(state["given"])
        x, y, z = work
        nodes = tb.update(x, y, z, box)
        centers = torch.zeros(nodes, 4, device="cuda", dtype=torch.float64)
        mp = torch.zeros(nodes, 8, device="cuda", dtype=real)
        ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
        levels = tb.levelRange
        ryo.upsweep_centers(tb.maxTreeLevel, levels, tb.childOffsets(), centers)
        ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
        for level in range(tb.maxTreeLevel - 1, -1, -1):
            ryo.upsweep_multipoles(levels[level], levels[level + 1], tb.childOffsets(), centers, mp)
        ryo.set_mac(tb.nodeKeys(), centers, 1.0 / case["theta"], box)
        groups = ryo.compute_fixed_groups(0, case["n"], ryo.bh_max_target_size())
        out.zero_()
        pot = ryo.traverse(groups, 1 if nodes > 1 else 0, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(),
                           tb.internalToLeaf(), tb.layout(), centers, mp, 1.0, 0, box.lengths, *out)
        return dict(bodies=work, field=out, energy=pot, order=tb.order(),
                    stats=np.array(ryo.read_bh_stats()[:4], np.int64))
    out = state["out"]
    out.zero_()
    x, y, z, m, h = state["bodies"]
    ryo.direct_sum(0, case["n"], case["n"], (0.0, 0.0, 0.0), 0, x, y, z, m, h, *out)
    return dict(field=out)


# ------------------------------------------------------------------------------------------------------- work

def _solve_flops(n, bucket, theta):
    """operations of one tree evaluation, 23 per direct pair and 65 per cell (the reference's counting): about 60
    buckets of direct bodies and 70 cells per doubling of the leaf count at theta 0.5, as (1 / theta)^3"""
    open_ = (0.5 / theta) ** 3
    pairs = min(n, 60 * bucket * open_)
    cells = 70 * max(0.0, math.log2(n / bucket)) * open_
    return n * (23.0 * pairs + 65.0 * min(cells, n / bucket))


def work(case):
    kind = case["kind"]
    if kind in ("solve", "host"):
        n = case["n"]
        replicas = 4 if case["set"] == "periodic" else 1
        return dict(bytes=n * (4.0 * (5 + 5 + 4 + 1 + (6 if case.get("moving") else 0))),
                    flops=replicas * _solve_flops(n, case["bucket"], case["theta"]))
    if kind == "batch":
        sizes = _systems(case)[0]
        return dict(bytes=60.0 * int(sizes.sum()),
                    flops=sum(_solve_flops(int(k), case["bucket"], case["theta"]) for k in sizes))
    if kind == "served":
        reqs = _requests(case, 0)
        return dict(bytes=sum((32.0 + 40.0) * r["n"] for r in reqs),
                    flops=sum((r["steps"] + 1) * _solve_flops(r["n"], case["bucket"], case["theta"]) for r in reqs))
    n = case["n"]
    if kind == "steps":
        real = 8 if case["precision"] == "f64" else 4
        return dict(bytes=n * (48.0 + 6.0 * real + 4.0), flops=_solve_flops(n, case["bucket"], case["theta"]))
    return dict(bytes=36.0 * n, flops=23.0 * n * n)


# ------------------------------------------------------------------------------------------------------- exact

def _field(x, y, z, m, h):
    """m phi and acceleration of every body, all pairs in float64 (softening: distances below h_i + h_j count as it)"""
    n = x.numel()
    out = torch.empty(4, n, device=x.device, dtype=torch.float64)
    step = max(1, (1 << 26) // n)
    for a in range(0, n, step):
        t = slice(a, min(n, a + step))
        dx, dy, dz = (v[None, :] - v[t, None] for v in (x, y, z))
        r2 = dx * dx + dy * dy + dz * dz
        w = torch.maximum(r2, (h[None, :] + h[t, None]) ** 2).rsqrt_().pow_(3).mul_(m[None, :])
        out[0, t] = -m[t] * r2.mul_(w).sum(1)
        for k, d in enumerate((dx, dy, dz)):
            out[1 + k, t] = d.mul_(w).sum(1)
    return out


def _hilbert_keys(x, y, z, limits):
    """63-bit Hilbert keys of points in a cubic box, in the coordinates' own type"""
    cells = []
    for v, lo, hi in zip((x, y, z), limits[0::2], limits[1::2]):
        one = torch.ones((), device=v.device, dtype=v.dtype)
        lo, hi = one * lo, one * hi
        scale = (one / (hi - lo)) * (1 << 21)
        a, b = v * scale, lo * scale
        c = (a.floor() - b.floor()).long() - ((a - a.floor()) < (b - b.floor())).long()
        cells.append(c.clamp(0, (1 << 21) - 1))
    px, py, pz = cells
    digit = torch.tensor([0, 1, 3, 2, 7, 6, 4, 5], device=x.device)
    key = torch.zeros_like(px)
    for level in range(20, -1, -1):
        bx, by, bz = ((p >> level) & 1 for p in (px, py, pz))
        key = key * 8 + digit[4 * bx + 2 * by + bz]
        ny, nz = 1 - by, 1 - bz
        px = px ^ -(bx & (ny | bz))
        py = py ^ -((bx & (by | bz)) | (by & nz))
        pz = pz ^ -((bx & ny & nz) | (by & nz))
        turn, swap = bz == 1, (bz == 0) & (by == 0)
        px, py, pz = (torch.where(turn, py, torch.where(swap, pz, px)), torch.where(turn, pz, py),
                      torch.where(turn, px, torch.where(swap, px, pz)))
    return key


def _sorted(x, y, z, limits):
    if limits is None:  # the cube around the bodies, lower corner at the minimum
        lo = [float(v.min()) for v in (x, y, z)]
        ext = max(float(v.max()) - a for v, a in zip((x, y, z), lo))
        limits = []
        for v, a in zip((x, y, z), lo):
            top = np.float32(a + ext)
            limits += [a, float(top if top >= float(v.max()) else np.nextafter(top, np.float32(3e38)))]
    return torch.sort(_hilbert_keys(x, y, z, limits), stable=True).indices


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "host"):
        if case["set"] == "periodic" or float(case["n"]) ** 2 > MAX_PAIRS:
            return None
        b = _bodies(case["set"], case["n"], seed)
        x, y, z, m, h = (b[k].float() for k in (0, 1, 2, 6, 7))
        box = _box(case["set"])
        o = _sorted(x, y, z, box.limits if box else None)
        f = _field(*(v[o].double() for v in (x, y, z, m, h)))
        energy = 0.5 * float(f[0].sum())
        if kind == "host":
            return dict(field=[f[k] for k in range(4)], order=None, energy=energy, p2p=None, m2p=None)
        moving = [b[k].float() for k in (3, 4, 5)] if case["moving"] else []
        return dict(bodies=torch.stack([v[o] for v in [x, y, z, m, h] + moving]).double(), field=f, order=None,
                    energy=None if case["set"] == "signed" else energy, p2p=None, m2p=None)
    if kind == "batch":
        sizes, radii = _systems(case)
        if float((sizes.astype(np.float64) ** 2).sum()) > MAX_PAIRS:
            return None
        bodies = ds.plummer_ensemble(sizes, radii, seed=int(seed))[:5]
        parts, fields, first = [], [], 0
        for k in sizes:
            one = [v[first:first + int(k)] for v in bodies]
            o = _sorted(one[0], one[1], one[2], None)
            parts.append(torch.stack([v[o] for v in one]).double())
            fields.append(_field(*parts[-1]))
            first += int(k)
        energy = np.array([0.5 * float(f[0].sum()) for f in fields])
        return dict(bodies=torch.cat(parts, 1), field=torch.cat(fields, 1), order=None, energy=energy, p2p=None,
                    m2p=None)
    if kind == "served":
        reqs = _requests(case, seed)
        if sum((r["steps"] + 1) * float(r["n"]) ** 2 for r in reqs) > MAX_PAIRS:
            return None
        states = {}
        for r in reqs:
            if r["kind"] == "periodic":
                states[r["tag"]] = None
                continue
            x, y, z, m, h, vx, vy, vz = (v.double() for v in ds.request_bodies(r))
            pos, vel, half = torch.stack([x, y, z]), torch.stack([vx, vy, vz]), 0.5 * float(np.float32(r["dt"]))
            f = _field(*pos, m, h)
            for _ in range(r["steps"]):
                vel += half * f[1:]
                pos += 2 * half * vel
                f = _field(*pos, m, h)
                vel += half * f[1:]
            states[r["tag"]] = torch.cat([pos, vel, f[1:], f[:1]])
        return dict(states=states)
    if float(case["n"]) ** 2 > MAX_PAIRS:
        return None
    b = _bodies(case["set"], case["n"], seed)
    if kind == "steps":
        real = torch.float64 if case["precision"] == "f64" else torch.float32
        side = 50.0 if case["set"] == "plummer" else 1.0
        o = _sorted(b[0], b[1], b[2], [-side, side] * 3)
        x, y, z = (v[o] for v in b[:3])
        f = _field(x, y, z, b[6].to(real).double(), b[7].to(real).double())
        return dict(bodies=torch.stack([x, y, z]), field=f, energy=0.5 * float(f[0].sum()), order=None, stats=None)
    return dict(field=_field(*(b[k].float().double() for k in (0, 1, 2, 6, 7))))
