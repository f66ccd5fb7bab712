"""The packed float direct sum at the edges of its blocks, tiles and splits, against float64 sums on the CPU."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(first, last, x, y, z, m, h, shells, L):
    X, Y, Z, M, H = (torch.from_numpy(a).double() for a in (x, y, z, m, h))
    t = slice(first, last)
    out, mag = torch.zeros(4, last - first, dtype=torch.float64), torch.zeros(last - first, dtype=torch.float64)
    for k in np.ndindex(*(2 * shells + 1,) * 3):
        s = [(i - shells) * l for i, l in zip(k, L)]
        d = [V[None, :] - (V[t, None] + o) for V, o in zip((X, Y, Z), s)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        w = M[None, :] / torch.maximum(r2, (H[t, None] + H[None, :]) ** 2) ** 1.5
        out[0] -= M[t] * (w * r2).sum(1)
        for c in range(3):
            out[1 + c] += (w * d[c]).sum(1)
        mag += (w.abs() * r2.sqrt()).sum(1)
    return out, mag


# targets around a block of 256 and its share per split, sources around a tile of 128 and eight splits of it, an offset
# first target, replicas, one softening or many, and one whose square is no normal float
@pytest.mark.parametrize("n,first,last", [(1, 0, 1), (127, 0, 127), (128, 3, 128), (129, 0, 129), (255, 0, 255),
                                          (257, 0, 257), (1000, 700, 957), (2049, 0, 2049), (5000, 1, 515)])
@pytest.mark.parametrize("soft,shells", [("one", 0), ("many", 0), ("one", 1), ("tiny", 0)])
def test_packed_direct_sum(n, first, last, soft, shells):
    import ryoanji_b200 as ryo
    rng = np.random.default_rng(n + first)
    x, y, z = (rng.uniform(-1, 1, n).astype(np.float32) for _ in range(3))
    m = (rng.uniform(-0.5, 1.5, n) / n).astype(np.float32)
    h = {"one": np.full(n, 0.02), "many": rng.uniform(0.0, 0.05, n), "tiny": np.full(n, 3e-20)}[soft].astype(np.float32)
    base = 0.5
    if soft == "tiny":  # a body's own term, m / h^3 times zero, stays finite
        m, base = (m * np.float32(1e-20)).astype(np.float32), 0.0
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z, m, h)]
    out = [torch.full((n,), base, device="cuda") for _ in range(4)]  # the sums are added to the outputs
    L = (2.0, 2.5, 3.0)
    ryo.direct_sum(first, last, n, L, shells, *dev, *out)
    got = torch.stack(out).cpu().double() - base
    assert (got[:, :first] == 0).all() and (got[:, last:] == 0).all()
    ref, mag = _exact(first, last, x, y, z, m, h, shells, L)
    # the result's rounding beside 0.5, and each term's: rsqrt to 2 ulp cubed, distances and products
    bound = 1e-6 * mag + 1.2e-7 * base
    for c in range(1, 4):
        assert ((got[c, first:last] - ref[c]).abs() <= bound).all(), c
    # (of the tiny set m phi is a denormal, a multiple of 1.4e-45)
    assert ((got[0, first:last] - ref[0]).abs() <= 1e-6 * ref[0].abs().max() + 1.2e-7 * base + 1.4e-45).all()
