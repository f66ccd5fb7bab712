"""Direct sums of bodies with NaN or infinite values follow IEEE arithmetic term by term, as the plain formula in
float64 does; and the potential may be left out in either type."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _formula(x, y, z, m, h):
    d = [v[None, :] - v[:, None] for v in (x, y, z)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    hh = (h[:, None] + h[None, :]) ** 2
    w = torch.where(r2 < hh, hh, r2).rsqrt()
    w = m[None, :] * w * (w * w)
    return torch.stack([-m * (w * r2).sum(1)] + [(w * v).sum(1) for v in d])


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
@pytest.mark.parametrize("what,value", [(None, 0.0), (0, np.nan), (1, np.inf), (3, np.nan), (3, np.inf), (3, -np.inf),
                                        (4, np.nan), (4, np.inf), (4, -0.02), (4, 0.5)])
def test_special_values(real, what, value):
    import ryoanji_b200 as ryo
    rng = np.random.default_rng(4)
    n = 300
    b = [rng.uniform(-1, 1, n) for _ in range(3)] + [rng.uniform(0.5, 1.5, n) / n, np.full(n, 0.02)]
    if what is not None:
        b[what][130] = value
    b = [torch.from_numpy(v).to(real) for v in b]
    out = torch.zeros(4, n, dtype=real, device="cuda")
    ryo.direct_sum(0, n, n, (0.0, 0.0, 0.0), 0, *(v.cuda() for v in b), *out)
    ref, got = _formula(*(v.double() for v in b)), out.cpu().double()
    assert torch.equal(got.isnan(), ref.isnan())
    inf = ref.isinf()
    assert torch.equal(got.isinf(), inf) and torch.equal(got[inf], ref[inf])
    ok = ref.isfinite()
    if ok.any():  # terms of up to m / h^2, each to a few ulp
        assert float((got - ref)[ok].abs().max()) <= 1e-6 * float(ref[ok].abs().max())


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
def test_no_potential(real):
    import ryoanji_b200 as ryo
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    n = 500
    b = [torch.rand(n, generator=gen, device="cuda", dtype=real) for _ in range(4)] + [
        torch.full((n,), 0.01, device="cuda", dtype=real)]
    out = [torch.zeros(4, n, device="cuda", dtype=real) for _ in range(2)]
    ryo.direct_sum(0, n, n, (0.0, 0.0, 0.0), 0, *b, *out[0])
    ryo.direct_sum(0, n, n, (0.0, 0.0, 0.0), 0, *b, None, *out[1][1:])
    assert torch.equal(out[0][1:], out[1][1:])
