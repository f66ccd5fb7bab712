"""The Ewald correction of more groups than their warps' threads can be numbered in 32 bits: single targets as groups,
against the same targets in groups of 64. A target's correction does not depend on its group."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_than_2_to_the_26_groups():
    import ryoanji_b200 as ryo
    n = (1 << 26) + 67
    gen = torch.Generator(device="cuda")
    gen.manual_seed(8)
    x, y, z = (torch.rand(n, generator=gen, device="cuda") for _ in range(3))
    m = torch.ones(n, device="cuda")
    box = ryo.Box.cube(0.0, 1.0, ryo.BOUNDARY_PERIODIC)
    root = [1.0, 0.1, 0.02, 0.03, 0.2, 0.01, 0.3, 0.6]
    few = ryo.EwaldSettings(numReplicaShells=0, lCut=0.1, hCut=1.0, alpha_scale=2.0)  # an image or two, six waves
    out = []
    for groups in (torch.arange(n + 1, device="cuda", dtype=torch.int32), ryo.compute_fixed_groups(0, n, 64)):
        f = torch.zeros(4, n, device="cuda")
        e = ryo.compute_gravity_ewald([0.5, 0.5, 0.5], root, groups, x, y, z, m, box, 1.0, *f, settings=few)
        out.append((f, e))
    assert torch.equal(out[0][0], out[1][0]) and bool((out[0][0] != 0).any(0).all())
    assert out[0][1] == pytest.approx(out[1][1], rel=1e-9)
