"""Stack capacities accepted and refused: up to what four warps' stacks of the fused kernels hold, in every form of the
traversal; none of them changes the results, and a refused call leaves no error behind for the next one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# lists with divided and with whole walks, the fused kernel
@pytest.mark.parametrize("n,group", [(3000, 64), (60000, 8), (60000, 1)])
def test_float_limits(n, group):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = ds.plummer(n, seed=n, velocities=False)
    ctx = ryo.Context()

    def run(capacity):
        out = torch.empty(4, n, device="cuda")
        ryo.solve(*(torch.from_numpy(a).cuda() for a in (p.x, p.y, p.z, p.m, p.h)), *out,
                  ryo.SolveParams(group_size=group, stack_capacity=capacity), ctx=ctx)
        return out
    base = run(0)
    for capacity in (1025, 12285, 12344):
        assert torch.equal(run(capacity), base)
    for capacity in (12345, 13200, 1 << 20, (1 << 31) - 1):
        with pytest.raises(ryo.RyoError) as e:
            run(capacity)
        assert e.value.status == 2
    assert torch.equal(run(0), base)


@pytest.mark.parametrize("real", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,group", [(3000, 64), (60000, 1)])
def test_double_limits(real, n, group):
    import ryoanji_b200 as ryo
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x, y, z = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) for _ in range(3))
    tb, box = ryo.TreeBuilder(64), ryo.Box.cube(0.0, 1.0)
    nn = tb.update(x, y, z, box)
    m, h = torch.ones(n, device="cuda", dtype=real), torch.full((n,), 1e-3, device="cuda", dtype=real)
    centers = torch.zeros(nn, 4, device="cuda", dtype=torch.float64)
    mp = torch.zeros(nn, 8, device="cuda", dtype=real)
    ryo.compute_leaf_source_center(x, y, z, m, tb.leafToInternal(), tb.layout(), centers)
    ryo.upsweep_centers(tb.maxTreeLevel, tb.levelRange, tb.childOffsets(), centers)
    ryo.compute_leaf_multipoles(x, y, z, m, tb.leafToInternal(), tb.layout(), centers, mp)
    for level in range(tb.maxTreeLevel - 1, -1, -1):
        ryo.upsweep_multipoles(tb.levelRange[level], tb.levelRange[level + 1], tb.childOffsets(), centers, mp)
    ryo.set_mac(tb.nodeKeys(), centers, 2.0, box)
    groups = torch.arange(0, n + 1, group, device="cuda", dtype=torch.int32)
    if int(groups[-1]) < n:
        groups = torch.cat([groups, torch.tensor([n], device="cuda", dtype=torch.int32)])

    def run(capacity):
        out = [torch.zeros(n, device="cuda", dtype=real) for _ in range(4)]
        ryo.traverse(groups, 1, x, y, z, m, h, x, y, z, m, h, tb.childOffsets(), tb.internalToLeaf(), tb.layout(),
                     centers, mp, 1.0, 0, box.lengths, *out, stack_capacity=capacity)
        return torch.stack(out)
    base = run(0)
    for capacity in (1025, 12993, 13120):
        assert torch.equal(run(capacity), base)
    for capacity in (13121, 14000):
        with pytest.raises(ryo.RyoError) as e:
            run(capacity)
        assert e.value.status == 2
    assert np.isfinite(base.cpu().numpy()).all()
