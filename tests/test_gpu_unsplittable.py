"""A single target that overflows the traversal stack has no result: solves that store their results leave zeros there,
not what the caller's arrays held before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bodies(n, seed):
    from ryoanji_b200 import datasets as ds
    p = ds.plummer(n, seed=seed, velocities=False)
    return [torch.from_numpy(a).cuda() for a in (p.x, p.y, p.z, p.m, p.h)]


def _check(out):
    p, a = out[0], torch.stack(out[1:])
    assert torch.isfinite(p).all() and torch.isfinite(a).all()
    zero = (p == 0) & (a == 0).all(0)
    assert zero.any()
    return zero


@pytest.mark.parametrize("n", [2000, 30011])
def test_solve_leaves_zeros(n):
    import ryoanji_b200 as ryo
    out = [torch.full((n,), float("nan"), device="cuda") for _ in range(4)]
    with pytest.raises(ryo.RyoError) as e:
        ryo.solve(*_bodies(n, 1), *out, ryo.SolveParams(theta=0.5, bucket_size=16, stack_capacity=2))
    assert e.value.status == 4
    _check(out)


def test_batch_leaves_zeros():
    import ryoanji_b200 as ryo
    sizes = [700, 5, 3001]
    bodies = [torch.cat(v) for v in zip(*(_bodies(n, k) for k, n in enumerate(sizes)))]
    out = [torch.full((sum(sizes),), float("nan"), device="cuda") for _ in range(4)]
    b = ryo.solve_batch([ryo.BatchSystem(n) for n in sizes], *bodies, *out,
                        params=ryo.SolveParams(theta=0.5, bucket_size=16, stack_capacity=2))
    zero = _check(out).cpu().numpy()
    assert not zero[700:705].any()  # five bodies in a leaf need no stack
    assert b.stats.max_p2p == 0xffffffff and np.isfinite(b.energies).all()
