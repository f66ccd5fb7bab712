"""Contexts in different host threads and streams do not disturb one another, whatever their stack capacities."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# the fused kernel (a group per body), divided walks, whole walks; a stack of 1,000 entries needs more shared memory
# than a kernel may use without having asked for it
@pytest.mark.parametrize("n,group", [(60000, 1), (20000, 64), (60000, 8)])
def test_solves_in_two_threads(n, group):
    import ryoanji_b200 as ryo
    from ryoanji_b200 import datasets as ds
    p = ds.plummer(n, seed=n, velocities=False)
    bodies = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (p.x, p.y, p.z, p.m, p.h)]
    errors, results = [], {}

    def work(capacity):
        try:
            stream = torch.cuda.Stream()
            ctx, own = ryo.Context(), [b.clone() for b in bodies]
            out, base = torch.empty(4, n, device="cuda"), None
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                for _ in range(60):
                    for w, b in zip(own, bodies):
                        w.copy_(b)
                    out.fill_(float("nan"))
                    ryo.solve(*own, *out, ryo.SolveParams(group_size=group, stack_capacity=capacity), ctx=ctx)
                    got = out.clone()
                    base = got if base is None else base
                    assert torch.equal(got, base)
            stream.synchronize()
            results[capacity] = base
        except Exception as e:
            errors.append(repr(e))
    threads = [threading.Thread(target=work, args=(c,)) for c in (0, 800, 1000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert torch.equal(results[0], results[800]) and torch.equal(results[0], results[1000])
