"""A view of a tree builder's arrays keeps the builder, whose memory it shows."""
import gc
import weakref

import pytest

torch = pytest.importorskip("torch")
ryo = pytest.importorskip("ryoanji_b200")


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["order", "layout", "nodeKeys", "childOffsets", "internalToLeaf", "leafToInternal",
                                  "parents", "leaves", "sortedKeys"])
def test_view_keeps_builder(name):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    x, y, z = (torch.rand(3000, generator=gen, device="cuda") for _ in range(3))
    builder = ryo.TreeBuilder(16)
    builder.update(x, y, z, ryo.Box.cube(0.0, 1.0))
    view = getattr(builder, name)()
    copy, alive = view.clone(), weakref.ref(builder)
    del builder
    gc.collect()
    assert alive() is not None
    assert torch.equal(view, copy)
    del view
    gc.collect()
    assert alive() is None
