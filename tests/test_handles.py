"""Order in which the Python binding destroys its handles, over a fake library: children before
their lattice, lattices before their context, each once - closed by hand, dropped one by one, or
ended by the garbage collector as one cycle (an exception's traceback makes such cycles)."""
import gc

import numpy as np
import pytest


class FakeLibrary:
    def __init__(self):
        self.next, self.parent, self.alive, self.order = 1, {}, {}, []

    def _create(self, kind, parent, out):
        n, self.next = self.next, self.next + 1
        self.alive[n], self.parent[n] = kind, parent
        out._obj.value = n
        return 0

    def _destroy(self, kind, handle):
        n = handle.value
        assert self.alive.pop(n) == kind, "destroyed twice"
        self.order.append(kind)
        left = [self.alive[c] for c in self.alive if self.parent[c] == n]
        if left:
            self.order.append("children left: %s" % left)
        return 0

    def __getattr__(self, name):
        kind, _, what = name[3:].rpartition("_")
        if what == "create":
            return lambda *a: self._create(kind, getattr(a[0], "value", None), a[-1])
        if what == "destroy":
            return lambda h: self._destroy(kind, h)
        return lambda *a: 0


@pytest.mark.parametrize("how", ["close", "context", "drop", "cycle"])
def test_destroy_order(hw, monkeypatch, how):
    fake = FakeLibrary()
    monkeypatch.setattr(hw, "lib", lambda: fake)
    dims = (2, 2, 2, 2)
    ctx = hw.Context(0)
    made = []
    for _ in range(2):
        lat = hw.Lattice(ctx, dims)
        made += [lat, hw.GaugeField(lat, np.zeros((4, 16, 3, 3, 2))), hw.Field(lat), hw.StaggeredField(lat)]
    assert len(fake.alive) == 9
    if how == "close":
        for m in made[::4]:
            m.close()
        for m in made:
            m.close()
        assert list(fake.alive.values()) == ["context"]
    elif how == "cycle":
        for m in made:
            m.cycle = made
        ctx.cycle = made
    if how in ("close", "context"):
        ctx.close()
    del made, lat, ctx
    m = None  # noqa: F841
    gc.collect()
    assert not fake.alive and not [o for o in fake.order if o.startswith("children")], fake.order
    assert sorted(fake.order) == sorted(["context"] + 2 * ["lattice", "gauge", "field", "stag_field"])
