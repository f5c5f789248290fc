"""Level ranges (tree_info) that name the same tree in another way: the first
clusters' level twice, the root left out, an empty first level. None of them
changes a solve here (the root's and the first level's clusters are in no
list), so each equals the plain ranges' (1e-13 relative L2: the order of the
work items' additions); the proxies' places must not follow from the ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def variants(ls, nc):
    first = [0, 1, 1 + nc]
    assert list(ls[:3]) == first
    return {"twice": [*first, 1, *ls[2:]], "no root": list(ls[1:]), "empty": [0, *ls]}


@pytest.mark.parametrize("dim,kind", [(2, 0), (3, 2)])
def test_level_ranges(dim, kind):
    import barytreek_b200 as btk
    from barytreek_b200 import datagen

    class Renamed(btk.Treecode):
        ranges = None

        def _create_plan(self):
            if self.ranges is not None:
                self.tree_t.level_start = np.asarray(self.ranges, np.int32)
            super()._create_plan()

    pts, q = datagen.uniform_box(21, 4001, dim, 0.0, 1.0)
    make = lambda: Renamed(pts, degree=4, cluster_size=20, theta=0.6, eps=1e-3, kind=kind)
    tc = make()
    nc = 1 << dim
    pp, pc, cp, cc = tc.lists
    used = np.concatenate([pc["source_panel"], cc["source_panel"], cp["target_panel"], cc["target_panel"]])
    assert len(used) > 0 and used.min() > nc
    ref = tc.solve(q).cpu().numpy()
    for name, ranges in variants(tc.tree_t.level_start, nc).items():
        Renamed.ranges = ranges
        out = make().solve(q).cpu().numpy()
        for c in range(len(ref)):
            assert np.linalg.norm(out[c] - ref[c]) <= 1e-13 * np.linalg.norm(ref[c]), (name, c)
