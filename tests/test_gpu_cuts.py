"""Work items cut for the schedule (work_split): a mixed solve keeps every
256- (or 128-) source chunk's FP32 sums, so its result moves only by the order
of FP64 additions (tolerance 1e-13 relative L2, a few thousand roundings), and
an FP64 solve likewise; leaf sizes leave odd remainders at the cuts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim,kind,n,leaf,tile", [(3, 2, 3001, 130, 256), (3, 0, 3001, 130, 128), (3, 1, 5003, 700, 256),
                                                  (2, 2, 4001, 257, 256), (3, 0, 999, 2000, 256)])
def test_cuts_keep_the_result(dim, kind, n, leaf, tile, precision):
    import barytreek_b200 as btk
    from barytreek_b200 import datagen
    pts, q = datagen.uniform_box(3, n, dim, 0.0, 1.0)
    outs, items = [], []
    for split in (1, 8, 1024):
        tc = btk.Treecode(pts, degree=4, cluster_size=leaf, theta=0.7, eps=1e-3, kind=kind, precision=precision,
                          tile_targets=tile, work_split=split)
        outs.append(tc.solve(q).cpu().numpy())
        items.append(tc.stats()["work_items"])
    assert items[2] >= items[0]
    for o in outs[1:]:
        for c in range(len(o)):
            assert np.linalg.norm(o[c] - outs[0][c]) <= 1e-13 * np.linalg.norm(outs[0][c])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim,kind,n,leaf,tile", [(3, 2, 20011, 300, 256), (3, 1, 20011, 300, 256), (3, 0, 20011, 60, 128),
                                                  (2, 2, 20011, 300, 256)])
def test_coarse_and_fine_cuts_against_the_oracle(dim, kind, n, leaf, tile, precision, oracle):
    """Sizes where a coarser schedule cuts less (both sides of the leaf pairs' 5e7 evaluations): the lists differ, the
    FP64 results are the oracle's (1e-12), the mixed ones each other's."""
    import barytreek_b200 as btk
    from barytreek_b200 import datagen
    pts, q = datagen.uniform_box(5, n, dim, 0.0, 1.0)
    outs, items = [], []
    for split in (1, 8, 64):
        tc = btk.Treecode(pts, degree=6, cluster_size=leaf, theta=0.6, eps=1e-3, kind=kind, precision=precision,
                          tile_targets=tile, work_split=split)
        outs.append(tc.solve(q).cpu().numpy())
        items.append(tc.stats()["work_items"])
    assert items[0] < items[1] <= items[2], items  # the finest may be at the shortest piece already
    if precision == 0:
        t, (pp, pc, cp, cc) = tc.tree_t, tc.lists
        tree = {"dim": dim, "degree": 6, "eps": 1e-3, "thresh": leaf, "targets": tc.targets, "sources": tc.targets,
                "panels_t": t.panels, "panels_s": t.panels, "level_start_t": t.level_start,
                "level_start_s": t.level_start, "leaf_of_s": t.point_leaf_panel, "inside_t": t.panel_points_inside,
                "inside_s": t.panel_points_inside, "pp": pp, "pc": pc, "cp": cp, "cc": cc}
        ref, tol = oracle.solve(tree, kind, q)["out"], 1e-12
    else:
        ref, tol = outs[0], 1e-13
    for o in outs:
        for c in range(len(o)):
            assert np.linalg.norm(o[c] - ref[c]) <= tol * np.linalg.norm(ref[c])
