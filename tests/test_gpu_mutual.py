"""Leaf pairs evaluated once for both directions (FP64, targets = sources, at
least 5e7 leaf-pair evaluations) against the one-sided form of the same plan,
which the same points in other arrays take. Leaves of 1 to 290 points (rows of
32 targets and blocks of 32 sources cut anywhere), tiles of 256 and 128, every
kernel. Tolerance: 1e-12 relative L2 (the same pairs in another order; the
reciprocals' 4e-14 a pair). Lists with directions missing and pairs listed
twice run against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve_one_sided(tc, q):
    """The plan's solve with the sources in arrays of their own."""
    import torch

    from barytreek_b200 import _lib
    out = torch.empty((tc.ncomp, tc.nt), dtype=torch.float64, device="cuda")
    t, s = tc._t, [a.clone() for a in tc._t]
    qd = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    z = lambda a: _lib.ptr(a[2]) if tc.dim == 3 else None
    _lib.check(_lib.load().btk_plan_execute(tc._plan, _lib.ptr(t[0]), _lib.ptr(t[1]), z(t), _lib.ptr(s[0]), _lib.ptr(s[1]),
                                            z(s), _lib.ptr(qd), _lib.ptr(out), None))
    return out.cpu().numpy()


def close(a, b, tol=1e-12):
    for c in range(len(b)):
        e = np.linalg.norm(a[c] - b[c]) / np.linalg.norm(b[c])
        assert e <= tol, (c, e)


@pytest.mark.parametrize("dim,kind,n,leaf,tile,dist", [
    (3, 0, 30011, 290, 256, "cube"), (3, 2, 30011, 290, 256, "cube"), (3, 1, 30011, 290, 256, "cube"),
    (2, 0, 40009, 129, 256, "cube"), (2, 2, 40009, 129, 128, "cube"), (3, 2, 20011, 700, 128, "plummer"),
    (3, 0, 25013, 33, 256, "plummer"), (3, 1, 12007, 3000, 256, "mixture")])
def test_mutual_matches_one_sided(dim, kind, n, leaf, tile, dist):
    import barytreek_b200 as btk
    from barytreek_b200 import datagen
    pts, q = (datagen.uniform_box(3, n, dim, 0.0, 1.0) if dist == "cube" else datagen.plummer(3, n) if dist == "plummer"
              else datagen.gaussian_mixture(3, n))
    tc = btk.Treecode(pts, degree=3, cluster_size=leaf, theta=0.6, eps=1e-4, kind=kind, tile_targets=tile)
    assert tc.stats()["evals_pp"] >= 50000000
    a, b = tc.solve(q).cpu().numpy(), solve_one_sided(tc, q)
    close(a, b)
    close(tc.solve(2.0 * q).cpu().numpy(), 2.0 * b)  # the sums' arrays are cleared each time


def test_unsymmetric_and_repeated_pairs(oracle):
    """Lists that are not symmetric: a direction left out, a pair listed twice."""
    import barytreek_b200 as btk
    from barytreek_b200 import datagen

    class Edited(btk.Treecode):
        def _create_plan(self):
            pp = self.lists[0]
            off = np.flatnonzero(pp["target_panel"] != pp["source_panel"])
            drop, twice = off[5::97], off[11::89]
            pp = np.concatenate([np.delete(pp, drop), pp[twice]])
            self.lists = (pp, *self.lists[1:])
            self.cfg.fmm_pp_count = len(pp)
            super()._create_plan()

    pts, q = datagen.uniform_box(8, 9001, 3, 0.0, 1.0)
    tc = Edited(pts, degree=2, cluster_size=200, theta=0.3, eps=1e-3, kind=btk.KIND_FIELD)
    assert tc.stats()["evals_pp"] >= 50000000
    t, (pp, pc, cp, cc) = tc.tree_t, tc.lists
    tree = {"dim": 3, "degree": 2, "eps": 1e-3, "thresh": 200, "targets": tc.targets, "sources": tc.targets,
            "panels_t": t.panels, "panels_s": t.panels, "level_start_t": t.level_start, "level_start_s": t.level_start,
            "leaf_of_s": t.point_leaf_panel, "inside_t": t.panel_points_inside, "inside_s": t.panel_points_inside,
            "pp": pp, "pc": pc, "cp": cp, "cc": cc}
    ref = oracle.solve(tree, btk.KIND_FIELD, q)["out"]
    close(tc.solve(q).cpu().numpy(), ref)
    close(solve_one_sided(tc, q), ref)


def test_captured_batch():
    """An FP64 batch (one captured graph) whose problems together reach the
    mutual form, replayed with new charges, against each problem's own plan."""
    import barytreek_b200 as btk
    from barytreek_b200 import datagen
    from barytreek_b200.batch import Batch
    probs = [datagen.gaussian_mixture(40 + k, n) for k, n in enumerate((9001, 4097, 12000))]
    b = Batch([p[0] for p in probs], degree=4, theta=0.6, eps=1e-4, kind=btk.KIND_FIELD, precision=btk.PREC_FP64,
              cluster_size=[400, 200, 900])
    assert b.stats()["evals_pp"] >= 50000000
    q = np.concatenate([p[1] for p in probs])
    b.solve(q)
    out = b.split(b.solve(-3.0 * q).cpu().numpy())
    for (pts, qi), leaf, o in zip(probs, (400, 200, 900), out):
        tc = btk.Treecode(pts, degree=4, cluster_size=leaf, theta=0.6, eps=1e-4, kind=btk.KIND_FIELD)
        close(o, -3.0 * solve_one_sided(tc, qi))


def test_wait_limit_timeout_then_recovery():
    """The mutual launch's bounded waits: none allowed, an error status; then the plan solves again."""
    import barytreek_b200 as btk
    from barytreek_b200 import _lib, datagen
    pts, q = datagen.uniform_box(6, 30011, 3, 0.0, 1.0)
    tc = btk.Treecode(pts, degree=3, cluster_size=290, theta=0.6, eps=1e-4, kind=btk.KIND_FIELD)
    assert tc.stats()["evals_pp"] >= 50000000
    ref = solve_one_sided(tc, q)
    tc.set_wait_limit(0)
    tc.solve(q)
    with pytest.raises(_lib.BtkError) as ei:
        tc.last_timing()
    assert ei.value.status == _lib.ERR_DEVICE_TIMEOUT
    tc.set_wait_limit(-1)
    close(tc.solve(q).cpu().numpy(), ref)
    tc.last_timing()


@pytest.mark.parametrize("dim,kind,n,leaf", [(3, 0, 30011, 290), (3, 2, 30011, 290), (3, 1, 30011, 290),
                                             (2, 0, 40009, 129), (2, 2, 40009, 129)])
@pytest.mark.parametrize("value", [0.0, np.inf, np.nan])
def test_zero_and_non_finite_charges(dim, kind, n, leaf, value):
    """Weight 0 fills idle lanes: charges that are 0 (every third), and one infinite or not a number among them, give
    what the one-sided form gives."""
    import barytreek_b200 as btk
    from barytreek_b200 import datagen
    pts, q = datagen.uniform_box(3, n, dim, 0.0, 1.0)
    q = q.copy()
    q[::3] = 0.0
    q[n // 2] = value
    tc = btk.Treecode(pts, degree=3, cluster_size=leaf, theta=0.6, eps=1e-4, kind=kind)
    assert tc.stats()["evals_pp"] >= 50000000
    a, b = tc.solve(q).cpu().numpy(), solve_one_sided(tc, q)
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(a[np.isinf(a)], b[np.isinf(b)])
    for c in range(len(b)):
        fine = np.isfinite(b[c])
        assert np.array_equal(fine, np.isfinite(a[c]))
        assert np.linalg.norm((a[c] - b[c])[fine]) <= 1e-12 * np.linalg.norm(b[c][fine])
