"""The up and down passes' basis where its fast reciprocals hand over to the
divisions: points on the interpolation nodes and box faces, a flat axis,
coordinates far below and above one, against the oracle (1e-12 relative L2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(dim, case, n):
    from barytreek_b200 import datagen
    pts, q = datagen.uniform_box(17, n, dim, 0.0, 1.0)
    pts = [p.copy() for p in pts]
    if case == "nodes":  # every axis on Chebyshev points of the dyadic boxes, and their corners
        u = 0.5 + 0.5 * np.cos(np.pi / 5 * np.arange(6))
        rng = np.random.default_rng(2)
        for p in pts:
            w = 0.5 ** rng.integers(0, 4, n)
            p[:] = np.floor(p / w) * w + w * u[rng.integers(0, 6, n)] + np.where(rng.random(n) < 0.3, 1e-17, 0.0)
    elif case == "flat":
        pts[-1][:] = 0.25
    elif case == "tiny":
        pts = [1e-14 * p for p in pts]
    elif case == "huge":
        pts = [1e30 * p for p in pts]
    return tuple(pts), q


@pytest.mark.parametrize("dim,kind,case,deg", [(3, 0, "nodes", 5), (2, 2, "nodes", 5), (3, 2, "flat", 4), (2, 0, "flat", 6),
                                               (2, 2, "tiny", 5), (3, 1, "tiny", 3), (2, 0, "huge", 7), (3, 0, "nodes", 1)])
def test_basis_edges(dim, kind, case, deg, oracle):
    import barytreek_b200 as btk
    pts, q = cloud(dim, case, 1700)
    eps = {"tiny": 1e-17, "huge": 1e20}.get(case, 1e-4)
    tc = btk.Treecode(pts, degree=deg, cluster_size=60, theta=0.7, eps=eps, kind=kind)
    t, (pp, pc, cp, cc) = tc.tree_t, tc.lists
    assert len(pc) + len(cp) + len(cc) > 0
    ref = oracle.solve({"dim": dim, "degree": deg, "eps": eps, "thresh": 60, "targets": tc.targets, "sources": tc.targets,
                        "panels_t": t.panels, "panels_s": t.panels, "level_start_t": t.level_start,
                        "level_start_s": t.level_start, "leaf_of_s": t.point_leaf_panel,
                        "inside_t": t.panel_points_inside, "inside_s": t.panel_points_inside, "pp": pp, "pc": pc,
                        "cp": cp, "cc": cc}, kind, q)["out"]
    out = tc.solve(q).cpu().numpy()
    for c in range(tc.ncomp):
        scale = np.linalg.norm(ref[c]) if np.linalg.norm(ref[c]) > 0 else 1.0
        assert np.linalg.norm(out[c] - ref[c]) <= 1e-12 * scale, (c, np.linalg.norm(out[c] - ref[c]) / scale)


@pytest.mark.parametrize("deg", [2, 4, 8, 12])
def test_basis_error_is_the_division_forms(deg):
    """One leaf over [-1, 1]^2 and one node's value 1: a point gets Lx_a(x) Ly_b(y). The rms relative error against
    extended precision is at most 1 % (the sampling of 6000 points and 3 nodes) above that of the formula in FP64
    with divisions."""
    import ctypes
    import math

    import torch

    import barytreek_b200 as btk
    from barytreek_b200 import _lib
    rng, n, m = np.random.default_rng(9), 6000, deg + 1
    pts = rng.uniform(-1.0, 1.0, (2, n))
    pts[:, 0], pts[:, 1] = -1.0, 1.0
    cfg = btk.make_run_config(2, deg, n + 1, 0.7, 1e-4)
    tree = btk.tree_construction(cfg, pts)
    box = tree.panels[0]
    assert tree.panel_count == 1 and [box[k] for k in ("min_x", "max_x", "min_y", "max_y")] == [-1.0, 1.0, -1.0, 1.0]
    dev, p = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda(), _lib.ptr
    x, panels, inside, info = [dev(a) for a in pts], dev(tree.panels.view(np.uint8)), dev(tree.panel_points_inside), tree.tree_info()
    w = np.array([(-1.0) ** i * (0.5 if i in (0, deg) else 1.0) for i in range(m)])
    node = np.array([math.cos(math.pi * i / deg) for i in range(m)])
    inner = np.all(np.abs(pts[:, :, None] - node).min(axis=2) > 1e-12, axis=0)

    def basis(v, kind):
        terms = [kind(wi) / (v.astype(kind) - kind(ni)) for wi, ni in zip(w, node)]
        total = terms[0].copy()
        for t in terms[1:]:
            total += t
        return [t / total for t in terms]
    div, ext = [[basis(v[inner], k) for v in pts] for k in (np.float64, np.longdouble)]
    err = {"kernel": [], "divisions": []}
    for a, b in ((0, m // 2), (m // 2, deg), (1, 1)):
        ptw = torch.zeros((1, m * m), dtype=torch.float64, device="cuda")
        ptw[0, a * m + b] = 1.0
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        _lib.check(_lib.load().btk_downward_pass_2d(ctypes.byref(cfg), ctypes.byref(info), p(x[0]), p(x[1]), p(out),
                                                    p(panels), p(ptw), p(inside), n, None))
        ref = ext[0][a] * ext[1][b]
        err["kernel"].append((out.cpu().numpy()[inner] - ref) / ref)
        err["divisions"].append((div[0][a] * div[1][b] - ref) / ref)
    rms = {k: float(np.sqrt(np.mean(np.square(np.concatenate(v))))) for k, v in err.items()}
    assert rms["kernel"] <= 1.01 * rms["divisions"], rms
