"""The drop-in cache's entries: a call with another eps on the same arrays gets
its own results, and programs that alternate between many trees keep theirs
(every result against the plan path, 1e-12 relative L2)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Program:
    """Tree, lists and device arrays of one drop-in program."""

    def __init__(self, seed, n=3000):
        import torch

        import barytreek_b200 as btk
        from barytreek_b200 import datagen
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.pts, self.q = datagen.uniform_box(seed, n, 3, 0.0, 1.0)
        self.cfg = btk.make_run_config(3, 4, 80, 0.7, 1e-4)
        self.tree = btk.tree_construction(self.cfg, self.pts)
        lists = btk.split_interactions(self.cfg, btk.dual_tree_traversal(self.cfg, self.tree))
        self.info, self.x, self.qd = self.tree.tree_info(), [dev(a) for a in self.pts], dev(self.q)
        self.arrays = [dev(a) for a in (self.tree.panels.view(np.uint8), self.tree.point_leaf_panel,
                                        self.tree.panel_points_inside)]
        self.lists = [dev(a.view(np.uint8)) if len(a) else None for a in lists]

    def check(self, eps):
        import torch

        import barytreek_b200 as btk
        from barytreek_b200 import _lib
        lib, p, n, P = _lib.load(), _lib.ptr, len(self.q), self.tree.panel_count
        self.cfg.ker_eps = eps
        psw, ptw = (torch.zeros((P, self.cfg.interp_point_count), dtype=torch.float64, device="cuda") for _ in range(2))
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        cfg, info, x = ctypes.byref(self.cfg), ctypes.byref(self.info), [p(a) for a in self.x]
        panels, leaf_of, inside = [p(a) for a in self.arrays]
        _lib.check(lib.btk_upward_pass_3d(cfg, info, *x, p(self.qd), panels, p(psw), leaf_of, n, None))
        _lib.check(lib.btk_poisson_fmm_interactions_3d(cfg, *x, *x, p(self.qd), p(out), inside, inside, p(psw), p(ptw),
                                                       *[p(a) for a in self.lists], panels, panels, n, n, P, P, None))
        _lib.check(lib.btk_downward_pass_3d(cfg, info, *x, p(out), panels, p(ptw), inside, n, None))
        ref = btk.Treecode(self.pts, degree=4, cluster_size=80, theta=0.7, eps=eps).solve(self.q).cpu().numpy()[0]
        assert np.linalg.norm(out.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)


def test_another_eps_on_the_same_arrays():
    a = Program(3)
    for eps in (1e-4, 0.3, 1e-4):
        a.check(eps)


def test_many_trees_in_turn():
    programs = [Program(10 + k, 1500 + 100 * k) for k in range(18)]  # 54 entries: more than are kept
    for _ in range(2):
        for a in programs:
            a.check(1e-3)


class Gather:
    """The interaction call alone on one tree whose arrays are large for its points (small leaves, high degree),
    with empty far lists and the leaf pairs of the tree; a copy of the panels in a buffer of its own is another tree
    to the cache."""

    def __init__(self, n, leaf, degree, pairs):
        import torch

        import barytreek_b200 as btk
        from barytreek_b200 import datagen
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        pts, q = datagen.uniform_box(5, n, 3, 0.0, 1.0)
        self.cfg = btk.make_run_config(3, degree, leaf, 0.7, 1e-2)
        self.tree = btk.tree_construction(self.cfg, pts)
        pp = btk.split_interactions(self.cfg, btk.dual_tree_traversal(self.cfg, self.tree))[0][:pairs]
        self.cfg.fmm_pp_count, self.cfg.fmm_pc_count, self.cfg.fmm_cp_count, self.cfg.fmm_cc_count = len(pp), 0, 0, 0
        self.x, self.q, self.n = [dev(a) for a in pts], dev(q), n
        self.panels, self.inside = dev(self.tree.panels.view(np.uint8)), dev(self.tree.panel_points_inside)
        self.pp = dev(pp.view(np.uint8)) if pairs else None
        self.psw, self.ptw = (torch.zeros((self.tree.panel_count, self.cfg.interp_point_count), dtype=torch.float64,
                                          device="cuda") for _ in range(2))
        self.out = torch.zeros(n, dtype=torch.float64, device="cuda")

    def call(self, panels):
        from barytreek_b200 import _lib
        p, P, n = _lib.ptr, self.tree.panel_count, self.n
        self.out.zero_()
        x = [p(a) for a in self.x]
        return _lib.load().btk_poisson_fmm_interactions_3d(
            ctypes.byref(self.cfg), *x, *x, p(self.q), p(self.out), p(self.inside), p(self.inside), p(self.psw),
            p(self.ptw), p(self.pp), None, None, None, p(panels), p(panels), n, n, P, P, None)


def free_bytes():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_entries_stay_within_their_bytes():
    """More than six trees: the entries hold at most 2 GiB, or six of them what they need, and the one in use."""
    from barytreek_b200 import _lib
    g = Gather(100000, 25, 12, 0)
    copies = [g.panels.clone() for _ in range(12)]
    _lib.check(_lib.load().btk_dropin_cache_clear())
    free = [free_bytes()]
    for panels in copies:
        _lib.check(g.call(panels))
        free.append(free_bytes())
    held = [free[0] - f for f in free[1:]]
    assert held[0] > 200 << 20  # else the limit is not reached
    assert max(held) <= max(2 << 30, 6 * held[0]) + held[0] + (64 << 20), held
    _lib.check(_lib.load().btk_dropin_cache_clear())
    assert free[0] - free_bytes() <= 64 << 20


def test_memory_given_back_when_an_allocation_does_not_fit():
    """Entries of earlier trees make room for a new one, and for a plan, on a device without free memory."""
    import torch

    import barytreek_b200 as btk
    from barytreek_b200 import _lib, datagen
    g = Gather(100000, 25, 10, 1000)
    copies = [g.panels.clone() for _ in range(6)]
    _lib.check(_lib.load().btk_dropin_cache_clear())
    free0 = free_bytes()
    _lib.check(g.call(copies[0]))
    ref, entry = g.out.cpu().numpy(), free0 - free_bytes()
    for panels in copies[1:5]:
        _lib.check(g.call(panels))
    pts, q = datagen.uniform_box(5, 20000, 3, 0.0, 1.0)
    make = lambda: btk.Treecode(pts, degree=10, cluster_size=40, theta=0.7, eps=1e-2)
    tc = make()
    sol = tc.solve(q).cpu().numpy()
    tc.close()
    room = 40 << 20
    assert entry > 2 * room
    fill = torch.empty(free_bytes() - room, dtype=torch.uint8, device="cuda")
    try:
        assert free_bytes() < entry
        _lib.check(g.call(copies[5]))  # needs the other entries' memory
        out = g.out.cpu().numpy()
        assert np.linalg.norm(out - ref) <= 1e-13 * np.linalg.norm(ref)  # pieces add in any order
        del fill
        for panels in copies[:5]:
            _lib.check(g.call(panels))
        fill = torch.empty(free_bytes() - room, dtype=torch.uint8, device="cuda")
        tc = make()
        out = tc.solve(q).cpu().numpy()
    finally:
        fill = None
        torch.cuda.empty_cache()
        _lib.check(_lib.load().btk_dropin_cache_clear())
    assert np.linalg.norm(out - sol) <= 1e-13 * np.linalg.norm(sol)
