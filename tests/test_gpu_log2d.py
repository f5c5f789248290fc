"""The 2-D FP64 kernel's table logarithm and the reciprocal that shares its
seed: one source of charge 1 at the origin, so the potential is
log(r^2 + eps^2) / (4 pi) and the field (x, y) / (2 pi (r^2 + eps^2)), against
extended precision. Radii around 1 (the logarithm's zero), at the table's
steps, small, huge, and beyond the table's range (the guarded kernel).
Tolerances: the potential to 8 roundings of max(1, |log|) (r^2, the table, the
sum, the scale), the field to 1e-12 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi,eps", [(0.999, 1.001, 1e-9), (0.5, 2.0, 1e-9), (1e-12, 1e-3, 1e-15), (1e-3, 1e4, 1e-4),
                                       (1e100, 1e150, 1.0), (1e152, 4e153, 1.0), (1e-3, 1e3, 0.0)])
def test_log_and_reciprocal(lo, hi, eps):
    import barytreek_b200 as btk
    rng = np.random.default_rng(5)
    n = 4099
    r = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    r[:513] = np.sqrt(np.clip(1.0 / (0.5 + np.arange(513) / 1024.0), (lo / r.max()) ** 2, None)) * lo  # table steps
    a = rng.uniform(0.0, 2.0 * np.pi, n)
    x, y = r * np.cos(a), r * np.sin(a)
    src = (np.array([0.0, lo, -lo]), np.array([0.0, lo, lo]))
    tc = btk.Treecode((x, y), src, degree=2, cluster_size=5000, theta=0.7, eps=eps, kind=btk.KIND_FIELD)
    out = tc.solve(np.array([1.0, 0.0, 0.0])).cpu().numpy()
    X, Y, E = (np.asarray(v, np.longdouble) for v in (x, y, eps))
    r2 = X * X + Y * Y + E * E
    pi = np.longdouble("3.14159265358979323846264338327950288")
    err = np.abs(out[0] - np.log(r2) / (4 * pi))
    assert np.all(err <= 8 * 2.0 ** -53 * np.maximum(1.0, np.abs(np.log(r2))) / (4 * pi)), float(err.max())
    if hi < 1e18:  # the reciprocal of r^2 has the FP32 range where the guarded kernel runs
        for c, v in ((1, X), (2, Y)):
            ref = -v / (2 * pi * r2)
            assert np.all(np.abs(np.abs(out[c]) - np.abs(ref)) <= 1e-12 * np.abs(ref) + 1e-300)


@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("log2_eps", [508.5, 509.5, 510.75, 511.5])
def test_large_eps(log2_eps, same):
    """eps^2 up to and beyond the table's range: the potential is the charges' sum times log(eps^2) / (4 pi),
    to a rounding a charge and 8 of the rest."""
    import barytreek_b200 as btk
    rng = np.random.default_rng(6)
    n = 300
    pts, q = (rng.random(n), rng.random(n)), rng.uniform(0.5, 1.0, n)
    tc = btk.Treecode(pts, None if same else tuple(p[::-1].copy() for p in pts), degree=2, cluster_size=40, theta=0.7,
                      eps=2.0 ** log2_eps, kind=btk.KIND_POT)
    ref = float(q.sum()) * 2 * log2_eps * np.log(2.0) / (4 * np.pi)
    assert np.all(np.abs(tc.solve(q).cpu().numpy()[0] - ref) <= (n + 8) * 2.0 ** -53 * ref)


@pytest.mark.parametrize("direct", [False, True])
def test_relative_error_near_one(direct):
    """r^2 around 1, exact in FP64 (x of 26 bits, y = 0): the logarithm keeps its relative accuracy through its
    zero. 7 roundings: 3 of the logarithm, its table's value against the sum 2, the constant factor 2."""
    import torch

    import barytreek_b200 as btk
    from barytreek_b200 import _lib
    rng = np.random.default_rng(7)
    j = np.concatenate([np.arange(-1500, 0), np.arange(1, 1500), rng.integers(-2 ** 22, 2 ** 22, 5000)])
    x = 1.0 + (j[j != 0] * 2.0 ** -25)
    t, s, q = (x, np.zeros_like(x)), (np.array([0.0, 3.0]), np.zeros(2)), np.array([1.0, 0.0])
    if direct:
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        T, S, Q, out = [dev(a) for a in t], [dev(a) for a in s], dev(q), torch.empty(len(x), dtype=torch.float64, device="cuda")
        p = _lib.ptr
        _lib.check(_lib.load().btk_direct_sum(2, btk.KIND_POT, 2.0 ** -60, len(x), p(T[0]), p(T[1]), None, 2, p(S[0]),
                                              p(S[1]), None, p(Q), p(out), None))
        out = out.cpu().numpy()
    else:
        out = btk.Treecode(t, s, degree=2, cluster_size=9000, theta=0.7, eps=2.0 ** -60).solve(q).cpu().numpy()[0]
    ref = 2 * np.log1p(np.asarray(x - 1.0, np.longdouble)) / (4 * np.longdouble("3.14159265358979323846264338327950288"))
    assert np.max(np.abs((out - ref) / ref)) <= 7 * 2.0 ** -53


@pytest.mark.parametrize("lo,hi,eps", [(1e-3, 1e4, 1e-4), (1e17, 1e30, 1.0), (1e100, 1e150, 1.0)])
def test_signed_field(lo, hi, eps):
    """Both components with their signs, and radii beyond the FP32 range, where the reciprocal comes with the
    logarithm's exponent: 1e-12 relative."""
    import barytreek_b200 as btk
    rng = np.random.default_rng(8)
    r, a = np.exp(rng.uniform(np.log(lo), np.log(hi), 3001)), rng.uniform(0.0, 2.0 * np.pi, 3001)
    x, y = r * np.cos(a), r * np.sin(a)
    src = (np.array([0.0, lo, -lo]), np.array([0.0, lo, lo]))
    tc = btk.Treecode((x, y), src, degree=2, cluster_size=5000, theta=0.7, eps=eps, kind=btk.KIND_FIELD)
    out = tc.solve(np.array([1.0, 0.0, 0.0])).cpu().numpy()
    X, Y, E = (np.asarray(v, np.longdouble) for v in (x, y, eps))
    for c, v in ((1, X), (2, Y)):
        ref = -v / (2 * np.longdouble("3.14159265358979323846264338327950288") * (X * X + Y * Y + E * E))
        assert np.all(np.abs(out[c] - ref) <= 1e-12 * np.abs(ref))
