"""btk_direct_sum at the edges of its split (64 targets a tile, 4 warps a block,
slices of the sources added by a second kernel, 32 sources at a time) and outside the fast
reciprocals' range, against the oracle's direct sum. Tolerance: 1e-13 relative
L2 (FP64 sums of at most 20,000 terms in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def direct(dim, kind, eps, t, s, q):
    import torch

    from barytreek_b200 import _lib, treecode
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()
    T, S, Q = [dev(a) for a in t], [dev(a) for a in s], dev(q)
    out = torch.empty((treecode.ncomp(dim, kind), len(t[0])), dtype=torch.float64, device="cuda")
    z = lambda a: _lib.ptr(a[2]) if dim == 3 else None
    _lib.check(_lib.load().btk_direct_sum(dim, kind, eps, len(t[0]), _lib.ptr(T[0]), _lib.ptr(T[1]), z(T), len(q),
                                          _lib.ptr(S[0]), _lib.ptr(S[1]), z(S), _lib.ptr(Q), _lib.ptr(out), None))
    return out.cpu().numpy()


@pytest.mark.parametrize("dim,kind", [(2, 0), (2, 2), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("nt,ns", [(1, 1), (63, 31), (64, 33), (65, 255), (129, 2049), (3000, 511), (500, 20011),
                                   (9999, 77)])
def test_split_edges(dim, kind, nt, ns, oracle):
    rng = np.random.default_rng(nt + ns)
    t, s, q = rng.random((dim, nt)), rng.random((dim, ns)), rng.uniform(-1, 1, ns)
    out, ref = direct(dim, kind, 1e-4, t, s, q), oracle.direct(dim, kind, 1e-4, t, s, q)
    for c in range(len(ref)):
        assert np.linalg.norm(out[c] - ref[c]) <= 1e-13 * np.linalg.norm(ref[c])


@pytest.mark.parametrize("dim,kind", [(2, 0), (2, 2), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("scale,eps", [(1e-30, 1e-25), (1.0, 0.0), (1e25, 1.0), (1.0, 1e20), (1e17, 1e-3)])
def test_outside_the_seed_range(dim, kind, scale, eps, oracle):
    """Tiny and zero eps, coordinates and eps beyond the FP32 range."""
    rng = np.random.default_rng(3)
    t, s, q = scale * rng.random((dim, 300)), scale * rng.random((dim, 700)), rng.uniform(-1, 1, 700)
    out, ref = direct(dim, kind, eps, t, s, q), oracle.direct(dim, kind, eps, t, s, q)
    for c in range(len(ref)):
        assert np.linalg.norm(out[c] - ref[c]) <= 1e-13 * np.linalg.norm(ref[c])


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_non_finite(kind, oracle):
    """A coincident pair at eps 0, an infinite and a NaN coordinate: the same targets are finite."""
    rng = np.random.default_rng(4)
    t, s, q = rng.random((3, 200)), rng.random((3, 100)), rng.uniform(0.1, 1, 100)
    t[:, 5] = s[:, 7]
    t[0, 70], t[1, 80] = np.inf, np.nan
    with np.errstate(all="ignore"):
        out, ref = direct(3, kind, 0.0, t, s, q), oracle.direct(3, kind, 0.0, t, s, q)
    for c in range(len(ref)):
        fine = np.isfinite(ref[c])
        assert np.array_equal(fine, np.isfinite(out[c]))
        assert np.array_equal(np.isnan(ref[c]), np.isnan(out[c]))
        assert np.linalg.norm((out[c] - ref[c])[fine]) <= 1e-13 * np.linalg.norm(ref[c][fine])


@pytest.mark.parametrize("dim,kind", [(2, 2), (3, 1)])
def test_quotients_are_rounded_once(dim, kind):
    """One source, r^2 exact (whole numbers, eps 1): the vector sums are the rounded w / r^2 times x and the factor,
    each product rounded, bit for bit."""
    rng = np.random.default_rng(9)
    t = rng.integers(-30000, 30000, (dim, 4001)).astype(np.float64)
    r2 = (t * t).sum(0) + 1.0
    factor = -1.0 / ((2.0 if dim == 2 else 4.0) * np.pi)
    for w in (1.0, 3.0, float(rng.integers(1, 2 ** 40)), -1.0 / 3.0, 1e-200, 1e199, 1e250):
        out = direct(dim, kind, 1.0, t, np.zeros((dim, 1)), np.array([w]))
        for c in range(dim):
            assert np.array_equal(out[len(out) - dim + c], t[c] * (w / r2) * factor), (w, c)


@pytest.mark.parametrize("dim,kind", [(2, 0), (2, 2), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("bad", ["target inf", "target nan", "source inf", "source nan", "charge inf", "charge nan"])
def test_non_finite_at_ordinary_eps(dim, kind, bad, oracle):
    """Where eps lets the fast reciprocals be taken: the same results are infinite or not numbers."""
    rng = np.random.default_rng(4)
    t, s, q = rng.random((dim, 200)), rng.random((dim, 100)), rng.uniform(0.1, 1, 100)
    what, v = bad.split()
    {"target": t[0], "source": s[0], "charge": q}[what][70] = float(v)
    with np.errstate(all="ignore"):
        out, ref = direct(dim, kind, 1e-4, t, s, q), oracle.direct(dim, kind, 1e-4, t, s, q)
        for c in range(len(ref)):
            fine = np.isfinite(ref[c])
            assert np.array_equal(np.isnan(ref[c]), np.isnan(out[c])) and np.array_equal(ref[c][~fine], out[c][~fine], equal_nan=True)
            assert np.linalg.norm((out[c] - ref[c])[fine]) <= 1e-13 * np.linalg.norm(ref[c][fine])
