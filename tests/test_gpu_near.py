"""FP64 near field at the sizes where its runs and batches end, and at odd distances.

One-leaf problems (at most nbox sources and targets) are the near field alone, so every output is
compared with the oracle's direct sum.  Each pair term is a handful of FP64 operations (relative
error below 40 eps with the approximate reciprocal square root refined to 2 eps) and a sum of n
terms adds n eps of the sum of magnitudes; with at most 320 random terms 1e-13 relative L2 is asked.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import fmmlib3d_b200
    return fmmlib3d_b200


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("charges,dipoles", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 31), (31, 1), (32, 32), (33, 64), (64, 65), (97, 160), (160, 3)])
def test_one_leaf(F, n, m, charges, dipoles):
    rng = np.random.default_rng(1000 * n + m)
    src, trg = rng.random((n, 3)), rng.random((m, 3))
    q = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) if charges else None
    ds = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) if dipoles else None
    dv = rng.normal(size=(n, 3)) if dipoles else None
    ier, pot, fld, pt, ft = F.lfmm3dparttarg(1, src, int(charges), q, int(dipoles), ds, dv, 1, 1, trg, 1, 1)
    assert ier == 0
    p0, f0 = O.direct_at(src, src, np.arange(n), q, ds, dv)
    p1, f1 = O.direct_at(src, trg, None, q, ds, dv)
    if n > 1:
        assert rel(pot, p0) < 1e-13 and rel(fld, f0) < 1e-13
    else:
        assert not np.any(pot) and not np.any(fld)
    assert rel(pt, p1) < 1e-13 and rel(ft, f1) < 1e-13


@pytest.mark.parametrize("gap", [1e-30, 1e-100, 1e-148])
def test_pairs_at_extreme_distances(F, gap):
    """Distances whose squares lie inside and outside the range of the fast reciprocal square root."""
    src = np.array([[0.0, 0, 0], [gap, 0, 0], [1, 1, 1], [0.3, 0.9, 0.2]])
    q = np.array([1.0, 0.5, -0.25, 0.75]) + 0j
    ier, pot, _ = F.lfmm3dpartself(1, src, 1, q, 0, None, None, 1, 0)
    assert ier == 0
    p0, _ = O.direct_at(src, src, np.arange(4), q)
    assert np.allclose(pot, p0, rtol=1e-13, atol=0)


def test_coincident_points_give_infinities_and_leave_the_others(F):
    """Two sources at one place: infinite potentials there (1/0), the other points as without them."""
    rng = np.random.default_rng(3)
    src = rng.random((70, 3))
    src[41] = src[7]
    q = rng.uniform(0.1, 1, 70) + 0j
    ier, pot, fld = F.lfmm3dpartself(1, src, 1, q, 0, None, None, 1, 1)
    assert ier == 0
    assert np.isinf(pot[[7, 41]].real).all()
    keep = np.setdiff1d(np.arange(70), [7, 41])
    p0, f0 = O.direct_at(src, src[keep], keep, q)
    assert rel(pot[keep], p0) < 1e-13 and rel(fld[keep], f0) < 1e-13


@pytest.mark.parametrize("charges,dipoles", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("zk", [1e-6, 2.5, 3 + 0.5j, 0.7j, 3e5, 3e5 + 0.2j])
@pytest.mark.parametrize("n,m", [(1, 1), (31, 33), (32, 32), (65, 97), (160, 3)])
def test_helmholtz_one_leaf(F, n, m, zk, charges, dipoles):
    """The Helmholtz near field alone.  The phase |k| r carries at most 16 roundings on both sides
    together, so 16 eps |k| sqrt(3) is added to the bound; |k| = 3e5 has phases on both sides of
    2^17, where the sine and cosine change from the polynomial to the library."""
    rng = np.random.default_rng(1000 * n + m)
    src, trg = rng.random((n, 3)), rng.random((m, 3))
    q = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) if charges else None
    ds = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) if dipoles else None
    dv = rng.normal(size=(n, 3)) if dipoles else None
    tol = 1e-13 + 16 * 2.0 ** -52 * abs(zk) * 3 ** 0.5
    ier, pot, fld, pt, ft = F.hfmm3dparttarg(1, zk, src, int(charges), q, int(dipoles), ds, dv, 1, 1, trg, 1, 1)
    assert ier == 0, F.last_error()
    p0, f0 = O.hdirect_at(zk, src, src, np.arange(n), q, ds, dv)
    p1, f1 = O.hdirect_at(zk, src, trg, None, q, ds, dv)
    if n > 1:
        assert rel(pot, p0) < tol and rel(fld, f0) < tol
    else:
        assert not np.any(pot) and not np.any(fld)
    assert rel(pt, p1) < tol and rel(ft, f1) < tol
