"""Folded dense M2L (m2l_mode 0 / 2) against the rotate-shift-rotate kernel on the CUDA cores (mode 3).

Both apply the same linear maps in FP64, in different orders: a target's local expansion sums at
most 189 translations of at most (p + 1)^2 terms each, so the outputs agree to
189 (p + 1)^2 eps ~ 3e-11 in the worst case and to a few sqrt of that in practice; 1e-12 relative L2
is asked.  The sizes put the number of target boxes below, at and above one tile, below and above
the count from which a tile's partial sums run in one CTA, and leave boxes without sources, without
targets and without most of their reflections (surfaces, clusters).
"""
import numpy as np
import pytest

from test_gpu_lap import geometry

pytestmark = pytest.mark.gpu


@pytest.fixture()
def F():
    import fmmlib3d_b200 as F
    yield F
    F.set_m2l_mode(0)


def _call(F, iprec, src, q, trg, self_out):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    s, c, e = t(src), t(q), t(trg)
    new = lambda k, w: torch.full((k, w), np.nan, dtype=torch.float64, device="cuda")
    o = [new(len(src), 2), new(len(src), 6)] if self_out else [None, None]
    o += [new(len(trg), 2), new(len(trg), 6)]
    torch.cuda.synchronize()
    assert F.lfmm3dparttarg_device(iprec, s, c, None, None, o[0], o[1], e, o[2], o[3]) == 0, F.last_error()
    return [a.cpu().numpy() for a in o if a is not None]


@pytest.mark.parametrize("geom,n,m,iprec,self_out", [
    ("cube", 200, 150, 1, True),          # two levels or fewer: a few boxes, one ragged tile
    ("cube", 2000, 2000, 1, True),
    ("cube", 40, 9000, 1, True),          # few sources: most boxes empty of them
    ("cube", 6000, 30, -2, True),         # order 2, deep tree for its size
    ("sphere", 20011, 1, 0, True),
    ("two_clusters", 9000, 500, -1, True),
    ("plummer", 30011, 4001, 1, False),   # targets only: boxes without targets are pruned
    ("cube", 400003, 1000, 0, True),      # more than 296 tiles: all partial sums in one CTA
    ("plummer", 20000, 3000, 2, True),    # order 26
    ("sphere", 300007, 100, 2, False),
    ("cube", 400003, 1000, 2, True),      # order 26, sums in two pieces
])
def test_folded_m2l_matches_rotations(F, geom, n, m, iprec, self_out):
    rng = np.random.default_rng(n + m)
    src, trg = geometry(geom, n, rng), geometry(geom, m, rng) * 1.05
    q = rng.uniform(-1, 1, (n, 2))
    F.set_m2l_mode(0)
    a = _call(F, iprec, src, q, trg, self_out)
    F.set_m2l_mode(3)
    b = _call(F, iprec, src, q, trg, self_out)
    for x, y in zip(a, b):
        assert np.all(np.isfinite(x))
        assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("geom,n,iprec", [("cube", 20011, 1), ("plummer", 30011, 0), ("sphere", 9001, -1)])
def test_mixed_form_with_the_folded_m2l(F, geom, n, iprec):
    """The mixed form's FP64 M2L (the default there): error against the direct sum at most twice the
    FP64 form's, or, where that is below the floor of the FP32 near field (1e-8), no worse than with
    the FP32 M2L on the CUDA cores."""
    import oracle as O
    rng = np.random.default_rng(n)
    src = geometry(geom, n, rng)
    q = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    call = lambda: F.lfmm3dpartself(iprec, src, 1, q, 0, None, None, 1, 1)
    full = call()
    F.set_precision(1)
    try:
        F.set_tensor_m2l(0)
        cuda = call()
        F.set_tensor_m2l(3)
        fold, again = call(), call()
    finally:
        F.set_tensor_m2l(3)
        F.set_precision(0)
    si = rng.choice(n, 400, replace=False)
    exact = O.direct_at(src, src[si], si, q)
    err = lambda a, d: np.linalg.norm(a[si] - d) / np.linalg.norm(d)
    for k in (1, 2):
        assert np.array_equal(fold[k], again[k])
        e, e64, e32 = (err(x[k], exact[k - 1]) for x in (fold, full, cuda))
        assert e <= 2 * e64 or (e < 1e-8 and e <= 1.02 * e32), (e, e64, e32)
