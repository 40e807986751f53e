"""Octrees whose depth or size crosses a line of the builder.

The builder sorts the key bits of 13 levels first and all bits when a tree goes deeper, builds
several levels between two reads of their counts, and grows its arrays when a level does not fit.
The tree of every case must equal the oracle's box for box (count, levels, leaves) and the FMM its
direct sum within the precision's bound; exact equality, no tolerance, for the tree.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import fmmlib3d_b200
    return fmmlib3d_b200


def nested(n, levels, rng):
    """n points in each of `levels` shells, every one half the size of the last."""
    return np.concatenate([0.4 * 0.5 ** k * (rng.random((n, 3)) - 0.3) for k in range(levels)])


@pytest.mark.parametrize("name", ["shells 11", "shells 13", "shells 14", "shells 17", "one box", "line", "targets only deep"])
def test_tree_equals_oracle(F, name):
    rng = np.random.default_rng(len(name))
    trg = rng.random((500, 3)) * 0.3
    if name.startswith("shells"):
        src = nested(400, int(name.split()[1]), rng)
    elif name == "one box":
        src, trg = rng.random((160, 3)), rng.random((160, 3))
    elif name == "line":
        # 2^-k spacings on a line: many levels with few boxes, more boxes than points / nbox suggests
        src = np.zeros((6000, 3))
        src[:, 0] = 0.5 ** (np.arange(6000) / 450.0)
    else:
        src, trg = rng.random((50, 3)), nested(400, 15, rng)
    q = rng.uniform(-1, 1, len(src)) + 0j
    F.set_stats(True)
    ier, pot, _, pt, _ = F.lfmm3dparttarg(1, src, 1, q, 0, None, None, 1, 0, trg, 1, 0)
    F.set_stats(False)
    assert ier == 0, F.last_error()
    st = F.last_stats()
    T = O.Tree(src, trg, 160)
    assert (st["nboxes"], st["nlev"], st["nleaves"]) == (T.nboxes, T.nlev, int(np.sum(T.box[:, 5] < 0)))
    i = rng.choice(len(src), min(len(src), 200), replace=False)
    j = rng.choice(len(trg), min(len(trg), 200), replace=False)
    p0, _ = O.direct_at(src, src[i], i, q)
    p1, _ = O.direct_at(src, trg[j], None, q)
    for a, b in ((pot[i], p0), (pt[j], p1)):
        assert np.linalg.norm(a - b) <= 5e-4 * np.linalg.norm(b)
