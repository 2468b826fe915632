"""Charges that are not finite reach no sum that does not contain them: a point's potential is its own sum's
IEEE value, whatever the kernels keep beside it in a tile, a panel or a warp."""
import numpy as np
import pytest

import afmm2d_b200 as A

pytestmark = pytest.mark.gpu


def leaf_members(a):
    """Original indices of every leaf's points."""
    counts, _ = a.leaves()
    return np.split(a.permutation(), np.cumsum(counts)[:-1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_infinite_charge_in_the_far_field_tables(precision):
    """The log kernel is negative inside the unit square, and a leaf's far field holds no charge of the leaf:
    with one infinite charge the other points of its leaf have -inf.  Ranks near 30 give each warp of a box
    more far-field columns than it stages at once; leaves of 64 points fill the near field's blocks."""
    N, M = 16384, 64
    rng = np.random.default_rng(5)
    a = A.AFMM(N, M, 10, rng.uniform(0, 1, (N, 2)), kernel="log")
    a.assemble()
    assert a.ranks(a.nLevels).mean() > 26
    members = leaf_members(a)
    q0 = rng.standard_normal(N)
    for leaf in range(0, len(members), 37):
        q = q0.copy()
        j = members[leaf][leaf % M]
        q[j] = np.inf
        others = members[leaf][members[leaf] != j]
        y = a.computeMatVecProduct(q, precision=precision)
        assert np.all(y[others] == -np.inf), leaf
        if precision == "fp64" and leaf % 2 == 0:
            st = A.AFMMSet([a])
            assert np.all(st.matvec([q])[0][others] == -np.inf), leaf
            st.close()


@pytest.mark.parametrize("N,M", [(7168, 7), (41984, 41), (8320, 130)])
def test_infinite_charge_in_ragged_leaves(N, M):
    """Leaves that do not fill the near field's blocks of 32 sources: a block then holds sources of the leaf
    itself beside others, and unused lanes.  The Gaussian is positive, at distance zero too, so one infinite
    charge makes its leaf's potentials +inf, and no far field of the leaf holds it."""
    rng = np.random.default_rng(N)
    a = A.AFMM(N, M, 6, rng.uniform(0, 1, (N, 2)), kernel="gaussian", kparam=0.1)
    a.assemble()
    members = leaf_members(a)
    q0 = rng.standard_normal(N)
    for leaf in range(0, len(members), max(1, len(members) // 11)):
        q = q0.copy()
        q[members[leaf][leaf % len(members[leaf])]] = np.inf
        assert np.all(a.computeMatVecProduct(q)[members[leaf]] == np.inf), leaf
