"""One LDL^T handle through factorisations whose pivots differ: the solve's plan is made once and
follows each factorisation's pivots through the device's own maps. Dense supernodes on both sides of
the 64-column panel and of several panels, two of them beside one another and the rows of a third
below both, so that a child's rows are found through the pivots of its own columns and of its
parent's; each test finds the three in the structure first.

The residual of a solve with a factor of bounded element growth is within n eps growth of
||A|| ||x||: 300 x 1.1e-16 with a growth of a few hundred at most here, under 1e-11."""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import LdltFactor, Symbolic, UpperColumns

pytestmark = pytest.mark.gpu


def matrix(w, other, tail, seed):
    """Dense indefinite blocks of w and `other` columns with zeros on their diagonals (2 x 2 pivots),
    joined by an indefinite separator of `tail` columns."""
    rng = np.random.default_rng(seed)
    n = w + other + tail
    a = rng.standard_normal((n, n))
    a = a + a.T
    a[:w, w:w + other] = 0.0
    a[w:w + other, :w] = 0.0
    a[np.arange(1, n, 3), np.arange(1, n, 3)] = 0.0
    return a


@pytest.mark.parametrize("w,other,tail", [(1, 2, 1), (8, 5, 3), (63, 9, 10), (64, 64, 65), (65, 3, 1), (129, 40, 30),
                                          (200, 70, 17)])
@pytest.mark.parametrize("nrhs", [1, 5, 70])
def test_solves_follow_each_factorisations_pivots(cuda, w, other, tail, nrhs):
    n = w + other + tail
    f = None
    orders = []
    for seed in (1, 2, 3):
        a = matrix(w, other, tail, seed)
        # the pattern is the first matrix's whatever values are zero
        keep = lambda i, j: not (i < w <= j < w + other or j < w <= i < w + other)  # noqa: E731
        csr = H.rows_to_csr([[(j, a[i, j]) for j in range(n) if keep(i, j)] for i in range(n)])
        up = UpperColumns.from_symmetric(csr)
        if f is None:
            sym = Symbolic(up, 2**62)
            s = sym.arrays()
            width = np.diff(s["first"])
            shapes = list(zip(width, np.diff(s["rptr"]) - width))
            assert (w, tail) in shapes and (other, tail) in shapes and (tail, 0) in shapes
            f = LdltFactor(sym)
            with pytest.raises(Exception, match="pivot orders"):
                f.solve(np.zeros(n))
        f.factor(up.val)
        b = np.asfortranarray(np.random.default_rng(seed + 9).standard_normal((n, nrhs)))
        x = b.copy(order="F")
        f.solve_many(x)
        assert np.linalg.norm(a @ x - b) <= 1e-11 * np.linalg.norm(a) * np.linalg.norm(x)
        before = f.values()
        again = b.copy(order="F")
        f.solve_many(again)
        assert np.array_equal(again, x) and np.array_equal(f.values(), before)
        orders.append(f.pivots()[1])
    if w > 8:
        assert not np.array_equal(orders[0], orders[1])
