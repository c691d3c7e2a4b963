"""One LDL^T handle through factorisations whose pivots differ: the solve's plan is made once and
follows each factorisation's pivots through the device's own maps. Dense supernodes on both sides of
the 64-column panel and of several panels, with rows of a second supernode below them.

The residual of a solve with a factor of bounded element growth is within n eps growth of
||A|| ||x||: 200 x 1.1e-16 with a growth of a few hundred at most here, under 1e-11."""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import LdltFactor, Symbolic, UpperColumns

pytestmark = pytest.mark.gpu


def matrix(w, tail, seed):
    """A dense indefinite block of w columns with zeros on its diagonal (2 x 2 pivots), joined to a
    definite tail."""
    rng = np.random.default_rng(seed)
    n = w + tail
    a = rng.standard_normal((n, n))
    a = a + a.T
    a[np.arange(1, w, 3), np.arange(1, w, 3)] = 0.0
    a[w:, w:] += np.eye(tail) * 4.0 * n
    return a


@pytest.mark.parametrize("w,tail", [(1, 0), (8, 3), (63, 10), (64, 65), (65, 1), (129, 30), (200, 17)])
@pytest.mark.parametrize("nrhs", [1, 5, 70])
def test_solves_follow_each_factorisations_pivots(cuda, w, tail, nrhs):
    n = w + tail
    f = None
    orders = []
    for seed in (1, 2, 3):
        a = matrix(w, tail, seed)
        csr = H.rows_to_csr([[(j, a[i, j]) for j in range(n)] for i in range(n)])
        up = UpperColumns.from_symmetric(csr)
        if f is None:
            f = LdltFactor(Symbolic(up, 2**62))
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
