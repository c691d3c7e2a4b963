"""The rows below a front's own columns, which the device's LDL^T panel leaves to a kernel of its own:
leaf supernodes (whose factor depends on A alone) of at most one panel come out the oracle's bit for
bit, with 1 x 1 and 2 x 2 pivots on both sides of that kernel's eight columns a thread and 32 rows a
block; a front of several panels, and one with more own rows than the panel holds columns for ahead,
solve to the residual bound of an indefinite factor."""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import LdltFactor, Symbolic, UpperColumns
from test_ldlt_panel_emulated import bits, dense_csr, indefinite, leaf_fronts, oracle_ldlt

pytestmark = pytest.mark.gpu


def two_blocks(w, below, seed):
    """Dense indefinite blocks of w and 2 columns joined by a separator of `below` columns."""
    n = w + 2 + below
    a = np.zeros((n, n))
    a[:w, :w] = indefinite(w, seed)
    a[w:w + 2, w:w + 2] = np.eye(2) * 9.0
    c = np.random.default_rng(seed + 1).standard_normal((w + 2, below))
    a[:w + 2, w + 2:] = c
    a[w + 2:, :w + 2] = c.T
    a[w + 2:, w + 2:] = np.eye(below) * (100.0 * n)
    return a


def device(csr):
    up = UpperColumns.from_symmetric(csr)
    f = LdltFactor(Symbolic(up, 2**62))
    f.factor(up.val)
    return f


@pytest.mark.parametrize("w,below", [(1, 1), (2, 33), (7, 31), (8, 32), (9, 70), (16, 64), (40, 129), (63, 5), (64, 200)])
def test_leaf_fronts_are_the_oracles_bit_for_bit(cuda, w, below):
    a = dense_csr(two_blocks(w, below, 10 * w + below))
    s, o = oracle_ldlt(a)
    f = device(a)
    values, want = f.values(), o.values()
    seen = []
    for _, front, width, _, vslice, cslice in leaf_fronts(a, s):
        assert np.array_equal(f.pivots()[1][cslice], o.pivots()[1][cslice])
        assert np.array_equal(bits(values[vslice]), bits(want[vslice]))
        seen.append((width, front.shape[0] - width))
    assert (w, below) in seen


@pytest.mark.parametrize("w,below", [(65, 40), (200, 77), (1100, 50)])
def test_many_panels(cuda, w, below):
    """||A x - b|| is within n eps growth of ||A|| ||x||: 1152 x 1.1e-16 with a growth of a hundred."""
    a = two_blocks(w, below, w)
    n = a.shape[0]
    csr = dense_csr(a)
    f = device(csr)
    b = np.random.default_rng(3).standard_normal(n)
    x = b.copy()
    f.solve(x)
    assert np.linalg.norm(a @ x - b) <= 1.5e-11 * np.linalg.norm(a, 2) * np.linalg.norm(x)
