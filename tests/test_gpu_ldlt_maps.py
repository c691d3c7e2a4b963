"""The LDL^T solve's maps as the device makes them after a factorisation (each column's place in the
solve's vectors, the permutation of the input, the row lists) against the host's fold of the same pivot
orders into the structure (csrc/host/ldlt_fold.cpp, itself checked in test_ldlt_fold.py), on trees of
many levels with interchanges, over two factorisations of one handle. The device keeps a row list in the
structure's order where the fold sorts it, so these are compared sorted, and through the fold's `from`
in the order it was sorted by."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import LdltFactor, Symbolic, UpperColumns, _lib
from oracle import oracle
from test_ldlt_fold import fold

pytestmark = pytest.mark.gpu

CASES = {
    "grid": lambda shift: H.shifted_grid([7, 6, 5], shift)[0],
    "saddle": lambda shift: H.saddle(8, 3),
    "wide": lambda shift: H.shifted_grid([14, 12, 10], shift)[0],
}


@pytest.mark.parametrize("name", list(CASES))
def test_maps_are_the_folds(cuda, name):
    f = None
    moved = 0
    for shift in (3.3, 2.7):
        a = CASES[name](shift)
        up = UpperColumns.from_symmetric(a)
        s = oracle.Sym(up.n, up.ptr, up.idx)
        first, rptr, rows = s.array("first"), s.array("rptr"), s.array("rows")
        if f is None:
            f = LdltFactor(Symbolic(up, 2**62))
        f.factor(up.val)
        order = f.pivots()[1]
        own, perm, listed = np.zeros(up.n, np.int32), np.zeros(up.n, np.int64), np.zeros(rows.size, np.int32)
        p = lambda v: C.c_void_p(v.ctypes.data)  # noqa: E731
        assert _lib.load().fc_test_ldlt_maps(f.handle, p(own), p(perm), p(listed)) == 0
        want_perm, want_rows, frm, _ = fold(s, order)
        assert np.array_equal(perm, want_perm)
        assert np.array_equal(s.array("perm"), want_perm[own])
        assert np.array_equal(listed, own[rows])
        at = 0
        for k in range(first.size - 1):
            w, m = first[k + 1] - first[k], rptr[k + 1] - rptr[k]
            here, want = listed[rptr[k]:rptr[k + 1]], want_rows[rptr[k]:rptr[k + 1]]
            assert np.array_equal(np.sort(here[:w]), want[:w]) and np.array_equal(here[w:][frm[at:at + m - w]], want[w:])
            at += m - w
        moved += int(np.sum(own != np.arange(up.n)))
    assert moved > 0
    f.close()
