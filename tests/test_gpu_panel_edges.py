"""The panel kernel at the edges of its strips, tiles and CTAs: supernodes of widths on both sides of 8
(inverted in the panel), 16 (the narrow launch), 64 and 128 (the panels), with 0, 1, 15, 16, 17, 127,
128, 129 and 300 rows below (groups of 16, CTAs of 128), in FP64 and in FP32. A dense block of w columns
and one of 2, both joined to a separator that makes the rows below; the handle is planned on the
analysis' own supernodes (merging would take block and separator together), which each test finds in
the structure before it trusts what it tested, and once more on the merged ones.

A Cholesky solve's residual is within n eps ||A|| ||x|| (n <= 500: 6e-14, held to 1e-13; the FP32 factor
after refinement to 1e-12), and a pivot that is not positive is named by its own column."""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import FP32_IR, FP64, NotPositiveDefinite, Symbolic, UpperColumns

pytestmark = pytest.mark.gpu


def matrix(w, rows, seed):
    rng = np.random.default_rng(seed)
    n = w + 2 + rows
    a = rng.standard_normal((n, n)) * 0.5
    a[:w, w:w + 2] = 0.0  # the two blocks meet in the separator only
    a[w:w + 2, :w] = 0.0
    return a + a.T + np.eye(n) * 3.0 * np.sqrt(n)


def csr_of(a):
    n = a.shape[0]
    return H.rows_to_csr([[(j, a[i, j]) for j in range(n) if a[i, j] != 0] for i in range(n)])


def analysed(a, w, rows):
    """The analysis of a, with a supernode of w columns and `rows` rows below them in it."""
    up = UpperColumns.from_symmetric(csr_of(a))
    sym = Symbolic(up, 2**62)
    s = sym.arrays()
    width = np.diff(s["first"])
    assert (w, rows) in zip(width, np.diff(s["rptr"]) - width)
    return up, sym


@pytest.mark.parametrize("w", [1, 7, 8, 9, 15, 16, 17, 33, 63, 64, 65, 127, 130])
@pytest.mark.parametrize("rows", [0, 1, 15, 16, 17, 127, 128, 129, 300])
def test_widths_and_rows(cuda, w, rows):
    a = matrix(w, rows, 7 * w + rows)
    up, sym = analysed(a, w, rows)
    b = np.random.default_rng(1).standard_normal(up.n)
    for merge in (False, True):
        f = H.factor_on(sym, merge)
        f.factor(up.val)
        x = b.copy()
        f.solve(x)
        assert np.linalg.norm(a @ x - b) <= 1e-13 * np.linalg.norm(a) * np.linalg.norm(x)
        f.close()


@pytest.mark.parametrize("w,rows", [(1, 1), (8, 17), (9, 128), (16, 130), (17, 16), (64, 129), (65, 300)])
def test_single_precision(cuda, w, rows):
    torch = cuda
    a = matrix(w, rows, w)
    csr = csr_of(a)
    up, sym = analysed(a, w, rows)
    for merge in (False, True):
        f = H.factor_on(sym, merge, FP32_IR)
        f.factor(up.val)
        dev = [torch.from_numpy(v).cuda() for v in (csr.ptr, csr.idx, csr.val)]
        b = torch.randn((1, csr.n), dtype=torch.float64, device="cuda")
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        rel, _ = f.refine_solve_device(dev, b, x, 1, csr.n, tol=1e-12, max_iter=20)
        assert rel[0] <= 1e-12
        f.close()


@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
@pytest.mark.parametrize("merge", [False, True], ids=["own", "merged"])
@pytest.mark.parametrize("w", [1, 8, 9, 64, 65, 130])
def test_a_failed_pivot_is_named(cuda, w, merge, precision):
    """The columns of the block are pivoted in their order: a negative diagonal entry at column c of it
    fails at c, wherever c lies in its strip and panel."""
    a = matrix(w, 20, 3 * w)
    up, sym = analysed(a, w, 20)
    perm = sym.arrays()["perm"]
    f = H.factor_on(sym, merge, precision)
    for at in sorted({0, w // 2, w - 1}):
        k = int(perm[np.flatnonzero(perm < w)[at]])  # a column of the block, by its place in the order
        bad = a.copy()
        bad[k, k] = -1.0
        with pytest.raises(NotPositiveDefinite) as e:
            f.factor(UpperColumns.from_symmetric(csr_of(bad)).val)
        assert e.value.column == k
    f.factor(up.val)
    b = np.ones(up.n)
    f.solve(b)
    assert np.linalg.norm(a @ b - 1.0) <= (1e-13 if precision == FP64 else 1e-4) * np.linalg.norm(a) * np.linalg.norm(b)
    f.close()
