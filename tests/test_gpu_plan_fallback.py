"""The plans that a handle falls back to where memory is short: the analysis' own supernodes when the
merged ones find no room, and the allocation-free solve without the split products' partial sums when
those do not fit its scratch. Both decide whether a call that was accepted still is; both solve to
n eps ||A|| ||x|| (n <= 14 000: 2e-12)."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import FP32_IR, FP64, Factor, LdltFactor, Symbolic, _lib, problems
from fieldcraft_b200._lib import Status
from fieldcraft_b200.cholesky import OutOfMemory

pytestmark = pytest.mark.gpu

SCRATCH = 32 << 20  # FC_NOALLOC_SCRATCH_BYTES


def residual(csr, x, b):
    rows = np.repeat(np.arange(csr.n), np.diff(csr.ptr))
    r = np.stack([np.bincount(rows, csr.val * x[csr.idx, j], minlength=csr.n) for j in range(b.shape[1])], axis=1) - b
    norm = np.max(np.bincount(rows, np.abs(csr.val)))
    return np.linalg.norm(r) / (norm * np.linalg.norm(x))


@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
@pytest.mark.parametrize("name", ["block", "plate", "beam"])
def test_a_refused_plan_is_made_on_the_analysis_own_supernodes(cuda, name, precision):
    torch = cuda
    p = {"block": lambda: problems.lognormal_block(8, nrhs=3), "plate": lambda: problems.plate(20, 14, 2),
         "beam": problems.cantilever}[name]()
    up = p.upper()
    sym = Symbolic(up, 2**62)
    b = np.asfortranarray(np.random.default_rng(2).standard_normal((p.n, 3)))
    merged, own, refused = (H.factor_on(sym, m, precision, k) for m, k in ((True, 0), (False, 0), (True, 1)))
    assert all(own.stat(k) > merged.stat(k) for k in (1, 17, 18))  # the plans' launches, levels, supernodes
    assert [refused.stat(k) for k in (1, 2, 3, 17, 18)] == [own.stat(k) for k in (1, 2, 3, 17, 18)]
    found = []
    for f in (merged, own, refused):
        f.factor(up.val)
        x = b.copy(order="F")
        if precision == FP64:
            f.solve_many(x)
        else:
            dev = [torch.from_numpy(v).cuda() for v in (p.csr.ptr, p.csr.idx, p.csr.val)]
            db = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
            dx = torch.zeros_like(db)
            torch.cuda.synchronize()
            f.refine_solve_device(dev, db, dx, 3, p.n, tol=1e-10, max_iter=40)
            x = dx.cpu().numpy().T
        assert residual(p.csr, x, b) <= 2e-12
        found.append((x, f.values()))
        f.close()
    assert np.array_equal(found[1][0], found[2][0]) and np.array_equal(found[1][1], found[2][1])
    if precision == FP64:  # the values as the parity tests hold them; the FP32 factor's follow its condition
        assert np.max(np.abs(found[0][1] - found[1][1])) <= 1e-11 * np.max(np.abs(found[1][1]))


@pytest.mark.parametrize("name", ["block", "beam"])
def test_the_analysis_levels_and_supernodes_whatever_the_plan(cuda, name):
    up = {"block": lambda: problems.lognormal_block(9, nrhs=1), "beam": problems.cantilever}[name]().upper()
    sym = Symbolic(up, 2**62)
    s = sym.arrays()
    owner = np.repeat(np.arange(s["ns"]), np.diff(s["first"]))
    height = np.ones(s["ns"], int)
    for k in range(s["ns"]):  # children before parents: the parent owns the first row below
        rows = s["rows"][s["rptr"][k] + s["first"][k + 1] - s["first"][k]:s["rptr"][k + 1]]
        if rows.size:
            height[owner[rows[0]]] = max(height[owner[rows[0]]], height[k] + 1)
    merged, own, ldlt = H.factor_on(sym, True), H.factor_on(sym, False), LdltFactor(sym)
    for f in (merged, own, ldlt):
        assert (f.stat(0), f.stat(4)) == (height.max(), s["ns"])
    assert (own.stat(17), own.stat(18)) == (ldlt.stat(17), ldlt.stat(18)) == (height.max(), s["ns"])


def test_no_plan_at_all_is_out_of_memory(cuda):
    sym = Symbolic(problems.cantilever().upper(), 2**62)
    with pytest.raises(OutOfMemory):
        H.factor_on(sym, True, refused=2)
    with pytest.raises(OutOfMemory):
        H.factor_on(sym, False, refused=1)
    H.factor_on(sym, True).close()


@pytest.mark.parametrize("precision", [FP64, FP32_IR], ids=["fp64", "fp32_ir"])
def test_the_allocation_free_solve_without_split_products(cuda, precision):
    torch = cuda
    lib = _lib.load()
    lib.fc_test_noalloc_need.restype = C.c_int64
    p = problems.lognormal_block(16, nrhs=1)
    up = p.upper()
    f = Factor(Symbolic(up, 2**62), precision=precision)
    f.factor(up.val)
    need = lambda r, split: lib.fc_test_noalloc_need(f.handle, r, split)  # noqa: E731
    counts = range(1, SCRATCH // (16 * p.n) + 1)
    only = [r for r in counts if need(r, 1) > SCRATCH >= need(r, 0)]
    assert only
    st = Status()
    for r in (only[0], only[-1]):
        b = np.asfortranarray(np.random.default_rng(r).standard_normal((p.n, r)))
        x = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
        want = x.clone()
        torch.cuda.synchronize()
        assert lib.fc_chol_solve_device_noalloc(f.handle, C.c_void_p(x.data_ptr()), r, p.n, C.byref(st)) == 0
        f.solve_device(want, r, p.n)
        torch.cuda.synchronize()
        assert ((x - want).norm() / want.norm()).item() <= (1e-10 if precision == FP64 else 1e-4)
        if precision == FP64:
            assert residual(p.csr, x.cpu().numpy().T, b) <= 2e-12
    over = next(r for r in range(only[-1], only[-1] + 2000) if need(r, 0) > SCRATCH)
    b = torch.zeros((over, p.n), dtype=torch.float64, device="cuda")
    assert lib.fc_chol_solve_device_noalloc(f.handle, C.c_void_p(b.data_ptr()), over, p.n, C.byref(st)) != 0
    assert str(need(over, 0)).encode() in st.message
    f.close()
