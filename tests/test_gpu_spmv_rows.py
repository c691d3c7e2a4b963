"""The compressed-row product's kernels at rows on both sides of their strides (16 lanes a row, one,
two or four entries a lane in flight; a warp a row with 4 or more vectors in rows) and at every
count of vectors a kernel is chosen by, against FP64 sums on the host; and flexible CG's fused
iteration on systems whose order is no multiple of three, for every number of kept directions.

A row's sum of k products in any order is within (k + 1) eps sum |a x| of the exact one."""
import numpy as np
import pytest

from fieldcraft_b200 import _lib
from fieldcraft_b200.unet import fcg

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 81, 82, 112, 113, 200]


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65])
def test_rows_of_every_length(cuda, nrhs):
    torch = cuda
    rng = np.random.default_rng(nrhs)
    n = 211
    counts = np.array([LENGTHS[i % len(LENGTHS)] for i in range(n)])
    ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in counts]).astype(np.int32)
    val = rng.standard_normal(idx.size)
    ld = n + 3
    x = rng.standard_normal((nrhs, ld))
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    d = [dev(a) for a in (ptr, idx, val, x)]
    y = torch.full((nrhs, ld), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = _lib.load().fc_csr_spmv_device(n, *[_lib.ptr(a) for a in d], _lib.ptr(y), nrhs, ld, None)
    assert rc == 0
    torch.cuda.synchronize()
    got = y.cpu().numpy()
    assert np.all(got[:, n:] == 7.0)
    a, mag = np.zeros((n, n)), np.zeros((n, n))
    rows = np.repeat(np.arange(n), counts)
    a[rows, idx], mag[rows, idx] = val, np.abs(val)
    bound = (counts + 1) * 2.3e-16 * (np.abs(x[:, :n]) @ mag.T)
    assert np.all(np.abs(got[:, :n] - x[:, :n] @ a.T) <= 2 * bound)  # the host's own sum rounds too


@pytest.mark.parametrize("n", [1, 2, 97, 256, 769, 4000])
@pytest.mark.parametrize("keep", [1, 2, 5, 8])
def test_fused_iteration(cuda, n, keep):
    """Plain flexible CG on a shifted path graph's Laplacian (condition below 10): 1e-10 within the
    40 iterations that CG's bound 2 ((sqrt k - 1) / (sqrt k + 1))^i gives, rounded up to the next
    look at the residuals."""
    torch = cuda
    ptr, idx, val = [0], [], []
    for i in range(n):
        for j in (i - 1, i, i + 1):
            if 0 <= j < n:
                idx.append(j)
                val.append(2.5 if i == j else -1.0)
        ptr.append(len(idx))
    csr = [torch.tensor(a, dtype=t, device="cuda") for a, t in
           ((ptr, torch.int64), (idx, torch.int32), (val, torch.float64))]
    b = torch.from_numpy(np.random.default_rng(n).standard_normal(n)).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    it, rel, fell_back = fcg(csr, b, x, tol=1e-10, max_iter=100, keep=keep)
    assert rel <= 1e-10 and not fell_back and it <= 40
