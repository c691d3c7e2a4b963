"""The panel's own 1 / sqrt(a) and 1 / a (csrc/cuda/kernels.cu, inverse_root) against 64-bit significands,
over every exponent, at powers of two and the numbers beside them, and on both sides of the two ends
(1e-280, 1e280) past which it takes CUDA's rsqrt.

With an estimate within 2^-20 of the root, e = 1 - a y^2 is at most 2^-19 and its own error 2^-53 (the
rounding of a y, times y), so that
  root     errs by half of e's error, its last rounding and 5 e^3 / 16: under 1.5 x 2^-53 + 2^-58,
  inverse  by e's error, the rounding of y^2, its last and e^3: under 3 x 2^-53 + 2^-57.
Past the ends: rsqrt's documented unit in the last place (2^-52), and twice that and two roundings."""
import ctypes as C

import numpy as np
import pytest

from fieldcraft_b200 import _lib

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def inputs():
    rng = np.random.default_rng(1)
    exponents = np.arange(-1022, 1024)
    some = np.ldexp(1.0 + rng.random((40, exponents.size)), exponents).ravel()
    powers = np.ldexp(1.0, exponents)
    ends = np.concatenate([v * (1.0 + np.arange(-8, 9) * 2.0 ** -52) for v in (1e-280, 1e280)])
    subnormal = np.ldexp(1.0 + rng.random(200), rng.integers(-1070, -1022, 200))
    return np.concatenate([some, powers, np.nextafter(powers, 0.0)[1:], np.nextafter(powers, np.inf), ends,
                           np.ldexp(1.0 + rng.random(100000), rng.integers(-3, 3, 100000)), subnormal])


def test_against_wider_significands(cuda):
    torch = cuda
    assert np.finfo(np.longdouble).nmant >= 63
    a = inputs()
    d = torch.from_numpy(a).cuda()
    out = [torch.empty_like(d) for _ in range(3)]
    torch.cuda.synchronize()
    assert _lib.load().fc_test_inverse_root(C.c_int64(a.size), *(C.c_void_p(t.data_ptr()) for t in (d, *out))) == 0
    up, root, inverse = (t.cpu().numpy() for t in out)
    assert np.all(np.frexp(up)[0] == 0.5)
    normal = (a >= np.ldexp(1.0, -1021)) & (a < np.ldexp(1.0, 1023))  # up is a's own power of two
    assert np.all((up[normal] <= a[normal]) & (a[normal] < 2.0 * up[normal]))
    wide = a.astype(np.longdouble)
    root_error = np.abs(root * np.sqrt(wide) - 1).astype(float)
    inverse_error = np.abs(inverse * (wide / up) - 1).astype(float)
    near = (a > 1e-280) & (a < 1e280)
    print(f"root {root_error[near].max() / EPS:.3f}, inverse {inverse_error[near].max() / EPS:.3f}; past the ends "
          f"{root_error[~near].max() / EPS:.3f}, {inverse_error[~near].max() / EPS:.3f} x 2^-53")
    assert root_error[near].max() <= 1.5 * EPS + 2.0 ** -58
    assert inverse_error[near].max() <= 3 * EPS + 2.0 ** -57
    assert root_error[~near].max() <= 2 * EPS
    assert inverse_error[~near].max() <= 6 * EPS


def test_what_is_not_positive(cuda):
    """The pivot test refuses a zero, a negative number, an infinity and a NaN by the pivot itself; the
    factors formed from them are no finite numbers, or zero, and nothing else."""
    torch = cuda
    a = np.array([0.0, -0.0, -1.0, -1e300, -1e-300, np.inf, -np.inf, np.nan])
    d = torch.from_numpy(a).cuda()
    out = [torch.empty_like(d) for _ in range(3)]
    torch.cuda.synchronize()
    assert _lib.load().fc_test_inverse_root(C.c_int64(a.size), *(C.c_void_p(t.data_ptr()) for t in (d, *out))) == 0
    root = out[1].cpu().numpy()
    assert np.all(~np.isfinite(root) | (a == np.inf) & (root == 0.0))
