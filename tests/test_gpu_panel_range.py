"""The Cholesky factor over FP64's exponent range. A matrix times a power of two, or scaled by a
diagonal of powers of two on both sides, has the same factor but for the exponents: the solve's
residual, with the scaling taken off again (exactly), is the unscaled one's, within n eps ||A|| ||x||
(n <= 180: 4e-14, held to 1e-13), and a matrix that is not definite is refused at its own column."""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import Factor, NotPositiveDefinite, UpperColumns

pytestmark = pytest.mark.gpu


def upper(a):
    n = a.shape[0]
    return UpperColumns.from_symmetric(H.rows_to_csr([[(j, a[i, j]) for j in range(n)] for i in range(n)]))


def definite(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n)) * 0.5
    return a + a.T + np.eye(n) * 3.0 * np.sqrt(n)


# 1e-250, 1e-165, 1e-160, 1e-156 and as far above 1, and both sides of 1e-280 and 1e280
EXPONENTS = [-930, -928, -830, -548, -532, -518, 0, 515, 532, 830, 928, 932]


@pytest.mark.parametrize("n", [8, 9, 64, 180])
@pytest.mark.parametrize("exponent", EXPONENTS)
def test_a_scaled_matrix(cuda, n, exponent):
    a = definite(n, n)
    f = Factor.new(upper(np.ldexp(a, exponent)), 2**62)
    b = np.random.default_rng(1).standard_normal(n)
    x = np.ldexp(b, exponent)
    f.solve(x)
    assert np.linalg.norm(a @ x - b) <= 1e-13 * np.linalg.norm(a) * np.linalg.norm(x)
    f.close()


@pytest.mark.parametrize("n", [8, 9, 64, 180])
@pytest.mark.parametrize("most", [100, 300, 450])
def test_a_matrix_of_uneven_scales(cuda, n, most):
    """D A D with D's exponents spread over +-most: entries of up to 2^(2 most) beside 2^(-2 most)."""
    a = definite(n, 3 * n)
    rng = np.random.default_rng(n + most)
    d = rng.integers(-most, most + 1, n)
    f = Factor.new(upper(np.ldexp(a, d[:, None] + d[None, :])), 2**62)
    b = rng.standard_normal(n)
    x = np.ldexp(b, d)
    f.solve(x)
    x = np.ldexp(x, d)
    assert np.linalg.norm(a @ x - b) <= 1e-13 * np.linalg.norm(a) * np.linalg.norm(x)
    f.close()


@pytest.mark.parametrize("exponent", EXPONENTS)
def test_a_scaled_indefinite_matrix_is_refused(cuda, exponent):
    a = definite(70, 5)
    a[66, 66] = -1.0
    with pytest.raises(NotPositiveDefinite) as e:
        Factor.new(upper(np.ldexp(a, exponent)), 2**62)
    assert e.value.column == 66
