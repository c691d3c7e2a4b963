"""How often the panel rounds an entry at the entry's own size. Dense matrices with a diagonal of 1 000 and the
rest between 1.2 and 1.8: an update takes about 0.002 from an entry, so each operation on the entry itself
rounds it by up to 2^-53 (uniformly: 2^-53 / sqrt 3 in the root mean square) and A - L L^T counts them.

An entry's division leaves about 1.85 x 2^-53: the root's error of 0.48 twice and the roundings of L's two
factors, 1.2 in all, times the entries' 1.5. All earlier strips' products are summed apart and taken from
the entry at once. In the panel's block the strip's own, 3.5 on average, come one by one: sqrt(4.5 / 3 +
1.85^2) = 2.2, held to 2.4 (each strip's sum taken by itself: 2.5, each product of the last strip too 2.9).
Below the block these are summed as well: sqrt(2 / 3 + 1.85^2) = 2.0, held to 2.2 (each product by
itself: 4.4). Over the panel's last four strips; in the host's extended format.
"""
import numpy as np
import pytest

import helpers as H
from fieldcraft_b200 import Factor, Symbolic, UpperColumns

pytestmark = pytest.mark.gpu


def test_roundings_in_a_panel(cuda):
    n, block, below = 194, [], []
    for seed in range(8):
        rng = np.random.default_rng(seed)
        a = rng.uniform(1.2, 1.8, (n, n))
        a = np.tril(a, -1) + np.tril(a, -1).T + np.diag(rng.uniform(1000.0, 1020.0, n))
        up = UpperColumns.from_symmetric(H.rows_to_csr([[(j, a[i, j]) for j in range(n)] for i in range(n)]))
        sym = Symbolic(up, 2**62)
        s = sym.arrays()
        assert s["ns"] == 1
        f = Factor(sym)
        f.factor(up.val)
        lower = np.zeros((n, n), np.longdouble)
        packed, at = f.values(), 0
        for c in range(n):
            lower[c:, c] = packed[at:at + n - c]
            at += n - c
        f.close()
        p = s["perm"]
        e = (a[np.ix_(p, p)].astype(np.longdouble) - lower @ lower.T).astype(float) / 2.0**-53
        block += [e[c + 1:64, c] for c in range(32, 64)]
        below += [e[64:, c] for c in range(32, 64)]
    rms = [np.sqrt(np.mean(np.concatenate(v)**2)) for v in (block, below)]
    print("%.2f %.2f" % tuple(rms))
    assert rms[0] <= 2.4 and rms[1] <= 2.2
