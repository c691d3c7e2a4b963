"""The weight and bias gradients' sums (conv3_dw) against 64-bit ones of the same BF16 numbers, on short
and long chunks and every pair of channel counts, for sums that cancel and sums of one sign.

The tensor pipe truncates the sums it holds, which four products of 16 voxels go through (at most four
times 2^-23 of a group's sum); a chunk's n groups are then added in rounded FP32, whose errors of 2^-24
at most add up as sqrt(n) where their signs are random. Kept in the pipe over a whole chunk the largest
grid's sums here were off by 1.0e-6 to 4.9e-6, five times this bound."""
import ctypes as C

import numpy as np
import pytest

from fieldcraft_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,pairs,passes", [((5, 5, 2), 1, 1), ((17, 17, 5), 8, 2), ((33, 33, 9), 1, 2),
                                               ((33, 33, 9), 8, 2), ((65, 65, 9), 8, 2), ((24, 7, 40), 3, 1)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (16, 32), (32, 16), (16, 16)])
@pytest.mark.parametrize("sign", ["both", "one"])
def test_against_64_bit_sums(cuda, grid, pairs, passes, cin, cout, sign):
    torch = cuda
    X, Y, Z = grid
    g = torch.Generator(device="cuda").manual_seed(X + cin)
    x = torch.randn((pairs * passes, Z, Y, X, cin), device="cuda", generator=g)
    x = torch.where(x > 0, x, 0.05 * x).bfloat16()  # activations
    dy = torch.randn((pairs * passes, Z, Y, X, cout), device="cuda", generator=g)
    dy = (dy if sign == "both" else dy.abs()).bfloat16()
    gw, gb = torch.empty((27, cout, cin), device="cuda"), torch.empty(cout, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert _lib.load().fc_test_unet_dw(X, Y, Z, cin, cout, pairs, passes, p(x), p(dy), C.c_float(1.0 / pairs), p(gw),
                                       p(gb)) == 0
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    d = dy.double().view(-1, cout) / pairs
    want = torch.stack([d.T @ xp[:, t // 9:t // 9 + Z, t // 3 % 3:t // 3 % 3 + Y, t % 3:t % 3 + X].reshape(-1, cin)
                        for t in range(27)])
    groups = X * Y * Z * pairs * passes / 148 / 64
    bound = 2.0**-24 * (8 + np.sqrt(groups))
    error = ((gw.double() - want).norm() / want.norm()).item()
    bias = ((gb.double() - d.sum(0)).norm() / d.sum(0).norm()).item()
    print(f"{error:.2e} {bias:.2e} of {bound:.2e}")
    assert error <= bound
    # a bias gradient that cancels is small beside its terms
    assert bias <= bound * (1 if sign == "one" else (d.abs().sum(0).norm() / d.sum(0).norm()).item())
