"""The odd network's output biases have no gradient: they cancel between a pair's two passes, whose output
gradients are each other's negatives to the last bit. Summed alike, pass by pass, that leaves an exact
zero and Adam does not touch them; a residue of rounding alone, however small, it would blow up to a
step of its own size (from 1e-9 to a tenth of the learning rate). On one tile and on many, for batches
of one pair up to past a group, and where only one pass fits at a time. The plain network's biases do
move."""
import ctypes as C

import numpy as np
import pytest

from fieldcraft_b200 import _lib
from test_gpu_unet_batch import network
from test_gpu_unet_room import pairs, room

pytestmark = pytest.mark.gpu

OUT = 16  # output channels, the last of the parameters


@pytest.mark.parametrize("dims,levels", [((7, 7, 1), 2), ((16, 9, 2), 3), ((32, 32, 8), 3), ((48, 31, 7), 2)])
@pytest.mark.parametrize("count", [1, 3, 8, 11])
@pytest.mark.parametrize("own", [1, 2])
def test_output_biases_stay(cuda, dims, levels, count, own):
    torch = cuda
    p, net, flat = network(dims, levels, True)
    if own == 1:
        room(net, 1, 0)
    r, e = pairs(torch, p.n, count)
    for step in (1, 2):
        net.train_batch(r, e, 1e-3, step)
        assert np.all(net.grads()[-OUT:] == 0.0) and np.array_equal(net.params()[-OUT:], flat[-OUT:])
    net.train_step(r[0], e[0], 1e-3, 3)
    assert np.all(net.grads()[-OUT:] == 0.0) and np.array_equal(net.params()[-OUT:], flat[-OUT:])
    assert np.any(net.params() != flat)
    net.close()


def test_plain_biases_move(cuda):
    p, net, flat = network((16, 9, 2), 3, False)
    r, e = pairs(cuda, p.n, 3)
    net.train_batch(r, e, 1e-3, 1)
    assert np.all(net.params()[-OUT:-OUT + 3] != flat[-OUT:-OUT + 3])
    net.close()


@pytest.mark.parametrize("grid", [(5, 5, 2), (33, 33, 9), (41, 23, 10)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (16, 32), (32, 16), (16, 16)])
def test_opposite_passes_cancel(cuda, grid, cin, cout):
    """One input and two opposite output gradients: weights' and biases' gradients are exactly zero."""
    torch = cuda
    X, Y, Z = grid
    g = torch.Generator(device="cuda").manual_seed(X)
    x = torch.randn((Z, Y, X, cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((Z, Y, X, cout), device="cuda", generator=g).bfloat16()
    x, dy = torch.stack([x, x]), torch.stack([dy, -dy])
    gw, gb = torch.ones((27, cout, cin), device="cuda"), torch.ones(cout, device="cuda")
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert _lib.load().fc_test_unet_dw(X, Y, Z, cin, cout, 1, 2, ptr(x), ptr(dy), C.c_float(1.0), ptr(gw), ptr(gb)) == 0
    assert not torch.any(gw) and not torch.any(gb)
