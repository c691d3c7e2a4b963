"""Minibatches through the network in groups of pairs: a batch's losses and its last pair's gradient
are those of the pairs run alone, at batches of one, of part of a group, of a whole group and past
it, on grids of one tile a pass and of several, with fewer tiles in a batch than SMs (one halo buffer, a
tile a chunk) and with more (two buffers, several tiles a chunk), with the odd form and without.

The forward pass of a pair is the same arithmetic alone or in a batch (the loss agrees to FP64
rounding); its gradient is summed in other chunks: FP32 sums of N terms in another order differ by
about sqrt(N) eps of their magnitude, 2e-5 for the 10^5 terms of a weight here."""
import numpy as np
import pytest

from fieldcraft_b200 import problems as P
from fieldcraft_b200.unet import UNet

pytestmark = pytest.mark.gpu


def network(dims, levels, odd):
    nx, ny, nz = dims
    p = P.plate(nx, ny, nz, corr=3.0)
    net = UNet(p, seed=3, levels=levels)
    net.set_odd(odd)
    flat = net.params()
    rng = np.random.default_rng(1)
    last = 27 * 32 * 16 + 16
    flat[-last:] = (0.05 * rng.standard_normal(last)).astype(np.float32)
    net.set_params(flat)
    return p, net, flat


@pytest.mark.parametrize("dims,levels,odd", [((7, 7, 1), 2, True), ((15, 8, 3), 3, True), ((16, 9, 2), 3, False),
                                             ((23, 17, 4), 4, True), ((48, 31, 7), 3, True)])
@pytest.mark.parametrize("count", [1, 3, 8, 11])
def test_batches_are_their_pairs(cuda, dims, levels, odd, count):
    torch = cuda
    p, net, flat = network(dims, levels, odd)
    g = torch.Generator(device="cuda").manual_seed(count)
    r = torch.randn((count, p.n), dtype=torch.float64, device="cuda", generator=g)
    e = torch.randn((count, p.n), dtype=torch.float64, device="cuda", generator=g)
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    total, last, mean = 0.0, None, np.zeros(flat.size)
    for q in range(count):
        net.set_params(flat)
        net.train_step(r[q], e[q], 1e-3, 1, loss=loss)
        last = net.grads()
        mean += last.astype(np.float64) / count
        total += float(loss[0])
    net.close()
    _, net, _ = network(dims, levels, odd)
    net.train_batch(r, e, 1e-3, 1, loss=loss)
    assert abs(float(loss[0]) - total) <= 1e-12 * abs(total)
    got = net.grads()
    scale = np.max(np.abs(last))
    assert np.max(np.abs(got - last)) <= 2e-5 * scale
    # the first Adam step from zero moments moves a weight by lr g / (|g| + 1e-8), g its mean gradient:
    # an error d of g moves that by at most lr d / 1e-8 (and by at most 2 lr), and the stored weight rounds
    moved = flat.astype(np.float64) - net.params()
    want = 1e-3 * mean / (np.abs(mean) + 1e-8)
    slack = min(2e-3, 1e-3 * 2e-5 * max(scale, np.max(np.abs(mean))) / 1e-8)
    assert np.max(np.abs(moved - want)) <= slack + 1e-3 * 1e-5 + 1.2e-7 * np.max(np.abs(flat))
    net.close()
