"""Minibatches where memory is short, and captured graphs beside them: batches in the handle's own room
for one pass or two and in larger rooms for fewer pairs than they have give the losses and gradients of
the batch in one group (the losses to FP64 rounding; the gradients' FP32 sums in other chunks, as
test_gpu_unet_batch.py bounds them), the network runs after every refusal, and a graph captured before a
batch made its larger room replays the same bits after it."""
import ctypes as C

import numpy as np
import pytest

from fieldcraft_b200 import _lib
from test_gpu_unet_batch import network

pytestmark = pytest.mark.gpu


def room(net, own, group):
    assert _lib.load().fc_test_unet_room(net.handle, own, group) == own


def pairs(torch, n, count):
    g = torch.Generator(device="cuda").manual_seed(count)
    return [torch.randn((count, n), dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]


@pytest.mark.parametrize("odd", [True, False], ids=["odd", "plain"])
@pytest.mark.parametrize("own,group", [(1, 0), (1, 2), (1, 6), (2, 0), (2, 4), (2, 10)])
@pytest.mark.parametrize("count", [1, 3, 8, 11])
def test_batches_in_less_room(cuda, odd, own, group, count):
    torch = cuda
    p, net, flat = network((15, 8, 3), 3, odd)
    r, e = pairs(torch, p.n, count)
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    found = []
    for limited in (False, True):
        if limited:
            room(net, own, group)
        net.set_params(flat)
        z = torch.empty_like(r[0])
        net.apply(r[0], z)
        net.train_batch(r, e, 1e-3, 1, loss=loss)
        grads = net.grads()
        x = torch.randn(16 * (p.eq.size // 3), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
        y = torch.empty_like(x)
        net.set_params(flat)
        net.forward_grid(x, y)
        net.backward_grid(x)
        found.append((float(loss[0]), grads, z.cpu().numpy(), y.cpu().numpy(), net.grads()))
    (loss0, grads0, z0, y0, b0), (loss1, grads1, z1, y1, b1) = found
    assert abs(loss1 - loss0) <= 1e-12 * abs(loss0)
    assert np.max(np.abs(grads1 - grads0)) <= 2e-5 * np.max(np.abs(grads0))
    assert np.max(np.abs(z1 - z0)) <= 1e-15 * np.max(np.abs(z0))  # the two passes added one by one
    assert np.array_equal(y1, y0) and np.array_equal(b1, b0)
    net.close()


def test_a_graph_outlives_a_larger_room(cuda):
    torch = cuda
    p, net, flat = network((23, 17, 4), 3, True)
    r, e = pairs(torch, p.n, 8)
    z, want = torch.empty_like(r[0]), torch.empty_like(r[0])
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    net.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    applied, trained = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    net.set_params(flat)  # the graphs start from the FP32 weights
    with torch.cuda.graph(applied, stream=stream):
        net.apply(r[0], z)
    net.set_params(flat)
    with torch.cuda.graph(trained, stream=stream):
        net.train_batch(r, e, 1e-3, 1, loss=loss)  # the handle's first batch

    def replay():
        net.set_params(flat)
        with torch.cuda.stream(stream):
            applied.replay()
            trained.replay()
        torch.cuda.synchronize()
        return z.clone(), loss.clone(), net.grads()

    before = replay()
    fresh = network((23, 17, 4), 3, True)[1]
    fresh.apply(r[0], want)
    fresh.train_batch(r, e, 1e-3, 1, loss=loss)
    torch.cuda.synchronize()
    assert torch.equal(before[0], want)
    assert abs(float(before[1][0]) - float(loss[0])) <= 1e-12 * abs(float(loss[0]))
    assert np.max(np.abs(before[2] - fresh.grads())) <= 2e-5 * np.max(np.abs(before[2]))
    for count in (3, 8):
        net.train_batch(r[:count], e[:count], 1e-3, 1)
    torch.cuda.synchronize()
    filler = torch.full((64 << 20,), 1e30, device="cuda")  # over whatever a larger room gave back
    after = replay()
    assert torch.equal(after[0], before[0]) and torch.equal(after[1], before[1]) and np.array_equal(after[2], before[2])
    del filler
    net.close()
    fresh.close()
