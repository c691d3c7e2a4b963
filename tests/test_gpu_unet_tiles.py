"""The convolutions' tiles against the CPU oracle's network: grids of one tile and of several, with
sides at and past a tile's largest, single voxels across, and more tiles than the GPU takes at once.

BF16 keeps 8 bits and the sums differ in order, which moves some roundings of an activation by one
unit: outputs agree to 2e-2 of their largest entry through the five convolutions of two levels."""
import numpy as np
import pytest

from fieldcraft_b200 import problems as P
from fieldcraft_b200.unet import UNet
from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 2, 1), (10, 10, 2), (23, 23, 1), (24, 3, 2), (47, 2, 15), (5, 4, 17), (48, 24, 9),
                                  (90, 77, 6)])
def test_forward_on_every_kind_of_tile(cuda, dims):
    torch = cuda
    nx, ny, nz = dims
    net = UNet(P.plate(nx, ny, nz, corr=3.0), seed=1, levels=2)
    flat = U.init_params(2, 2)
    net.set_params(flat)
    x = np.random.default_rng(4).standard_normal((nz + 1, ny + 1, nx + 1, U.CIO)).astype(np.float32)
    dx = torch.from_numpy(x.reshape(-1)).cuda()
    y = torch.empty_like(dx)
    net.forward_grid(dx, y)
    want = U.Net(flat.astype(np.float64), use_bf16=True, levels=2).forward(x.astype(np.float64))
    assert np.max(np.abs(y.cpu().numpy().reshape(want.shape) - want)) <= 2e-2 * np.max(np.abs(want))
    net.close()
