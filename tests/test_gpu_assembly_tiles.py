"""The device assembly and stress recovery at the edges of their tiles (six elements a block for the
element matrices, sixteen for the stresses, a warp a row or a held DOF): K, the reactions and the
stresses bit for bit the host's, for boxes of one element up to a few past a tile, thin boxes whose
axes are one element (two planes of nodes), and moduli so large that products overflow, where the
host's zeros times infinity must come out as its NaNs do."""
import numpy as np
import pytest

from fieldcraft_b200 import problems
from test_device_assembly import host_reactions, host_stresses

pytestmark = pytest.mark.gpu


def same(got, want):
    got, want = got.cpu().numpy(), np.asarray(want).reshape(-1)
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


@pytest.mark.parametrize("dims,scale", [((1, 1, 1), 1.0), ((5, 1, 1), 1.0), ((3, 2, 1), 1.0), ((7, 1, 1), 1.0),
                                        ((1, 4, 4), 1.0), ((17, 1, 1), 1.0), ((4, 3, 3), 1.0), ((3, 2, 2), 1e303)])
def test_tiles_are_the_hosts(cuda, dims, scale):
    torch = cuda
    nx, ny, nz = dims
    lengths = tuple(0.01 * d for d in dims)
    rng = np.random.default_rng(nx + 10 * ny)
    young = 2e5 * scale * np.exp(0.3 * rng.standard_normal(nx * ny * nz))
    p = problems.box(nx, ny, nz, *lengths, young, 0.3, problems.node_grid(nx, ny, nz)[0] == 0)
    d = problems.DeviceAssembly(p)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    e = dev(young)
    val = torch.empty(p.csr.val.size, dtype=torch.float64, device="cuda")
    d.assemble(e, val)
    assert same(val, p.csr.val)
    q, f = rng.standard_normal(p.n), rng.standard_normal(p.eq.size)
    r = torch.empty(p.eq.size, dtype=torch.float64, device="cuda")
    u = torch.empty_like(r)
    d.reactions(dev(q), r=r, u=u, f=dev(f))
    assert same(r, host_reactions(nx, ny, nz, *lengths, p, young, q, f))
    points = torch.empty(48 * young.size, dtype=torch.float64, device="cuda")
    nodal = torch.empty(2 * p.eq.size, dtype=torch.float64, device="cuda")
    mises = torch.empty(p.eq.size // 3, dtype=torch.float64, device="cuda")
    d.stresses(e, u, points, nodal, mises)
    for got, want in zip((points, nodal, mises), host_stresses(nx, ny, nz, *lengths, young, u.cpu().numpy())):
        assert same(got, want)
    d.close()
