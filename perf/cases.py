"""The work that users of this library have it do, as cases to time and to check: single solves
from host and device memory, refactorisation with new moduli on a kept analysis, solves on a kept
factor, many small systems at once, the mixed-precision and the indefinite factor, assembly and
stress recovery around the solve, and the learned preconditioner's passes and flexible CG.

`listed()` are the cases by name, `draw` more of the same ranges, `prepare` what a program holds
before the call (inputs on the GPU, analysis, handle), `run` one pass through the public entry
points, `work` the bytes and operations a pass cannot do without, `tolerance` how far another
correct implementation's outputs may be, `exact` the outputs in 64 bits or better by plain numpy
and torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch
import torch.nn.functional as F

from fieldcraft_b200 import FP32_IR, FP64, LDLT, Csr, Factor, LdltFactor, Symbolic, _lib
from fieldcraft_b200 import problems as P
from fieldcraft_b200.cholesky import Status, raise_for
from fieldcraft_b200.unet import UNet, fcg

NO_LIMIT = 2 ** 62
POISSON = 0.3


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # one small part solved from a host program's own arrays (the Rust caller's path)
        dict(name="cantilever-host", kind="host", nx=40, ny=4, nz=4, held="x", field="uniform", nrhs=1),
        # a design loop on a small part: new moduli, a few load cases, the product K x for the check
        dict(name="part-refactor", kind="direct", count=1, nx=23, ny=17, nz=19, held="z", field="iid", nrhs=7),
        # the benchmark's block: factorisation and 64 load cases at full size
        dict(name="block-64loads", kind="direct", count=1, nx=48, ny=48, nz=48, held="z", field="iid", nrhs=64),
        # many small uneven parts at once, eight load cases each
        dict(name="uneven-batch", kind="direct", count=40, nx=16, ny=16, nz=16, held="z", field="uniform", nrhs=8),
        # mixed precision: FP32 factor and FP64 refinement to 1e-10 on an uneven random medium
        dict(name="mixed-medium", kind="mixed", count=1, nx=40, ny=36, nz=33, held="z", field="smooth", nrhs=16),
        # a time step or an inverse iteration: one solve on a kept factor
        dict(name="plate-one-solve", kind="solve", count=1, nx=64, ny=64, nz=8, held="sides", field="smooth", nrhs=1),
        # many load cases on a kept factor
        dict(name="many-loads-solve", kind="solve", count=1, nx=29, ny=26, nz=24, held="z", field="iid", nrhs=48),
        # shift-invert on an indefinite K - sigma I: LDL^T and a block of four vectors
        dict(name="indefinite-shift", kind="ldlt", nx=16, ny=14, nz=13, held="z", field="iid", nrhs=4),
        # what surrounds the solve: K from the moduli, reactions and stresses from the solution
        dict(name="assemble-stress", kind="fem", nx=48, ny=40, nz=36, held="z", field="iid"),
        # the learned preconditioner: one Adam step on a minibatch, and one application
        dict(name="unet-train-batch", kind="train", nx=32, ny=32, nz=8, held="sides", field="smooth", levels=3, pairs=8),
        dict(name="unet-apply", kind="apply", nx=64, ny=64, nz=8, held="sides", field="smooth", levels=4),
        # flexible CG on its block-Jacobi part to 1e-10
        dict(name="plate-fcg", kind="fcg", nx=48, ny=48, nz=8, held="sides", field="smooth"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box_dims(rng, lo, hi, most=64):
    """Three uneven element counts whose product is about log-uniform in [lo, hi]."""
    n = _log_uniform(rng, lo, hi)
    e = [rng.uniform(-0.3, 0.3) for _ in range(3)]
    mean = sum(e) / 3
    return [max(2, min(most, round(n ** (1 / 3) * math.exp(v - mean)))) for v in e]


def _plate_dims(rng, lo, hi):
    nz = rng.randint(2, 9)
    nx = max(6, round(_log_uniform(rng, lo, hi)))
    return [nx, max(6, round(nx * rng.uniform(0.6, 1.0))), nz]


def draw(rng):
    kind = rng.choice(["host", "direct", "direct", "batch", "mixed", "solve", "solve", "ldlt", "fem", "train", "apply",
                       "fcg"])
    field = rng.choice(["iid", "smooth", "uniform"])
    nrhs = round(_log_uniform(rng, 1, 64))
    if kind == "host":
        nx, ny, nz = _box_dims(rng, 300, 6000)
        return dict(kind="host", nx=nx, ny=ny, nz=nz, held="x", field=field, nrhs=min(nrhs, 8))
    if kind == "batch":
        n = rng.randint(5, 16)
        return dict(kind="direct", count=rng.randint(5, 40), nx=n, ny=max(4, n - rng.randint(0, 3)), nz=n, held="z",
                    field="uniform", nrhs=min(nrhs, 16))
    if kind in ("direct", "mixed", "solve"):
        if rng.random() < 0.4:
            (nx, ny, nz), held = _plate_dims(rng, 12, 64), "sides"
        else:
            (nx, ny, nz), held = _box_dims(rng, 400, 50000, 44), "z"
        return dict(kind=kind, count=1, nx=nx, ny=ny, nz=nz, held=held, field=field, nrhs=nrhs)
    if kind == "ldlt":
        nx, ny, nz = _box_dims(rng, 200, 3000)
        return dict(kind="ldlt", nx=nx, ny=ny, nz=nz, held="z", field="iid", nrhs=min(nrhs, 16))
    if kind == "fem":
        nx, ny, nz = _box_dims(rng, 1000, 80000)
        return dict(kind="fem", nx=nx, ny=ny, nz=nz, held=rng.choice(["x", "z"]), field=field)
    nx, ny, nz = _plate_dims(rng, 12, 64 if kind == "apply" else 40)
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, held="sides", field="smooth")
    if kind != "fcg":
        case["levels"] = rng.randint(2, 4)
    if kind == "train":
        case["pairs"] = rng.randint(1, 8)
    return case


# ---- inputs ------------------------------------------------------------------------------------

def _moduli(field, dims, rng):
    """Young's modulus of each element (e = i + nx (j + ny k)): one value, iid lognormal (sigma
    0.5), or a smooth lognormal field spanning two decades at three sigma."""
    nx, ny, nz = dims
    if field == "uniform":
        return np.full(nx * ny * nz, float(rng.uniform(70000.0, 210000.0)))
    if field == "iid":
        return 210000.0 * np.exp(0.5 * rng.standard_normal(nx * ny * nz))
    g = P.gaussian_field((nz, ny, nx), 4.0, int(rng.integers(1 << 31)))
    return 210000.0 * np.exp(math.log(100.0) / 6.0 * g).reshape(-1)


def _held(case, dims):
    i, j, k = P.node_grid(*dims)
    if case["held"] == "x":
        return i == 0
    if case["held"] == "z":
        return k == 0
    return (i == 0) | (i == dims[0]) | (j == 0) | (j == dims[1])


def _problem(case, dims, rng):
    nx, ny, nz = dims
    young = _moduli(case["field"], dims, rng)
    p = P.box(nx, ny, nz, float(nx), float(ny), float(nz), young, POISSON, _held(case, dims))
    p.young = young
    return p


def _loads(p, nrhs, rng):
    """Gaussian forces on every node of the top face, a row per load case."""
    _, _, k = P.node_grid(*p.dims)
    e = p.eq.reshape(-1, 3)[k == p.dims[2]].reshape(-1)
    e = e[e >= 0]
    f = np.zeros((nrhs, p.n))
    f[:, e] = rng.standard_normal((nrhs, e.size))
    return f


def _systems(case, seed):
    """The case's systems and their loads. A batch's parts shrink from the named size by the
    seed-free rule below, so every seed has the same shapes and other values."""
    rng = np.random.default_rng(seed)
    out = []
    for b in range(case.get("count", 1)):
        dims = (case["nx"], case["ny"], case["nz"])
        if case.get("count", 1) > 1:
            dims = tuple(max(2, d - (b * q) % max(1, d - 3)) for d, q in zip(dims, (5, 7, 3)))
        p = _problem(case, dims, rng)
        out.append((p, _loads(p, case["nrhs"], rng)))
    return out


def _stack(systems):
    """The systems' rows as one block-diagonal matrix, and the loads side by side."""
    ptr, idx, val, at, nz = [np.zeros(1, np.int64)], [], [], 0, 0
    for p, _ in systems:
        ptr.append(p.csr.ptr[1:] + nz)
        idx.append(p.csr.idx.astype(np.int64) + at)
        val.append(p.csr.val)
        at, nz = at + p.n, nz + int(p.csr.ptr[-1])
    csr = Csr(at, np.concatenate(ptr), np.concatenate(idx).astype(np.int32), np.concatenate(val))
    return csr, np.concatenate([f for _, f in systems], axis=1)


def _shifted(p):
    """K - sigma I with sigma 2 % of the mean diagonal: a few dozen negative eigenvalues."""
    rows = np.repeat(np.arange(p.n), np.diff(p.csr.ptr))
    on = p.csr.idx == rows
    val = p.csr.val.copy()
    val[on] -= 0.02 * val[on].mean()
    return Csr(p.n, p.csr.ptr, p.csr.idx, val)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _csr_cuda(csr):
    return _cuda(csr.ptr), _cuda(csr.idx), _cuda(csr.val)


def _analysis(systems):
    parts = [p.upper() for p, _ in systems]
    if len(parts) == 1:
        return Symbolic(parts[0], NO_LIMIT), parts[0].val
    return Symbolic.batch(parts, NO_LIMIT)[0], np.concatenate([u.val for u in parts])


def _network(case, p, seed, operator):
    """A network whose every layer is live, the state any training leaves (a fresh one's last
    layer is zero)."""
    net = UNet(p, seed=1, kref=1e5, levels=case["levels"], operator=operator)
    flat = net.params()
    rng = np.random.default_rng(seed + 77)
    last = 27 * 32 * 16 + 16
    flat[-last:-16] = (rng.standard_normal(last - 16) * math.sqrt(1.0 / (27 * 32))).astype(np.float32)
    flat[-16:] = 0.01
    net.set_params(flat)
    return net, flat


def _unit_rows(a):
    return a / np.linalg.norm(a, axis=1, keepdims=True)


def prepare(case, seed):
    kind = case["kind"]
    dims = (case["nx"], case["ny"], case["nz"])
    s = {"kind": kind, "stream": torch.cuda.Stream()}
    stream = s["stream"].cuda_stream
    if kind == "host":
        (p, f), = _systems(case, seed)
        s["val"] = p.upper().val
        s["b"] = np.asfortranarray(f.T)
        s["factor"] = Factor(Symbolic(p.upper(), NO_LIMIT), FP64)
    elif kind in ("direct", "mixed", "solve"):
        systems = _systems(case, seed)
        sym, val = _analysis(systems)
        csr, f = _stack(systems)
        s["factor"] = Factor(sym, FP32_IR if kind == "mixed" else FP64)
        s["factor"].set_stream(stream)
        s["val"], s["b"], s["R"], s["n"] = _cuda(val), _cuda(f), case["nrhs"], csr.n
        s["x"] = torch.empty_like(s["b"])
        if kind != "solve":
            s["csr"] = _csr_cuda(csr)
        if kind == "direct":
            s["y"] = torch.empty_like(s["b"])
        if kind == "solve":
            torch.cuda.synchronize()
            _factor_device(s)
    elif kind == "ldlt":
        rng = np.random.default_rng(seed)
        p = _problem(case, dims, rng)
        f = _loads(p, case["nrhs"], rng)
        upper = P.UpperColumns.from_symmetric(_shifted(p))
        s["factor"] = LdltFactor(Symbolic(upper, NO_LIMIT))
        s["factor"].set_stream(stream)
        s["val"], s["b"], s["R"], s["n"] = _cuda(upper.val), _cuda(f), case["nrhs"], p.n
        s["x"] = torch.empty_like(s["b"])
    elif kind == "fem":
        rng = np.random.default_rng(seed)
        p = _problem(case, dims, rng)
        s["assembly"] = P.DeviceAssembly(p)
        s["young"], s["q"] = _cuda(p.young), _cuda(1e-3 * rng.standard_normal(p.n))
        s["val"] = torch.empty(p.csr.val.size, dtype=torch.float64, device="cuda")
        s["r"] = torch.empty(p.eq.size, dtype=torch.float64, device="cuda")
        s["u"] = torch.empty_like(s["r"])
        s["points"] = torch.empty(48 * p.young.size, dtype=torch.float64, device="cuda")
        s["nodal"] = torch.empty(2 * p.eq.size, dtype=torch.float64, device="cuda")
        s["mises"] = torch.empty(p.eq.size // 3, dtype=torch.float64, device="cuda")
    else:
        rng = np.random.default_rng(seed)
        p = _problem(case, dims, rng)
        s["csr"], s["n"] = _csr_cuda(p.csr), p.n
        if kind == "fcg":
            s["net"] = UNet(p, seed=1, kref=1e5, levels=2, operator=s["csr"])
            s["net"].enable(False)
            s["b"] = _cuda(_unit_rows(_loads(p, 1, rng))[0])
            s["x"] = torch.empty_like(s["b"])
        else:
            s["net"], s["params"] = _network(case, p, seed, s["csr"])
            r = _unit_rows(rng.standard_normal((case.get("pairs", 1), p.n)))
            s["r"] = _cuda(r)
            if kind == "apply":
                s["z"] = torch.empty_like(s["r"][0])
            else:
                f = Factor(Symbolic(p.upper(), NO_LIMIT), FP64)
                f.factor(p.upper().val)
                e = np.asfortranarray(r.T.copy())
                f.solve_many(e)
                f.close()
                s["e"], s["step"] = _cuda(e.T), 0
                s["loss"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["net"].set_stream(stream)
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------------------

def _factor_device(s):
    st = Status()
    _lib.load().fc_chol_factor_device(s["factor"].handle, C.c_void_p(s["val"].data_ptr()), s["val"].numel(), C.byref(st))
    raise_for(st)


def run(s):
    kind = s["kind"]
    if kind == "host":
        s["factor"].factor(s["val"])
        x = s["b"].copy(order="F")
        s["factor"].solve_many(x)
        return {"x": x.T}
    with torch.cuda.stream(s["stream"]):
        stream = s["stream"].cuda_stream
        if kind in ("direct", "solve", "ldlt"):
            if kind != "solve":
                _factor_device(s)
            s["x"].copy_(s["b"])
            s["factor"].solve_device(s["x"], s["R"], s["n"])
            if kind != "direct":
                return {"x": s["x"]}
            ptr, idx, val = s["csr"]
            _lib.load().fc_csr_spmv_device(s["n"], _lib.ptr(ptr), _lib.ptr(idx), _lib.ptr(val), _lib.ptr(s["x"]),
                                           _lib.ptr(s["y"]), s["R"], s["n"], stream)
            return {"x": s["x"], "Kx": s["y"]}
        if kind == "mixed":
            _factor_device(s)
            s["factor"].refine_solve_device(s["csr"], s["b"], s["x"], s["R"], s["n"], tol=1e-10, max_iter=40)
            return {"x": s["x"]}
        if kind == "fem":
            a = s["assembly"]
            a.assemble(s["young"], s["val"], POISSON, stream)
            a.reactions(s["q"], r=s["r"], u=s["u"], stream_ptr=stream)
            a.stresses(s["young"], s["u"], s["points"], s["nodal"], s["mises"], POISSON, stream)
            return {k: s[k] for k in ("val", "r", "u", "points", "nodal", "mises")}
        if kind == "fcg":
            fcg(s["csr"], s["b"], s["x"], net=s["net"], tol=1e-10, max_iter=4000, keep=4)
            return {"x": s["x"]}
        if kind == "apply":
            s["net"].apply(s["r"][0], s["z"])
            return {"z": s["z"]}
        s["step"] += 1
        s["net"].train_batch(s["r"], s["e"], 3e-4, s["step"], loss=s["loss"], csr_device=s["csr"])
        # the last pair's gradient and the updated weights, as a training loop logs and saves them
        return {"loss": s["loss"], "grads": s["net"].grads(), "params": s["net"].params()}


# ---- what a pass cannot do without --------------------------------------------------------------

def _conv_flops(case):
    x, y, z = case["nx"] + 1, case["ny"] + 1, case["nz"] + 1
    total, params, first = 0.0, 0, 0.0
    for lv in range(case["levels"]):
        v = x * y * z
        layers = [(16, 32), (32, 32)] if lv == 0 else [(32, 32)] * 2
        if lv < case["levels"] - 1:
            layers += [(32, 32)] * 2
        if lv == 0:
            layers.append((32, 16))
            first = 2.0 * 27 * 16 * 32 * v
        total += sum(2.0 * 27 * a * b * v for a, b in layers)
        params += sum(27 * a * b + b for a, b in layers)
        x, y, z = (x + 1) // 2, (y + 1) // 2, (z + 1) // 2
    return total, first, params


def work(case):
    kind = case["kind"]
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if kind in ("train", "apply"):
        flops, first, params = _conv_flops(case)
        pairs = case.get("pairs", 1)
        if kind == "apply":  # the odd form: a pass on r and one on -r
            return {"bytes": 2.0 * params + 48.0 * nodes, "flops": 2 * flops}
        return {"bytes": 16.0 * params + 48.0 * nodes * pairs, "flops": 2.0 * pairs * (3 * flops - first)}
    if kind == "fem":
        elements = case["nx"] * case["ny"] * case["nz"]
        nnz = 9 * (3 * case["nx"] + 1) * (3 * case["ny"] + 1) * (3 * case["nz"] + 1)
        return {"bytes": 8.0 * (nnz + 49 * elements + 16 * nodes), "flops": 2.0 * 81 * 8 * 8 * elements}
    systems = _systems(case, 0) if kind in ("host", "direct", "mixed", "solve") else \
        [(_problem(case, (case["nx"], case["ny"], case["nz"]), np.random.default_rng(0)), None)]
    n = sum(p.n for p, _ in systems)
    nnz = sum(int(p.csr.ptr[-1]) for p, _ in systems)
    if kind == "fcg":  # each input once: how many iterations it takes is the method's own
        return {"bytes": 12.0 * nnz + 16.0 * n, "flops": 2.0 * nnz}
    a = _analysis(systems)[0].arrays()
    m, w = np.diff(a["rptr"]).astype(np.float64), np.diff(a["first"]).astype(np.float64)
    # sum over a supernode's columns of (m - c)^2, c = 0 .. w - 1
    factor = float(np.sum(w * m * m - m * w * (w - 1) + (w - 1) * w * (2 * w - 1) / 6))
    entries, nrhs, es = float(a["entries"]), case["nrhs"], 4 if kind == "mixed" else 8
    vectors, solve = 16.0 * n * nrhs, 4.0 * entries * nrhs
    if kind == "solve":
        return {"bytes": 8 * entries + vectors, "flops": solve}
    upper = (nnz + n) / 2
    out = {"bytes": 8 * upper + es * entries + vectors, "flops": factor + solve}
    if kind == "direct":
        out["bytes"] += 12.0 * nnz + 8.0 * n * nrhs
        out["flops"] += 2.0 * nnz * nrhs
    if kind == "mixed":
        out["bytes"] += 12.0 * nnz
    return out


def tolerance(case):
    kind = case["kind"]
    # FP64 rounding through another elimination order: 5e-15 to 4e-14 off 80 bits on blocks, 3e-12
    # on a slender part
    if kind == "host":
        return {"rel": 2e-11, "max": 1e-10}
    if kind in ("direct", "solve"):
        return {"rel": 2e-12, "max": 1e-10}
    if kind == "ldlt":  # near an eigenvalue the shifted matrix is worse conditioned
        return {"rel": 1e-10, "max": 1e-8}
    # both stop at a relative residual of 1e-10 and leave an error of about 2e-10
    if kind in ("mixed", "fcg"):
        return {"rel": 2e-9, "max": 1e-7}
    if kind == "fem":
        return {"rel": 2e-14, "max": 1e-12}
    return {"rel": 2e-2, "max": 0.5}  # BF16 activations through 7 to 15 convolutions


# ---- the same in 64 bits or better --------------------------------------------------------------

def _sharpened(csr, f, solve, rounds=3):
    """Rows of x with A x = f: `solve`, then its corrections of the residual in 80 bits."""
    starts = csr.ptr[:-1]
    val = csr.val.astype(np.longdouble)
    x = np.zeros(f.shape, np.longdouble)
    for _ in range(rounds):
        r = np.empty_like(f)
        for j in range(f.shape[0]):
            r[j] = f[j] - np.add.reduceat(val * x[j][csr.idx], starts)
        x += solve(r)
    return x.astype(np.float64)


def _dense(csr, f):
    a = torch.zeros((csr.n, csr.n), dtype=torch.float64, device="cuda")
    rows = torch.repeat_interleave(torch.arange(csr.n, device="cuda"), _cuda(np.diff(csr.ptr)))
    a[rows, _cuda(csr.idx).long()] = _cuda(csr.val)
    lu = torch.linalg.lu_factor(a)
    del a
    return _sharpened(csr, f, lambda r: torch.linalg.lu_solve(*lu, _cuda(r.T)).T.cpu().numpy())


def _iterated(csr, f):
    """Conjugate gradients preconditioned by the diagonal, each right-hand side's own recurrence."""
    a = torch.sparse_csr_tensor(_cuda(csr.ptr), _cuda(csr.idx).long(), _cuda(csr.val), (csr.n, csr.n))
    rows = np.repeat(np.arange(csr.n), np.diff(csr.ptr))
    inv = _cuda(1.0 / csr.val[csr.idx == rows])[:, None]

    def solve(r_rows):
        r = _cuda(r_rows.T)
        x, stop = torch.zeros_like(r), 1e-9 * torch.linalg.vector_norm(r, dim=0)
        z = inv * r
        p, rz = z.clone(), (r * z).sum(0)
        for it in range(20000):
            q = a @ p
            alpha = torch.nan_to_num(rz / (p * q).sum(0))
            x += alpha * p
            r -= alpha * q
            if it % 25 == 24 and bool((torch.linalg.vector_norm(r, dim=0) <= stop).all()):
                break
            z = inv * r
            new = (r * z).sum(0)
            p = z + torch.nan_to_num(new / rz) * p
            rz = new
        return x.T.cpu().numpy()

    return _sharpened(csr, f, solve, rounds=4)


def _unit_element(nu):
    """The hex8 unit cube's stiffness at unit modulus, its stress matrices at the Gauss points, and
    the extrapolation from the points to the corners."""
    corners = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                        [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], np.float64)
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    d = np.diag([2 * mu] * 3 + [mu] * 3)
    d[:3, :3] += lam
    g = 1 / math.sqrt(3.0)
    k, stress, at = np.zeros((24, 24)), [], []
    for pz in (-g, g):
        for py in (-g, g):
            for px in (-g, g):
                t = 1 + corners * np.array([px, py, pz])
                dn = np.stack([corners[:, 0] * t[:, 1] * t[:, 2], corners[:, 1] * t[:, 0] * t[:, 2],
                               corners[:, 2] * t[:, 0] * t[:, 1]], axis=1) / 8 * 2  # dx = dxi / 2
                b = np.zeros((6, 24))
                for row, col, axis in ((0, 0, 0), (1, 1, 1), (2, 2, 2), (3, 0, 1), (3, 1, 0), (4, 0, 2), (4, 2, 0),
                                       (5, 1, 2), (5, 2, 1)):
                    b[row, col::3] += dn[:, axis]
                k += b.T @ d @ b / 8
                stress.append(d @ b)
                at.append(np.sign([px, py, pz]))
    # the trilinear functions of the points' own box, in the order the recovery pairs them with the
    # points: the corners' order
    w = np.prod(1 + math.sqrt(3.0) * corners[:, None, :] * corners[None, :, :], axis=2) / 8
    return k, np.array(stress), w


def _fem_exact(case, seed):
    dims = nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    p = _problem(case, dims, rng)
    q = 1e-3 * rng.standard_normal(p.n)
    ke, stress, w = _unit_element(POISSON)
    e = np.arange(nx * ny * nz)
    i, j, k = e % nx, e // nx % ny, e // (nx * ny)
    offs = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    nodes = np.stack([(i + a) + (nx + 1) * ((j + b) + (ny + 1) * (k + c)) for a, b, c in offs], axis=1)
    u = np.where(p.eq >= 0, q[np.maximum(p.eq, 0)], 0.0)
    dofs = (3 * nodes[:, :, None] + np.arange(3)).reshape(-1, 24)
    eq = p.eq[dofs]
    val = np.zeros(p.csr.val.size)
    key = np.repeat(np.arange(p.n), np.diff(p.csr.ptr)) * np.int64(p.n) + p.csr.idx
    for a in range(24):
        for b in range(24):
            on = (eq[:, a] >= 0) & (eq[:, b] >= 0)
            val += np.bincount(np.searchsorted(key, eq[on, a] * np.int64(p.n) + eq[on, b]), p.young[on] * ke[a, b],
                               minlength=val.size)
    ue = u[dofs]
    r = np.bincount(dofs.reshape(-1), (p.young[:, None] * (ue @ ke)).reshape(-1), minlength=u.size)
    r[p.eq >= 0] = 0.0
    points = p.young[:, None, None] * np.einsum("psd,ed->eps", stress, ue)
    corner = np.einsum("np,eps->ens", w, points)
    count = np.bincount(nodes.reshape(-1))
    nodal = np.stack([np.bincount(nodes.reshape(-1), corner[:, :, s].reshape(-1)) / count for s in range(6)], axis=1)
    x, y, z, xy, xz, yz = nodal.T
    mises = np.sqrt(0.5 * ((x - y) ** 2 + (y - z) ** 2 + (z - x) ** 2) + 3 * (xy ** 2 + xz ** 2 + yz ** 2))
    return {"val": val, "r": r, "u": u, "points": points.reshape(-1), "nodal": nodal.reshape(-1), "mises": mises}


def _net64(flat, levels, x):
    """The network on x [1, 16, Z, Y, X] in 64 bits."""
    at = 0

    def conv(x, cin, cout, relu=True):
        nonlocal at
        weight = flat[at:at + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        bias = flat[at + 27 * cin * cout:at + 27 * cin * cout + cout]
        at += 27 * cin * cout + cout
        x = F.conv3d(x, weight, bias, padding=1)
        return F.leaky_relu(x, 0.05) if relu else x

    skips = []
    for lv in range(levels):
        x = conv(conv(x, 16 if lv == 0 else 32, 32), 32, 32)
        if lv < levels - 1:
            skips.append(x)
            odd = [v % 2 for v in x.shape[:1:-1]]
            x = F.avg_pool3d(F.pad(x, (0, odd[0], 0, odd[1], 0, odd[2])), 2)
    for skip in reversed(skips):
        for axis in (2, 3, 4):
            x = x.repeat_interleave(2, axis).narrow(axis, 0, skip.shape[axis])
        x = conv(conv(x + skip, 32, 32), 32, 32)
    return conv(x, 32, 16, relu=False)


def _unet_exact(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    s = prepare(case, seed)
    rng = np.random.default_rng(seed)
    p = _problem(case, dims, rng)
    grid = [d + 1 for d in dims][::-1]
    free = _cuda(p.eq >= 0)
    eq = _cuda(np.maximum(p.eq, 0))
    feat = _cuda(P.node_feature(p)).double()
    rows = np.repeat(np.arange(p.n), np.diff(p.csr.ptr))
    same = p.csr.idx // 3 == rows // 3
    blocks = np.zeros((p.n // 3, 3, 3))
    blocks[rows[same] // 3, rows[same] % 3, p.csr.idx[same] % 3] = p.csr.val[same]
    jacobi = _cuda(np.linalg.inv(blocks))
    flat = _cuda(s["params"]).double().requires_grad_()
    k = torch.sparse_csr_tensor(_cuda(p.csr.ptr), _cuda(p.csr.idx).long(), _cuda(p.csr.val), (p.n, p.n))

    def one(r):
        norm = torch.linalg.vector_norm(r)
        x = torch.zeros((p.eq.size // 3, 16), dtype=torch.float64, device="cuda")
        x[:, :3] = torch.where(free, r[eq], 0.0).view(-1, 3) * (math.sqrt(p.n) / norm)
        x[:, 3] = feat
        y = _net64(flat, case["levels"], x.view(*grid, 16).permute(3, 0, 1, 2)[None])
        y = y[0].permute(1, 2, 3, 0).reshape(-1, 16)[:, :3].reshape(-1)
        out = torch.zeros_like(r)
        out[eq[free]] = y[free] * (norm / (math.sqrt(p.n) * 1e5))
        return out

    def apply(r):
        return torch.einsum("kab,kb->ka", jacobi, r.view(-1, 3)).reshape(-1) + 0.5 * (one(r) - one(-r))

    if case["kind"] == "apply":
        with torch.no_grad():
            return {"z": apply(s["r"][0])}
    total, mean = 0.0, torch.zeros_like(flat)
    for r, e in zip(s["r"], s["e"]):
        d = apply(r) - e
        loss = (d * (k @ d.detach())).sum()  # its gradient is half the quadratic form's
        grad, = torch.autograd.grad(2 * loss / (e * r).sum(), flat)
        total, mean = total + float(loss) / float((e * r).sum()), mean + grad / len(s["r"])
    # the first Adam step of zero moments moves each weight by lr g / (|g| + eps)
    moved = flat.detach() - 3e-4 * mean / (mean.abs() + 1e-8)
    return {"loss": torch.tensor([total], dtype=torch.float64), "grads": grad, "params": moved}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fem":
        return _fem_exact(case, seed)
    if kind in ("train", "apply"):
        return _unet_exact(case, seed)
    if kind == "ldlt":
        rng = np.random.default_rng(seed)
        p = _problem(case, (case["nx"], case["ny"], case["nz"]), rng)
        return {"x": _dense(_shifted(p), _loads(p, case["nrhs"], rng))}
    if kind == "fcg":
        rng = np.random.default_rng(seed)
        p = _problem(case, (case["nx"], case["ny"], case["nz"]), rng)
        return {"x": _iterated(p.csr, _unit_rows(_loads(p, 1, rng)))[0]}
    csr, f = _stack(_systems(case, seed))
    if csr.idx.size * case["nrhs"] > 3e8:
        return None
    x = _dense(csr, f) if csr.n <= 12000 else _iterated(csr, f)
    return {"x": x, "Kx": f} if kind == "direct" else {"x": x}
