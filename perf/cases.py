"""The work that a user of this library has it do, as measurable cases.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program has in hand before the call, run() is one pass through the
public binding (cfm.py), work() the bytes and operations a pass cannot do
without, tolerance() how far another correct implementation may be, exact() the
result in 64 bits from plain torch.

Kinds of case:
  jacobi  Jacobi sweeps on a device-resident grid (cfm_jacobi_run)
  cg      conjugate gradients, CSR or matrix-free stencil (cfm_cg_solve_device)
  fpcg    flexible PCG on a 2D stencil, smoothed or with the network (cfm_fpcg_solve)
  batch   many uneven systems in one launch (cfm_batch_solve)
  unet    the network's gradient, forward and backward (cfm_unet_gradient_host)
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cpu-free-model_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import cfm  # noqa: E402

PRECISIONS = {"fp64": cfm.FP64, "fp32": cfm.FP32}
JACOBI_IMPLS = {"persistent": cfm.JACOBI_PERSISTENT, "resident": cfm.JACOBI_RESIDENT}
CG_IMPLS = {"standard": cfm.CG_PERSISTENT, "pipelined": cfm.CG_PERSISTENT_PIPELINED, "mixed": cfm.CG_MIXED}
MAXITER = 20000
SMOOTH = 4  # smoothing sweeps of the preconditioners


def _jacobi(dims, nx, ny, nz, precision, impl, niter, periodic_y=True, mirror=False):
    return {"kind": "jacobi", "dims": dims, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "impl": impl,
            "niter": niter, "periodic_y": periodic_y, "mirror": mirror}


def _cg(matrix, size, impl, tol=1e-8, maxiter=MAXITER):
    return {"kind": "cg", "matrix": matrix, "size": size, "impl": impl, "tol": tol, "maxiter": maxiter}


def _fpcg(ny, nx, net, precision):
    return {"kind": "fpcg", "ny": ny, "nx": nx, "net": net, "precision": precision, "tol": 1e-8}


def _batch(n2d, n3d, sizes, precision):
    return {"kind": "batch", "n2d": n2d, "n3d": n3d, "sizes": sizes, "precision": precision, "tol": 1e-8}


def _unet(height, width, batch):
    return {"kind": "unet", "height": height, "width": width, "batch": batch}


def listed():
    return [
        # the reference's smallest grid (its weak-scaling runs), where a sweep is all latency
        dict(_jacobi(2, 256, 256, 1, "fp32", "persistent", 1000), name="jacobi2d_256_fp32"),
        # the 2D benchmark: on-chip resident sweeps
        dict(_jacobi(2, 1024, 1024, 1, "fp64", "resident", 1000), name="jacobi2d_1024_fp64"),
        # the reference's largest 2D grid
        dict(_jacobi(2, 16384, 16384, 1, "fp32", "persistent", 50), name="jacobi2d_16384_fp32"),
        # the 3D benchmark (the headline figure)
        dict(_jacobi(3, 512, 512, 512, "fp64", "persistent", 100), name="jacobi3d_512_fp64"),
        # an odd 3D box whose rows are not a multiple of 16 bytes
        dict(_jacobi(3, 259, 253, 257, "fp32", "persistent", 100, periodic_y=False), name="jacobi3d_odd_fp32"),
        # the CG benchmark: 7-point Poisson matrix in CSR to 1e-8, FP32 iteration with FP64 updates
        dict(_cg("poisson", 128, "mixed"), name="cg_poisson128_mixed"),
        # the reference's random tridiagonal matrix, a fixed number of pipelined iterations
        dict(_cg("tridiag", 4194303, "pipelined", tol=0.0, maxiter=20), name="cg_tridiag_pipelined"),
        # matrix-free variable coefficients, plain FP64 CG to 1e-8: the plain solver users compare with
        dict(_cg("stencil2d", 512, "standard"), name="cg_stencil512"),
        # the same system with the smoothed flexible PCG, and with the network and FP32 vectors
        dict(_fpcg(512, 512, False, "fp64"), name="fpcg_smoothed_512"),
        dict(_fpcg(512, 512, True, "fp32"), name="fpcg_network_512_mixed"),
        # an uneven batch of 2D and 3D systems in one launch
        dict(_batch(24, 6, 1, "fp32"), name="batch_uneven_mixed"),
        # one training gradient of the network at its training shape
        dict(_unet(256, 256, 8), name="unet_gradient_256x8"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jacobi2d", "jacobi2d", "jacobi3d", "jacobi3d", "cg", "cg", "fpcg", "batch", "unet"])
    if kind == "jacobi2d":
        nx, ny = _log_int(rng, 64, 16384), _log_int(rng, 64, 16384)
        if rng.random() < 0.6:
            nx += -nx % 4  # most users' rows are a multiple of 16 bytes
        niter = max(3, min(rng.randint(20, 1000), int(2.0e9 / (nx * ny))))
        return _jacobi(2, nx, ny, 1, rng.choice(["fp32", "fp64"]), rng.choice(["persistent", "persistent", "resident"]),
                       niter, mirror=rng.random() < 0.2)
    if kind == "jacobi3d":
        nx, ny, nz = (_log_int(rng, 32, 512) for _ in range(3))
        if rng.random() < 0.6:
            nx += -nx % 4
        niter = max(3, min(rng.randint(10, 100), int(4.0e9 / (nx * ny * nz))))
        return _jacobi(3, nx, ny, nz, rng.choice(["fp32", "fp64"]), "persistent", niter, periodic_y=rng.random() < 0.5)
    if kind == "cg":
        matrix = rng.choice(["poisson", "tridiag", "stencil2d", "stencil3d", "csr2d"])
        impl = rng.choice(["standard", "pipelined", "mixed"])
        if matrix == "tridiag":
            impl = rng.choice(["standard", "pipelined"])
            return _cg(matrix, _log_int(rng, 10000, 4000000), impl, tol=0.0, maxiter=rng.randint(10, 20))
        lo, hi = {"poisson": (24, 120), "stencil2d": (64, 480), "stencil3d": (16, 80), "csr2d": (64, 320)}[matrix]
        return _cg(matrix, _log_int(rng, lo, hi), impl)
    if kind == "fpcg":
        net = rng.random() < 0.5
        ny = 16 * rng.randint(8, 32) if net else rng.randint(64, 512)
        return _fpcg(ny, 512 if net else rng.randint(64, 512), net, rng.choice(["fp32", "fp64"]))
    if kind == "batch":
        return _batch(rng.randint(2, 20), rng.randint(1, 5), rng.randint(2, 10**6), rng.choice(["fp32", "fp64"]))
    return _unet(8 * rng.randint(8, 32), 256, rng.randint(1, 8))


# ------------------------------------------------------------------ inputs
class _DeviceGrid:
    """The current grid of a Jacobi handle as torch can take it without a copy.
    A tensor made from it keeps it, and so the handle that owns the memory."""

    def __init__(self, jacobi):
        self.jacobi = jacobi
        self.__cuda_array_interface__ = {"shape": jacobi.shape, "typestr": np.dtype(jacobi.dtype).str,
                                         "data": (jacobi.device_grid(), False), "version": 3}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _jacobi_grid(case, seed):
    """Initial grid: every cell random, the halo rows and planes too (they need
    not be periodic images before the first sweep)."""
    shape = (case["nz"], case["ny"], case["nx"]) if case["dims"] == 3 else (case["ny"], case["nx"])
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    return torch.rand(shape, generator=_generator(seed), device="cuda", dtype=dtype) * 2 - 1


def _tridiag_values(n, seed):
    """(diagonal, off-diagonal) of a random symmetric tridiagonal matrix distributed as
    the reference's (diagonal in 10..11, off-diagonals in 0..1)."""
    u = torch.rand((2, n), generator=_generator(seed), device="cuda", dtype=torch.float64)
    return u[0] + 10.0, u[1, : n - 1]


def _tridiag_csr(diag, off):
    n = diag.numel()
    val = torch.zeros(3 * n, dtype=torch.float64, device="cuda").view(n, 3)
    val[1:, 0] = off
    val[:, 1] = diag
    val[:-1, 2] = off
    col = (torch.arange(n, device="cuda", dtype=torch.int32)[:, None] +
           torch.tensor([-1, 0, 1], device="cuda", dtype=torch.int32))
    rowptr = torch.arange(n + 1, device="cuda", dtype=torch.int32) * 3 - 1
    rowptr[0], rowptr[n] = 0, 3 * n - 2
    return (rowptr.cpu().numpy(), col.reshape(-1)[1:-1].contiguous().cpu().numpy(),
            val.reshape(-1)[1:-1].contiguous().cpu().numpy())


def _stencil_csr(k):
    """The variable-coefficient operator of a 2D grid assembled as CSR."""
    ny, nx = k.shape
    we, wn, _, dg = (a.reshape(ny, nx) for a in cfm.varcoef_coeffs(k))
    i = np.arange(ny * nx, dtype=np.int32).reshape(ny, nx)
    val = np.zeros((ny, nx, 5))
    col = np.zeros((ny, nx, 5), np.int32)
    keep = np.zeros((ny, nx, 5), bool)
    val[1:, :, 0], col[1:, :, 0], keep[1:, :, 0] = -wn[:-1], i[:-1], True
    val[:, 1:, 1], col[:, 1:, 1], keep[:, 1:, 1] = -we[:, :-1], i[:, :-1], True
    val[:, :, 2], col[:, :, 2], keep[:, :, 2] = dg, i, True
    val[:, :-1, 3], col[:, :-1, 3], keep[:, :-1, 3] = -we[:, :-1], i[:, 1:], True
    val[:-1, :, 4], col[:-1, :, 4], keep[:-1, :, 4] = -wn[:-1], i[1:], True
    rowptr = np.zeros(ny * nx + 1, np.int32)
    rowptr[1:] = np.cumsum(keep.reshape(-1, 5).sum(1))
    return rowptr, col[keep], val[keep]


def _cg_shape(case):
    side = case["size"]
    return (side, side, side) if case["matrix"] == "stencil3d" else (side, side)


def _batch_shapes(case):
    """Sides log-uniform, 64 to 512 in 2D and 32 to 80 in 3D."""
    rng = random.Random(case["sizes"])
    return ([(_log_int(rng, 64, 512),) * 2 for _ in range(case["n2d"])] +
            [(_log_int(rng, 32, 80),) * 3 for _ in range(case["n3d"])])


def _batch_systems(case, seed):
    return [cfm.varcoef_problem(shape, int(seed) * 1000 + i) for i, shape in enumerate(_batch_shapes(case))]


def _unet_inputs(case, seed):
    """Normalised residual and log k, and the gradient with respect to the output."""
    B, H, W = case["batch"], case["height"], case["width"]
    g = _generator(seed)
    x = torch.randn((B, H, W, 2), generator=g, device="cuda")
    dout = torch.randn((B, H, W), generator=g, device="cuda")
    return x.cpu().numpy(), dout.cpu().numpy()


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "jacobi":
        j = cfm.Jacobi(case["dims"], case["nx"], case["ny"], case["nz"], PRECISIONS[case["precision"]],
                       int(case["periodic_y"]), JACOBI_IMPLS[case["impl"]])
        if case["mirror"]:
            j.set_boundary(cfm.BOUNDARY_MIRROR)
        j.upload(_jacobi_grid(case, seed).cpu().numpy())
        s["jacobi"] = j
    elif kind == "cg":
        n, matrix = case["size"], case["matrix"]
        if matrix == "poisson":
            A = cfm.CSR(*cfm.poisson3d(n))
        elif matrix == "tridiag":
            A = cfm.CSR(*_tridiag_csr(*_tridiag_values(n, seed)))
        else:
            k, _ = cfm.varcoef_problem(_cg_shape(case), int(seed))
            A = cfm.CSR(*_stencil_csr(k)) if matrix == "csr2d" else cfm.Stencil(k)
        s["cg"] = cfm.CG(A, CG_IMPLS[case["impl"]], case["maxiter"], case["tol"])
        s["b"] = _cg_rhs(case, seed, A.n)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "fpcg":
        k, f = cfm.varcoef_problem((case["ny"], case["nx"]), int(seed))
        net = None
        if case["net"]:
            # random weights of the architecture, used at half the system's resolution
            net = cfm.UNet(case["ny"] // 2, case["nx"] // 2, max_batch=1, seed=int(seed))
            net.set_training_info(SMOOTH, 2)
        s["fpcg"] = cfm.FPCG(cfm.Stencil(k), k, net, maxiter=5000, tol=case["tol"], smooth=SMOOTH,
                             precision=PRECISIONS[case["precision"]])
        s["f"] = f
    elif kind == "batch":
        B = cfm.Batch(_batch_systems(case, seed))
        B.set_solver(SMOOTH, MAXITER, case["tol"])
        B.set_precision(PRECISIONS[case["precision"]])
        s["batch"] = B
    else:
        s["net"] = cfm.UNet(case["height"], case["width"], max_batch=case["batch"], seed=int(seed))
        s["x"], s["dout"] = _unet_inputs(case, seed)
    torch.cuda.synchronize()  # the library works on its own streams
    return s


def _cg_rhs(case, seed, n):
    return torch.randn(n, generator=_generator(int(seed) + 1), device="cuda", dtype=torch.float64)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "jacobi":
        j = s["jacobi"]
        j.run(case["niter"])
        return torch.as_tensor(_DeviceGrid(j), device="cuda")
    if kind == "cg":
        s["cg"].solve_device(s["b"].data_ptr(), s["x"].data_ptr())
        return s["x"]
    if kind == "fpcg":
        return s["fpcg"].solve(s["f"])[0]
    if kind == "batch":
        B = s["batch"]
        B.solve()
        return np.concatenate([B.solution(i) for i in range(B.n)])
    return s["net"].gradient(s["x"], s["dout"])


# ----------------------------------------------------- what a pass cannot do without
def _operator(matrix, shape):
    """(rows, nonzeros, typical CG iterations to 1e-8) of a system."""
    n = int(np.prod(shape))
    side = max(shape)
    faces = sum(2 * (n - n // d) for d in shape)
    its = {"poisson": 2.6 * side, "tridiag": 10.0}.get(matrix, 20.0 * side if len(shape) == 2 else 9.0 * side)
    return n, n + faces, its


def work(case):
    """bytes: each input once and each output once; flops: the updates of the
    asked sweeps, for the solvers those of a typical iteration count."""
    kind = case["kind"]
    if kind == "jacobi":
        cells = case["nx"] * case["ny"] * (case["nz"] if case["dims"] == 3 else 1)
        word = 8 if case["precision"] == "fp64" else 4
        return {"bytes": 2.0 * word * cells, "flops": (4.0 if case["dims"] == 2 else 6.0) * cells * case["niter"]}
    if kind == "cg":
        if case["matrix"] == "tridiag":
            n, nnz, its = case["size"], 3 * case["size"] - 2, case["maxiter"]
        else:
            shape = (case["size"],) * 3 if case["matrix"] == "poisson" else _cg_shape(case)
            n, nnz, its = _operator(case["matrix"], shape)
        matrix_free = case["matrix"].startswith("stencil")
        words = 8.0 * (3 if case["matrix"] == "stencil2d" else 4) * n if matrix_free else 12.0 * nnz + 4.0 * (n + 1)
        return {"bytes": words + 16.0 * n, "flops": its * (2.0 * nnz + 10.0 * n)}
    if kind == "fpcg":
        n = case["ny"] * case["nx"]
        its = 1.4 * max(case["ny"], case["nx"])
        flops = its * n * (2 * SMOOTH + 2) * 10.0
        if case["net"]:
            flops += its / 2 * _unet_flops(case["ny"] // 2, case["nx"] // 2)
        return {"bytes": 8.0 * 5 * n, "flops": flops}
    if kind == "batch":
        nbytes = flops = 0.0
        for shape in _batch_shapes(case):
            n, nnz, its = _operator("varcoef", shape)
            nbytes += 8.0 * (len(shape) + 3) * n
            flops += its / 5 * (2.0 * nnz * (SMOOTH + 1) + 14.0 * n)
        return {"bytes": nbytes, "flops": flops}
    B, H, W = case["batch"], case["height"], case["width"]
    return {"bytes": B * H * W * 12.0 + 8.0 * cfm.lib.cfm_unet_num_params(), "flops": 3.0 * B * _unet_flops(H, W)}


LAYERS = [("cin", 0, 2, 32), ("e1", 1, 32, 64), ("e2", 2, 64, 128), ("e3", 3, 128, 256), ("d3", 3, 256, 128),
          ("d2", 2, 128, 64), ("d1", 1, 64, 32), ("d0", 0, 32, 32), ("cout", 0, 32, 1)]


def _unet_flops(H, W):
    return sum(18.0 * ci * co * (H >> lev) * (W >> lev) for _, lev, ci, co in LAYERS)


def tolerance(case):
    kind = case["kind"]
    if kind == "jacobi":
        return "exact"  # the sum order of a cell is part of the contract
    if kind == "cg" and case["matrix"] == "tridiag":
        return {"rel": 1e-11}  # a fixed count past convergence: the pipelined recurrence's rounding (2e-12 seen)
    if kind in ("cg", "fpcg", "batch"):
        # solved to a relative residual of 1e-8; the solution's error is that
        # times the conditioning (up to 2.6e-7 seen against exact())
        return {"rel": 1e-6}
    return {"rel": 3e-2}


# ------------------------------------------------------------------ in 64 bits
def _exact_jacobi(case, seed):
    a = _jacobi_grid(case, seed).double()
    b = a.clone()
    three = case["dims"] == 3
    wrap_y = not three or case["periodic_y"]
    for _ in range(case["niter"]):
        if three:
            c = slice(1, -1)
            b[c, c, c] = (a[c, c, 2:] + a[c, c, :-2] + a[c, 2:, c] + a[c, :-2, c] + a[2:, c, c] + a[:-2, c, c]) / 6.0
            if wrap_y:
                b[c, 0], b[c, -1] = b[c, -2], b[c, 1]
            b[0], b[-1] = b[-2], b[1]
        else:
            mid = a[1:-1]
            if case["mirror"]:
                east = torch.cat([mid[:, 1:], mid[:, -1:]], 1)
                west = torch.cat([mid[:, :1], mid[:, :-1]], 1)
                b[1:-1] = (a[2:] + a[:-2] + east + west) / 4.0
            else:
                b[1:-1, 1:-1] = (mid[:, 2:] + mid[:, :-2] + a[2:, 1:-1] + a[:-2, 1:-1]) / 4.0
            b[0], b[-1] = b[-2], b[1]
        a, b = b, a
    return a


def _poisson_apply(shape):
    def apply(u):
        v = u.view(shape)
        t = 6.0 * v
        t[1:] -= v[:-1]
        t[:-1] -= v[1:]
        t[:, 1:] -= v[:, :-1]
        t[:, :-1] -= v[:, 1:]
        t[:, :, 1:] -= v[:, :, :-1]
        t[:, :, :-1] -= v[:, :, 1:]
        return t.view(-1)
    return apply, torch.full((int(np.prod(shape)),), 6.0, device="cuda", dtype=torch.float64)


def _tridiag_apply(diag, off):
    def apply(u):
        t = diag * u
        t[1:] += off * u[:-1]
        t[:-1] += off * u[1:]
        return t
    return apply, diag


def _varcoef_apply(k):
    """-div(k grad u) with harmonic means on the faces, 2 k on the boundary faces."""
    k = torch.from_numpy(np.ascontiguousarray(k)).cuda()
    faces, diag = [], torch.zeros_like(k)
    for axis in range(k.dim() - 1, -1, -1):
        m = k.shape[axis]
        lo, hi = k.narrow(axis, 0, m - 1), k.narrow(axis, 1, m - 1)
        w = 2.0 * lo * hi / (lo + hi)
        faces.append((axis, w))
        diag.narrow(axis, 1, m - 1).add_(w)
        diag.narrow(axis, 0, m - 1).add_(w)
        diag.narrow(axis, 0, 1).add_(2.0 * k.narrow(axis, 0, 1))
        diag.narrow(axis, m - 1, 1).add_(2.0 * k.narrow(axis, m - 1, 1))

    def apply(u):
        v = u.view(k.shape)
        t = diag * v
        for axis, w in faces:
            m = k.shape[axis]
            t.narrow(axis, 1, m - 1).sub_(w * v.narrow(axis, 0, m - 1))
            t.narrow(axis, 0, m - 1).sub_(w * v.narrow(axis, 1, m - 1))
        return t.view(-1)
    return apply, diag.reshape(-1)


def _solve(apply, diag, b, rel=1e-13, maxiter=40000):
    """Diagonally preconditioned CG in 64 bits, to the residual it can reach."""
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    stop = rel * float(b.norm())
    for it in range(maxiter):
        if it % 100 == 0 and float(r.norm()) <= stop:
            break
        q = apply(p)
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_unet(case, seed):
    """Gradient of sum(out * dout) by autograd in 64 bits, on the weights rounded
    to BF16 where the library's tensor-core layers hold them so."""
    net = cfm.UNet(case["height"], case["width"], max_batch=case["batch"], seed=int(seed))
    theta = torch.from_numpy(net.params()).cuda()
    net.close()
    params, at = {}, 0
    for name, _, ci, co in LAYERS:
        w = theta[at:at + 9 * co * ci].view(9, co, ci)
        b = theta[at + 9 * co * ci:at + 9 * co * ci + co]
        at += 9 * co * ci + co
        if name not in ("cin", "cout"):
            w = w.bfloat16()
        params[name] = (w.double().requires_grad_(), b.double().requires_grad_())
    x, dout = (torch.from_numpy(a).cuda().double() for a in _unet_inputs(case, seed))
    conv = torch.nn.functional.conv2d

    def layer(h, name, relu=True):
        w, b = params[name]
        h = conv(h, w.view(3, 3, *w.shape[1:]).permute(2, 3, 0, 1), b, padding=1)
        return torch.relu(h) if relu else h

    def up(h):
        return h.repeat_interleave(2, 2).repeat_interleave(2, 3)

    pool = torch.nn.functional.avg_pool2d
    h0 = layer(x.permute(0, 3, 1, 2), "cin")
    h1 = layer(pool(h0, 2), "e1")
    h2 = layer(pool(h1, 2), "e2")
    h3 = layer(pool(h2, 2), "e3")
    g3 = layer(h3, "d3")
    g2 = layer(up(g3) + h2, "d2")
    g1 = layer(up(g2) + h1, "d1")
    g0 = layer(up(g1) + h0, "d0")
    out = layer(g0, "cout", relu=False)
    (out[:, 0] * dout).sum().backward()
    return torch.cat([torch.cat([params[name][0].grad.reshape(-1), params[name][1].grad.reshape(-1)])
                      for name, *_ in LAYERS])


def exact(case, seed):
    kind = case["kind"]
    if kind == "jacobi":
        return _exact_jacobi(case, seed)
    if kind == "cg":
        if case["matrix"] == "poisson":
            apply, diag = _poisson_apply((case["size"],) * 3)
        elif case["matrix"] == "tridiag":
            apply, diag = _tridiag_apply(*_tridiag_values(case["size"], seed))
        else:
            apply, diag = _varcoef_apply(cfm.varcoef_problem(_cg_shape(case), int(seed))[0])
        return _solve(apply, diag, _cg_rhs(case, seed, diag.numel()))
    if kind == "fpcg":
        k, f = cfm.varcoef_problem((case["ny"], case["nx"]), int(seed))
        return _solve(*_varcoef_apply(k), torch.from_numpy(f.reshape(-1)).cuda())
    if kind == "batch":
        if case["n2d"] + case["n3d"] > 30:
            return None
        return torch.cat([_solve(*_varcoef_apply(k), torch.from_numpy(np.ascontiguousarray(b).reshape(-1)).cuda(),
                                 rel=1e-12) for k, b in _batch_systems(case, seed)])
    return _exact_unet(case, seed)
