"""The work that programs have this framework do, as timed cases on the GPU.

Systems (all made on the GPU from the seed):
  stencil2d / stencil3d  upwind convection-diffusion on an N x N or N x N x N grid (5 / 7 points)
  banded                 17 entries per row: the diagonal, 10 within +-64 and 6 far columns
  powerlaw               power-law row lengths with a few dense rows, uniform random columns
"""
import math

import torch

from hethyppar_gb300 import Context, Matrix, bicgstab, reorder_color
from hethyppar_gb300._lib import check, lib
from hethyppar_gb300.autograd import SparseSolve

MAXIT = 4000  # iteration cap of the solves
_ctx = None


def _context():
    """The one context (stream) that a program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def listed():
    return [
        # a host program's own Krylov step on the BLAS-1 entry points: latency and launches count
        {"name": "blas1_65k", "kind": "blas1", "n": 65_537},
        # the smallest product: one 5-point operator on a 256 x 256 grid inside an outer loop
        {"name": "spmv_stencil2d_256", "kind": "spmv", "system": "stencil2d", "N": 256, "dtype": "fp64"},
        # the ordinary product: SuiteSparse-sized rows, some of them far from the diagonal
        {"name": "spmv_banded_450k", "kind": "spmv", "system": "banded", "N": 450_000, "dtype": "fp64"},
        # a graph-like matrix: irregular rows, gathers without locality
        {"name": "spmv_powerlaw_3500k", "kind": "spmv", "system": "powerlaw", "N": 3_500_000, "dtype": "fp64"},
        # the single-precision product on a large 3D grid (memory traffic halved by the caller's choice)
        {"name": "spmv_f32_stencil3d_160", "kind": "spmv", "system": "stencil3d", "N": 160, "dtype": "fp32"},
        # y = alpha A x + beta y on a caller's own CSR arrays, for hosts that own all device memory
        {"name": "noalloc_banded_450k", "kind": "noalloc", "system": "banded", "N": 450_001},
        # the small solve, bound by launches: a 2D grid to the tolerance of the differentiable solve
        {"name": "solve_stencil2d_256", "kind": "solve", "system": "stencil2d", "N": 256, "precision": "fp64",
         "rtol": 1e-12},
        # the headline solve: few iterations on a matrix of SuiteSparse size
        {"name": "solve_banded_450k", "kind": "solve", "system": "banded", "N": 450_000, "precision": "fp64",
         "rtol": 1e-10},
        # the large solve in double precision
        {"name": "solve_stencil3d_160", "kind": "solve", "system": "stencil3d", "N": 160, "precision": "fp64",
         "rtol": 1e-13},
        # the same system by single-precision iterations refined in double
        {"name": "mixed_stencil3d_160", "kind": "solve", "system": "stencil3d", "N": 160, "precision": "mixed",
         "rtol": 1e-13},
        # a training step through a solve layer: new matrix values, forward solve, adjoint, gradients
        {"name": "train_banded_300k", "kind": "train", "system": "banded", "N": 300_000},
        # one application of the ILU(0) preconditioner in multicolour order
        {"name": "ilu_apply_stencil2d_1024", "kind": "ilu", "system": "stencil2d", "N": 1024},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["blas1", "spmv", "spmv", "spmv", "noalloc", "solve", "solve", "solve", "train", "ilu"])
    if kind == "blas1":
        return {"kind": kind, "n": log(1_000, 16_000_000)}
    if kind == "ilu":
        return {"kind": kind, "system": "stencil2d", "N": log(48, 1024)}
    if kind == "train":
        return {"kind": kind, "system": "banded", "N": log(4_000, 300_000)}
    if kind == "solve":
        system = rng.choice(["stencil2d", "banded", "stencil3d"])
        n = {"stencil2d": log(32, 256), "banded": log(4_000, 450_000), "stencil3d": log(16, 150)}[system]
        return {"kind": kind, "system": system, "N": n, "precision": rng.choice(["fp64", "fp64", "mixed"]),
                "rtol": 1e-13 if system == "stencil3d" else 1e-12}
    system = rng.choice(["stencil2d", "banded", "powerlaw", "stencil3d"])
    n = {"stencil2d": log(64, 2048), "banded": log(4_000, 450_000), "powerlaw": log(20_000, 3_500_000),
         "stencil3d": log(16, 160)}[system]
    case = {"kind": kind, "system": system, "N": n}
    if kind == "spmv":
        case["dtype"] = rng.choice(["fp64", "fp64", "fp32", "transpose"])
    return case


# ---- systems -----------------------------------------------------------------------------------
# Each gives (rowptr, col, val, mul): the CSR on the GPU and, where rows have a bounded length, the
# function x -> A x summed row by row in a fixed order (None for power-law rows).


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _padded(cols, vals, keep):
    """The CSR of rows given as dense (m, k) columns and values with a mask, and x -> A x."""
    counts = keep.sum(1)
    rowptr = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=rowptr[1:])
    cc, vv = torch.where(keep, cols, 0), torch.where(keep, vals, 0.0)

    def mul(x):
        y = torch.zeros(cols.shape[0], dtype=torch.float64, device="cuda")
        for k in range(cols.shape[1]):
            y += vv[:, k] * x[cc[:, k]]
        return y

    return rowptr.int(), cols[keep].int(), vals[keep].double(), mul


def _stencil(N, nd):
    """First-order upwind convection-diffusion scaled by h^2, as in the repository's benchmark:
    Pe 50 with velocity (1, 0.5) in 2D, Pe 20 with (1, 1, 1)/sqrt(3) in 3D."""
    pe, vel = (50.0, (1.0, 0.5)) if nd == 2 else (20.0, (3.0 ** -0.5,) * 3)
    h, m = 1.0 / (N + 1), N ** nd
    idx = torch.arange(m, device="cuda")
    cols = torch.empty(m, 2 * nd + 1, dtype=torch.int64, device="cuda")
    keep = torch.ones(m, 2 * nd + 1, dtype=torch.bool, device="cuda")
    vals = torch.empty(m, 2 * nd + 1, dtype=torch.float64, device="cuda")
    for d in range(nd):
        stride = N ** d
        at = (idx // stride) % N
        cols[:, nd - 1 - d], keep[:, nd - 1 - d], vals[:, nd - 1 - d] = idx - stride, at > 0, -1.0 - h * pe * vel[d]
        cols[:, nd + 1 + d], keep[:, nd + 1 + d], vals[:, nd + 1 + d] = idx + stride, at < N - 1, -1.0
    cols[:, nd], vals[:, nd] = idx, 2.0 * nd + h * pe * sum(vel)
    return _padded(cols, vals, keep)


def _banded(m, g):
    offs = torch.cat([torch.arange(-64, 0, device="cuda"), torch.arange(1, 65, device="cuda")])
    idx = torch.arange(m, device="cuda")[:, None]
    near = idx + offs
    key = torch.rand(m, 128, device="cuda", generator=g)
    key[(near < 0) | (near >= m)] = 2.0
    near = torch.gather(near, 1, key.topk(10, dim=1, largest=False).indices)
    # one far column in each sixth of the matrix; one that falls into the band moves out of it
    part = m // 6
    far = (torch.rand(m, 6, device="cuda", generator=g) * part).long() + torch.arange(6, device="cuda") * part
    far = torch.where((far - idx).abs() <= 64, (far + 131) % m, far)
    off = -torch.rand(m, 16, dtype=torch.float64, device="cuda", generator=g)
    cols = torch.cat([near, far, idx], 1)
    vals = torch.cat([off, 1.05 * off.abs().sum(1, keepdim=True)], 1)
    order = torch.sort(cols, dim=1, stable=True).indices
    cols, vals = torch.gather(cols, 1, order), torch.gather(vals, 1, order)
    return _padded(cols, vals, torch.ones_like(cols, dtype=torch.bool))


def _powerlaw(m, g):
    """Off-diagonal row lengths with a power-law tail (exponent 2.1, capped), 20 dense rows of
    m / 70 to m / 35 entries, a dominant diagonal."""
    top = max(64, m // 35)
    u = torch.rand(m, dtype=torch.float64, device="cuda", generator=g)
    lens = u.clamp_min(1e-12).pow(-1.0 / 1.1).floor().long().clamp(1, top)
    dense = torch.randint(0, m, (20,), device="cuda", generator=g)
    lens[dense] = torch.randint(top // 2, top + 1, (20,), device="cuda", generator=g)
    rows = torch.repeat_interleave(torch.arange(m, device="cuda"), lens)
    cols = torch.randint(0, m, (rows.numel(),), device="cuda", generator=g)
    vals = torch.randn(rows.numel(), dtype=torch.float64, device="cuda", generator=g)
    diag = torch.arange(m, device="cuda")
    rows, cols, vals = torch.cat([rows, diag]), torch.cat([cols, diag]), torch.cat([vals, 1.1 * lens.double()])
    order = torch.sort(rows * m + cols, stable=True).indices
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens + 1, 0, out=rowptr[1:])
    return rowptr.int(), cols[order].int(), vals[order], None


def _system(case, g):
    if case["system"] == "stencil2d":
        return _stencil(case["N"], 2)
    if case["system"] == "stencil3d":
        return _stencil(case["N"], 3)
    return _banded(case["N"], g) if case["system"] == "banded" else _powerlaw(case["N"], g)


def _rows_of(rowptr):
    m = rowptr.numel() - 1
    return torch.repeat_interleave(torch.arange(m, device="cuda"), rowptr.diff().long())


def _randn(n, g):
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def _uniform(n, g):
    return 2.0 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g) - 1.0


# ---- inputs ------------------------------------------------------------------------------------
def _inputs(case, seed):
    """The numbers of a case, before any of the framework's objects."""
    g = _generator(seed)
    kind = case["kind"]
    if kind == "blas1":
        n = case["n"]
        return {"x": _randn(n, g), "y": _randn(n, g), "alpha": 0.37, "beta": 0.91}
    rowptr, col, val, mul = _system(case, g)
    m = rowptr.numel() - 1
    d = {"rowptr": rowptr, "col": col, "val": val, "mul": mul, "m": m}
    if kind == "spmv":
        d["x"] = _randn(m, g).float() if case["dtype"] == "fp32" else _randn(m, g)
    elif kind == "noalloc":
        d |= {"x": _randn(m, g), "y0": _randn(m, g), "alpha": 1.25, "beta": -0.5}
    elif kind == "solve":
        d["x_target"] = _uniform(m, g)
        d["b"] = mul(d["x_target"])
    elif kind == "train":
        d["x_target"], d["fit"] = _randn(m, g), _randn(m, g)
        d["b"] = mul(d["x_target"])
    elif kind == "ilu":
        d["r"] = _randn(m, g)
    return d


def prepare(case, seed):
    ctx = _context()
    s = _inputs(case, seed)
    s.pop("mul", None)
    s["kind"], s["ctx"] = case["kind"], ctx
    kind = case["kind"]
    if kind == "blas1":
        s |= {"out": torch.empty(1, dtype=torch.float64, device="cuda"), "z": torch.empty_like(s["x"])}
        return s
    m = s["m"]
    if kind == "noalloc":
        s["y"] = s["y0"].clone()
        s["stream"] = torch.cuda.current_stream().cuda_stream
        return s
    if kind == "ilu":
        perm, _ = reorder_color(s["rowptr"].cpu().numpy(), s["col"].cpu().numpy())
        A = Matrix.from_csr(ctx, s["rowptr"].cpu().numpy(), s["col"].cpu().numpy(), s["val"].cpu().numpy(), perm=perm)
        s |= {"A": A, "r": s["r"][torch.from_numpy(perm).cuda().long()], "z": torch.empty(m, dtype=torch.float64, device="cuda")}
        A.ilu0_apply_dev(s["r"], s["z"])
    else:
        A = s["A"] = Matrix.from_csr_dev(ctx, m, m, s["rowptr"], s["col"], s["val"])
        if kind == "spmv":
            s["dtype"] = case["dtype"]
            s["y"] = torch.empty_like(s["x"])
            run(s)  # the layout is made once
        elif kind == "solve":
            s["precision"], s["rtol"] = case["precision"], case["rtol"]
            # workspace and loop graph, made once: a solve that is done at its first test
            bicgstab(ctx, A, s["b"], rtol=1.0, maxit=MAXIT, precision=s["precision"])
        else:
            s["val"].requires_grad_()
            s["b"].requires_grad_()
    if kind != "train":
        for k in ("rowptr", "col", "val"):
            s.pop(k)
    ctx.sync()
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "blas1":
        ctx.dot(s["x"], s["y"], out=s["out"])
        ctx.copy(s["y"], s["z"])
        ctx.axpy(s["alpha"], s["x"], s["z"])
        ctx.scal(s["beta"], s["z"])
        return s["out"], s["z"]
    if kind == "spmv":
        if s["dtype"] == "fp32":
            s["A"].spmv_f32_dev(s["x"], s["y"])
        elif s["dtype"] == "transpose":
            s["A"].spmv_t_dev(s["x"], s["y"])
        else:
            s["A"].spmv_dev(s["x"], s["y"])
        return s["y"]
    if kind == "noalloc":
        s["y"].copy_(s["y0"])
        check(lib().hhp_spmv_csr_noalloc(s["m"], s["m"], s["col"].numel(), s["rowptr"].data_ptr(), s["col"].data_ptr(),
                                         s["val"].data_ptr(), s["alpha"], s["x"].data_ptr(), s["beta"],
                                         s["y"].data_ptr(), s["stream"]), "hhp_spmv_csr_noalloc")
        return s["y"]
    if kind == "ilu":
        s["A"].ilu0_apply_dev(s["r"], s["z"])
        return s["z"]
    if kind == "solve":
        x, res = bicgstab(ctx, s["A"], s["b"], rtol=s["rtol"], maxit=MAXIT, precision=s["precision"])
        return x
    x = SparseSolve.apply(s["val"], s["b"], s["A"], ctx)
    dval, db = torch.autograd.grad(0.5 * (x - s["fit"]).square().sum(), (s["val"], s["b"]))
    return x.detach(), dval, db


# ---- what a pass cannot do without -----------------------------------------------------------------
def _shape(case):
    """(rows, entries) of a case's matrix; power-law entries on average."""
    N = case["N"]
    if case["system"] == "stencil2d":
        return N * N, 5 * N * N - 4 * N
    if case["system"] == "stencil3d":
        return N ** 3, 7 * N ** 3 - 6 * N * N
    return (N, 17 * N) if case["system"] == "banded" else (N, int(6.1 * N))


def work(case):
    kind = case["kind"]
    if kind == "blas1":
        return {"bytes": 72.0 * case["n"], "flops": 5.0 * case["n"]}
    m, nnz = _shape(case)
    spmv = 12.0 * nnz + 20.0 * m
    if kind == "spmv":
        return {"bytes": 8.0 * nnz + 12.0 * m if case["dtype"] == "fp32" else spmv, "flops": 2.0 * nnz}
    if kind == "noalloc":
        return {"bytes": spmv + 24.0 * m, "flops": 2.0 * nnz}
    if kind == "ilu":
        return {"bytes": 12.0 * nnz + 24.0 * m, "flops": 2.0 * nnz}
    # iterations of plain BiCGStab on these systems; each applies A twice and passes 16 vectors
    iters = {"stencil2d": 1.8 * case["N"], "stencil3d": 2.6 * case["N"], "banded": 20.0}[case["system"]]
    per = 2.0 * spmv + 128.0 * m
    flops = 4.0 * nnz + 24.0 * m
    if kind == "train":  # both solves, the values in, both gradients out
        return {"bytes": 2.0 * iters * per + 40.0 * nnz, "flops": 2.0 * iters * flops}
    if case["precision"] == "mixed":
        per = 2.0 * (8.0 * nnz + 12.0 * m) + 64.0 * m
    return {"bytes": iters * per, "flops": iters * flops}


# ---- the same results in 64 bits by plain torch ----------------------------------------------------
def _bicgstab(mul, b, rtol=1e-15, most=200):
    x, r = torch.zeros_like(b), b.clone()
    r0, p = b.clone(), b.clone()
    rho = r0 @ r
    for _ in range(most):
        v = mul(p)
        alpha = rho / (r0 @ v)
        s = r - alpha * v
        t = mul(s)
        omega = (t @ s) / (t @ t)
        x += alpha * p + omega * s
        r = s - omega * t
        if r.norm() <= rtol * b.norm():
            break
        new = r0 @ r
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    if kind == "blas1":
        return (d["x"] @ d["y"]).reshape(1), d["beta"] * (d["y"] + d["alpha"] * d["x"])
    if kind in ("spmv", "noalloc"):
        rows, cols, x = _rows_of(d["rowptr"]), d["col"].long(), d["x"].double()
        val = d["val"].float().double() if case.get("dtype") == "fp32" else d["val"]
        if case.get("dtype") == "transpose":
            rows, cols = cols, rows
        y = torch.zeros(d["m"], dtype=torch.float64, device="cuda").index_add_(0, rows, val * x[cols])
        return d["alpha"] * y + d["beta"] * d["y0"] if kind == "noalloc" else y
    if kind == "solve":
        return d["x_target"]
    if kind == "train":
        rows, cols, n = _rows_of(d["rowptr"]), d["col"].long(), d["m"]
        lam = _bicgstab(lambda x: torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, cols, d["val"] * x[rows]),
                        d["x_target"] - d["fit"])
        return d["x_target"], -lam[rows] * d["x_target"][cols], lam
    # ILU(0) on two colours (the parity of the grid point), in the order of the framework's permutation:
    # the second colour's pivot is a_ii - sum a_ik a_ki / a_kk
    N = case["N"]
    perm, _ = reorder_color(d["rowptr"].cpu().numpy(), d["col"].cpu().numpy())
    rows, cols, val, m = _rows_of(d["rowptr"]), d["col"].long(), d["val"], d["m"]
    idx = torch.arange(m, device="cuda")
    second = (idx // N + idx % N) % 2 == 1
    on = rows == cols
    a = torch.zeros(m, dtype=torch.float64, device="cuda")
    a[rows[on]] = val[on]
    r, c, v = rows[~on], cols[~on], val[~on]
    # a_ki of the mirrored entry: entries sorted by (column, row) are the transpose's, in the same places
    back = v[torch.argsort(c * m + r)]
    u = a - second * torch.zeros_like(a).index_add_(0, r, v * back / a[c])
    rhs = d["r"]
    z2 = second * (rhs - torch.zeros_like(a).index_add_(0, r, v * rhs[c] / a[c])) / u
    z1 = ~second * (rhs - torch.zeros_like(a).index_add_(0, r, v * z2[c])) / a
    return (z1 + z2)[torch.from_numpy(perm).cuda().long()]
