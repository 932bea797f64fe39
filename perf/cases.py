"""The work that is timed: what a program that links this library has it do.

The systems are the library's own: Q1 diffusion on uniform 2D and 3D grids
(lexicographic rows, Dirichlet rows as identity rows, a lognormal coefficient
exp(sigma g) per cell) and upwinded convection-diffusion in 2D.  They are made
here with torch, so that `exact` can solve the same systems in 64 bits without
the library.  Matrices go in as triplets on the device (TransformFromCOO), or
as host CSR where the call takes host arrays (the batch).

Kinds of case ("op"):
  lmp      a few CG iterations written call by call on vectors and a matrix
           (VectorMult, Dot, Axpy, ...): what the CG<LAD> template does on the
           vector and matrix classes; the smallest calls, where each launch
           and each blocking scalar read counts
  spmv     one VectorMult
  cg       Jacobi-PCG to a relative residual
  mp       mixed-precision refinement (FP32 inner solves) to an FP64 residual
  jacobi   a fixed number of damped Jacobi sweeps (smoothing)
  bicgstab BiCGSTAB with right Jacobi preconditioning
  gmres    restarted GMRES with right Jacobi preconditioning
  batch    many independent systems of uneven size solved together, solutions
           read back to host memory
  coo      TransformFromCOO of shuffled triplets, then one product with the
           new matrix
"""
import math

import numpy as np
import torch

from ba_b200 import lmp
from ba_b200.batch import Batch

DEV = "cuda:0"
F64, F32 = "f64", "f32"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # an application's own Krylov loop on a small operator: launch and read-back latency
        dict(name="lmp_calls_2d_32", op="lmp", dim=2, cells=32, sigma=1.0, dtype=F64, steps=3),
        # one product as a program gets it that never tunes: the CSR as assembled
        dict(name="spmv_csr_f64_3d_64", op="spmv", dim=3, cells=64, sigma=1.0, dtype=F64, tuned=False, shuffle=0),
        # a mesh generator's numbering: neighbours near, but no stencil of offsets; FP32, tuned
        dict(name="spmv_mesh_f32_2d_700", op="spmv", dim=2, cells=700, sigma=1.0, dtype=F32, tuned=True, shuffle=4096),
        # small solves inside a larger program (time steps, local problems)
        dict(name="cg_2d_48", op="cg", dim=2, cells=48, sigma=1.0, rtol=1e-10, tuned=False),
        # the ordinary 2D solve: 66,049 rows
        dict(name="cg_2d_256", op="cg", dim=2, cells=256, sigma=0.0, rtol=1e-10, tuned=True),
        # the large 3D solve: 2.1 M rows, 57 M entries
        dict(name="cg_3d_128", op="cg", dim=3, cells=128, sigma=0.0, rtol=1e-10, tuned=True),
        # mixed precision on a strongly varying coefficient at the same size
        dict(name="mp_3d_128", op="mp", dim=3, cells=128, sigma=2.0, rtol=1e-10, tuned=True),
        # smoothing as a multigrid cycle's FP32 level does it
        dict(name="jacobi_f32_3d_96", op="jacobi", dim=3, cells=96, sigma=1.0, dtype=F32, sweeps=10, tuned=True),
        # the solver for operators that may be nonsymmetric
        dict(name="bicgstab_3d_96", op="bicgstab", kind="diffusion", dim=3, cells=96, sigma=1.0, rtol=1e-8, tuned=True),
        # restarted GMRES at an ordinary 3D size
        dict(name="gmres_3d_64", op="gmres", kind="diffusion", dim=3, cells=64, sigma=0.0, rtol=1e-8, basis=50,
             maxits=300, tuned=True),
        # 1,024 uneven 2D systems (16..256 cells per axis) in one batch, mixed precision
        dict(name="batch_1024", op="batch", dim=2, count=1024, lo=16, hi=256, sigma=1.0, rtol=1e-8, mixed=True),
        # matrix ingestion: 24 M shuffled triplets
        dict(name="coo_3d_96", op="coo", dim=3, cells=96, sigma=1.0, dtype=F64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["lmp", "spmv", "cg", "cg", "mp", "jacobi", "bicgstab", "gmres", "batch", "coo"])
    dim = rng.choice([2, 3])
    sigma = rng.choice([0.0, 0.5, 1.0, 2.0])
    if op == "lmp":
        return dict(op=op, dim=2, cells=_log(rng, 16, 200), sigma=sigma, dtype=F64, steps=rng.randint(1, 6))
    if op == "spmv":
        return dict(op=op, dim=dim, cells=_log(rng, 16, 1200) if dim == 2 else _log(rng, 8, 128), sigma=sigma,
                    dtype=rng.choice([F64, F32]), tuned=rng.random() < 0.5, shuffle=rng.choice([0, 0, 512, 4096]))
    if op == "cg":
        return dict(op=op, dim=dim, cells=_log(rng, 16, 768) if dim == 2 else _log(rng, 8, 120), sigma=sigma,
                    rtol=rng.choice([1e-8, 1e-10]), tuned=rng.random() < 0.7)
    if op == "mp":
        return dict(op=op, dim=dim, cells=_log(rng, 24, 512) if dim == 2 else _log(rng, 12, 120), sigma=sigma,
                    rtol=rng.choice([1e-8, 1e-10]), tuned=True)
    if op == "jacobi":
        return dict(op=op, dim=dim, cells=_log(rng, 24, 1000) if dim == 2 else _log(rng, 12, 128), sigma=sigma,
                    dtype=rng.choice([F64, F32]), sweeps=rng.randint(3, 20), tuned=rng.random() < 0.7)
    if op == "bicgstab":
        kind = rng.choice(["diffusion", "convection"])
        if kind == "convection":
            return dict(op=op, kind=kind, dim=2, cells=_log(rng, 24, 400), sigma=20.0, rtol=1e-8, tuned=rng.random() < 0.7)
        return dict(op=op, kind=kind, dim=dim, cells=_log(rng, 24, 256) if dim == 2 else _log(rng, 12, 96),
                    sigma=min(sigma, 1.0), rtol=1e-8, tuned=rng.random() < 0.7)
    if op == "gmres":
        kind = rng.choice(["diffusion", "convection"])
        if kind == "convection":
            return dict(op=op, kind=kind, dim=2, cells=_log(rng, 24, 256), sigma=20.0, rtol=1e-8,
                        basis=rng.choice([30, 50, 100]), maxits=300, tuned=rng.random() < 0.7)
        return dict(op=op, kind=kind, dim=3, cells=_log(rng, 12, 80), sigma=min(sigma, 0.5), rtol=1e-8,
                    basis=rng.choice([30, 50, 100]), maxits=300, tuned=rng.random() < 0.7)
    if op == "batch":
        return dict(op=op, dim=dim, count=_log(rng, 8, 512 if dim == 2 else 64), lo=16 if dim == 2 else 8,
                    hi=rng.randint(64, 256) if dim == 2 else rng.randint(16, 48), sigma=1.0, rtol=1e-8,
                    mixed=rng.random() < 0.7)
    return dict(op="coo", dim=dim, cells=_log(rng, 32, 1000) if dim == 2 else _log(rng, 12, 110), sigma=1.0,
                dtype=rng.choice([F64, F32]))


# ------------------------------------------------------------------ systems (torch, 64 bits)
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _diffusion(dim, n, sigma, g):
    """CSR (rowptr, col, val) of Q1 diffusion on n^dim cells, Dirichlet rows as identity rows, and
    a right-hand side U[0, 1) that is 0 on those rows."""
    m = n + 1
    N = m ** dim
    kp = torch.zeros((n + 2,) * dim, dtype=torch.float64, device=DEV)
    core = (slice(1, n + 1),) * dim
    kp[core] = torch.exp(sigma * torch.randn((n,) * dim, dtype=torch.float64, device=DEV, generator=g)) if sigma else 1.0
    h = 1.0 / n
    elem = {0: 2 / 3, 1: -1 / 6, 2: -1 / 3} if dim == 2 else {0: h / 3, 1: 0.0, 2: -h / 12, 3: -h / 12}
    ax = [torch.arange(m, device=DEV).view([m if a == d else 1 for d in range(dim)]) for a in range(dim)]
    edge = torch.zeros((m,) * dim, dtype=torch.bool, device=DEV)
    for a in range(dim):
        edge |= (ax[a] == 0) | (ax[a] == m - 1)
    lin = torch.arange(N, device=DEV, dtype=torch.int32)
    offs = [tuple(v - 1 for v in o) for o in np.ndindex(*((3,) * dim))]
    cols = torch.empty((N, len(offs)), dtype=torch.int32, device=DEV)
    vals = torch.empty((N, len(offs)), dtype=torch.float64, device=DEV)
    mask = torch.empty((N, len(offs)), dtype=torch.bool, device=DEV)
    for k, d in enumerate(offs):
        ok = torch.ones((m,) * dim, dtype=torch.bool, device=DEV)
        for a in range(dim):
            if d[a]:
                ok &= (ax[a] >= 1) if d[a] < 0 else (ax[a] <= m - 2)
        pick = [((-1, 0) if v == 0 else ((0,) if v == 1 else (-1,))) for v in d]
        ks = torch.zeros((m,) * dim, dtype=torch.float64, device=DEV)
        for cs in np.ndindex(*[len(p) for p in pick]):
            ks += kp[tuple(slice(1 + pick[a][cs[a]], 1 + pick[a][cs[a]] + m) for a in range(dim))]
        ham = sum(1 for v in d if v)
        off = 0
        for v in d:
            off = off * m + v
        cols[:, k] = lin + off
        vals[:, k] = torch.where(edge, 1.0 if ham == 0 else 0.0, elem[ham] * ks).reshape(-1)
        mask[:, k] = ok.reshape(-1)
    rowptr = torch.zeros(N + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = torch.cumsum(mask.sum(1), 0)
    b = torch.rand(N, dtype=torch.float64, device=DEV, generator=g)
    b[edge.reshape(-1)] = 0.0
    return rowptr, cols[mask], vals[mask], b


def _convection(n, peclet, g):
    """5-point diffusion with first-order upwind convection on n x n interior nodes, scaled by h^2."""
    h = 1.0 / (n + 1)
    bx, by = peclet * math.cos(0.3), peclet * math.sin(0.3)
    N = n * n
    lin = torch.arange(N, device=DEV, dtype=torch.int32)
    ix, iy = lin % n, lin // n
    nb = [(-n, -1.0 - h * by, iy > 0), (-1, -1.0 - h * bx, ix > 0), (0, 4.0 + h * (bx + by), ix >= 0),
          (1, -1.0, ix < n - 1), (n, -1.0, iy < n - 1)]
    cols = torch.stack([lin + o for o, _, _ in nb], 1)
    vals = torch.tensor([c for _, c, _ in nb], dtype=torch.float64, device=DEV).expand(N, 5)
    mask = torch.stack([k for _, _, k in nb], 1)
    rowptr = torch.zeros(N + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = torch.cumsum(mask.sum(1), 0)
    return rowptr, cols[mask], vals[mask], torch.rand(N, dtype=torch.float64, device=DEV, generator=g)


def _rows(rowptr):
    n = rowptr.numel() - 1
    return torch.repeat_interleave(torch.arange(n, device=DEV, dtype=torch.int32), (rowptr[1:] - rowptr[:-1]).long())


def _system(case, seed):
    """(rows, cols, vals, b): the case's matrix as row-sorted triplets, and its right-hand side."""
    g = _gen(seed)
    if case.get("kind") == "convection":
        rowptr, col, val, b = _convection(case["cells"], case["sigma"], g)
    else:
        rowptr, col, val, b = _diffusion(case["dim"], case["cells"], case["sigma"], g)
    rows = _rows(rowptr)
    w = case.get("shuffle", 0)
    if w:  # renumber within windows of w nodes; triplets again sorted by row, then column
        n = b.numel()
        key = torch.arange(n, device=DEV) // w + torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
        new = torch.empty(n, dtype=torch.int64, device=DEV)
        new[torch.argsort(key)] = torch.arange(n, device=DEV)
        r, c = new[rows.long()], new[col.long()]
        order = torch.argsort(r * n + c)
        rows, col, val = r[order].int(), c[order].int(), val[order]
        b2 = torch.empty_like(b)
        b2[new] = b
        b = b2
    return rows, col, val, b


def _batch_sizes(case, seed):
    """Cells per axis, log-uniform and spread evenly over the range, so that every seed is the same work."""
    k = case["count"]
    u = (np.arange(k) + 0.5) / k
    sizes = np.rint(np.exp(math.log(case["lo"]) + u * (math.log(case["hi"]) - math.log(case["lo"])))).astype(int)
    np.random.RandomState(int(seed) % (1 << 31)).shuffle(sizes)
    return [int(v) for v in sizes]


def _batch_systems(case, seed):
    g = _gen(seed)
    return [_diffusion(case["dim"], n, case["sigma"], g) for n in _batch_sizes(case, seed)]


# ------------------------------------------------------------------ the library's side
_platform = None


def _plat():
    global _platform
    if _platform is None:
        _platform = lmp.init_platform(0)
    return _platform


def _np(dtype):
    return np.float64 if dtype == F64 else np.float32


def _torch(dtype):
    return torch.float64 if dtype == F64 else torch.float32


def _matrix(case, sys, dtype=F64):
    rows, col, val, b = sys
    A = lmp.B200_CSR_lMatrix.TransformFromCOO(rows, col, val, b.numel(), b.numel(), platform=_plat(), dtype=_np(dtype))
    if case.get("tuned"):
        A.tune()
    return A


def _view(t):
    return lmp.B200_lVector.from_torch(t, platform=_plat())


def _jacobi_pc():
    p = lmp.PreconditionerBlockJacobiStand()
    p.Init_Jacobi()
    return p


def prepare(case, seed):
    op = case["op"]
    st = dict(case=case, op=op)
    _plat()
    if op == "batch":
        host = [tuple(t.cpu().numpy() for t in s) for s in _batch_systems(case, seed)]
        B = Batch(len(host), mixed=case["mixed"], precond=True, rtol=case["rtol"], platform=_plat())
        st["slots"] = B.add_many(host)
        B.tune()
        B.restart()
        sizes = [s[3].shape[0] for s in host]
        st["x"] = torch.empty(sum(sizes), dtype=torch.float64, pin_memory=True)
        flat, at = st["x"].numpy(), 0
        st["views"] = []
        for n in sizes:
            st["views"].append(flat[at:at + n])
            at += n
        st["B"] = B
        return st
    sys = _system(case, seed)
    b = sys[3]
    n = b.numel()
    if op == "coo":
        g = _gen(seed, 1)
        order = torch.randperm(sys[0].numel(), device=DEV, generator=g)
        vt = _torch(case["dtype"])
        st["trip"] = tuple(t[order].contiguous() for t in (sys[0], sys[1], sys[2].to(vt)))
        st["n"] = n
        st["xt"] = torch.rand(n, dtype=torch.float64, device=DEV, generator=g).to(vt)
        st["yt"] = torch.empty_like(st["xt"])
        torch.cuda.synchronize()
        st["xv"], st["yv"] = _view(st["xt"]), _view(st["yt"])
        return st
    torch.cuda.synchronize()
    dtype = case.get("dtype", F64)
    A = _matrix(case, sys, dtype)
    st["A"] = A
    vt = _torch(dtype)
    g = _gen(seed, 2)
    start = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    if op in ("spmv", "jacobi"):
        st["xin"] = start.to(vt)
    st["bt"] = b.to(vt)
    st["xt"] = torch.zeros(n, dtype=vt, device=DEV)
    torch.cuda.synchronize()
    st["b"], st["x"] = _view(st["bt"]), _view(st["xt"])
    if "xin" in st:
        st["xs"] = _view(st["xin"])
    if op == "lmp":
        st["wt"] = {k: torch.zeros(n, dtype=vt, device=DEV) for k in ("r", "p", "q", "z", "d")}
        torch.cuda.synchronize()
        st["w"] = {k: _view(t) for k, t in st["wt"].items()}
        A.extract_invdiagelements(st["w"]["d"])
    elif op == "cg":
        st["s"] = lmp.setup_CG_solver(maxits=20000, atol=0.0, rtol=case["rtol"], dtol=1e8)
        st["s"].SetupOperator(A)
    elif op == "mp":
        s = lmp.MPIR()
        s.SetupOperator(A)
        s.SetMpirParameters(0, 50, 0.0, case["rtol"], 1e8)
        s.SetLowPrecErrCorSolverParameters(20000, 0.0, 0.1, 1e8)
        st["s"] = s
    elif op == "jacobi":
        s = lmp.Jacobi()
        s.Prepare(A)
        s.SetSolveMode(3)
        s.SetInnerIter(1)
        s.SetDampingParameter(0.8)
        s.InitControl(case["sweeps"], 0.0, 0.0, 1e8)
        st["s"] = s
    elif op == "bicgstab":
        s = lmp.BiCGSTAB()
        s.SetupPreconditioner(_jacobi_pc())
        s.SetupOperator(A)
        s.InitControl(20000, 0.0, case["rtol"], 1e8)
        st["s"] = s
    elif op == "gmres":
        s = lmp.GMRES()
        s.InitParameter(case["basis"], "RightPreconditioning")
        s.SetupPreconditioner(_jacobi_pc())
        s.SetupOperator(A)
        s.InitControl(case["maxits"], 0.0, case["rtol"], 1e8)
        st["s"] = s
    if "s" in st:
        st["s"]._ensure()  # the solver object that a program keeps over its solves
    _plat().synchronize()
    return st


def run(st):
    op = st["op"]
    if op == "lmp":
        A, x, b, w = st["A"], st["x"], st["b"], st["w"]
        r, p, q, z, d = (w[k] for k in ("r", "p", "q", "z", "d"))
        x.Zeros()
        r.CopyFrom(b)
        z.CopyFrom(r)
        z.ElementWiseMult(d)
        p.CopyFrom(z)
        rho = r.Dot(z)
        out = []
        for _ in range(st["case"]["steps"]):
            A.VectorMult(p, q)
            alpha = rho / p.Dot(q)
            x.Axpy(p, alpha)
            r.Axpy(q, -alpha)
            z.CopyFrom(r)
            z.ElementWiseMult(d)
            new = r.Dot(z)
            p.ScaleAdd(new / rho, z)
            rho = new
            out += [alpha, rho, r.Norm2()]
        return {"x": st["xt"], "r": st["wt"]["r"], "p": st["wt"]["p"], "scalars": np.array(out)}
    if op == "spmv":
        st["A"].VectorMult(st["xs"], st["x"])
        return st["xt"]
    if op == "coo":
        rows, cols, vals = st["trip"]
        dt = _np(st["case"]["dtype"])
        A = lmp.B200_CSR_lMatrix.TransformFromCOO(rows, cols, vals, st["n"], st["n"], platform=_plat(), dtype=dt)
        A.VectorMult(st["xv"], st["yv"])
        return st["yt"]
    if op == "batch":
        B = st["B"]
        B.restart()
        B.solve()
        res = B.results(st["slots"], out=st["views"])
        return {"x": st["x"], "state": np.array([r.solver_state for r in res])}
    if op == "jacobi":
        st["x"].CopyFrom(st["xs"])
        return {"x": st["xt"], "state": st["s"].Solve(st["b"], st["x"])}
    st["x"].Zeros()
    return {"x": st["xt"], "state": st["s"].Solve(st["b"], st["x"])}


# ------------------------------------------------------------------ the work a pass cannot do without
def _size(case):
    n = case["cells"]
    if case.get("kind") == "convection":
        return n * n, 5 * n * n - 4 * n
    d = case["dim"]
    return (n + 1) ** d, (3 * n + 1) ** d


def _iters(cells, sigma, rtol):
    """About how many Jacobi-PCG iterations a diffusion system takes (from recorded runs: 609 at 2D 256,
    302 at 3D 128, 685 at 3D 128 with sigma 2, all to 1e-10)."""
    return max(5.0, 2.37 * cells * (1 + 0.325 * sigma + 0.155 * sigma * sigma) * -math.log10(rtol) / 10)


def work(case):
    """Bytes: every value of the matrix once per product (its columns too where the call has no layout of its
    own for them), every vector that a step reads or writes once per step; iteration counts estimated."""
    op = case["op"]
    sv = 4 if case.get("dtype") == F32 else 8
    if op == "batch":
        by = fl = 0.0
        sb = 4 if case["mixed"] else 8
        for c in _batch_sizes(case, 0):
            n, nnz = (c + 1) ** case["dim"], (3 * c + 1) ** case["dim"]
            it = _iters(c, case["sigma"], case["rtol"])
            by += it * (nnz * sb + 10 * n * sb)
            fl += it * (2 * nnz + 12 * n)
        return {"bytes": by, "flops": fl}
    n, nnz = _size(case)
    if op == "lmp":
        return {"bytes": case["steps"] * (nnz * (sv + 4) + 12 * n * sv), "flops": case["steps"] * (2 * nnz + 12 * n)}
    if op == "spmv":
        return {"bytes": nnz * (sv + 4) + 4 * (n + 1) + 2 * n * sv, "flops": 2 * nnz}
    if op == "coo":
        return {"bytes": nnz * (8 + sv) + nnz * (4 + sv) + 4 * (n + 1) + nnz * (4 + sv) + 2 * n * sv, "flops": 2 * nnz}
    if op == "jacobi":
        return {"bytes": case["sweeps"] * (nnz * sv + 4 * n * sv), "flops": case["sweeps"] * (2 * nnz + 4 * n)}
    diff = case.get("kind") != "convection"
    it = _iters(case["cells"], case["sigma"] if diff else 0.0, case["rtol"])
    if op == "cg":
        return {"bytes": it * (nnz * 8 + 10 * n * 8), "flops": it * (2 * nnz + 12 * n)}
    if op == "mp":
        return {"bytes": it * (nnz * 4 + 10 * n * 4), "flops": it * (2 * nnz + 12 * n)}
    if op == "bicgstab":
        it *= 0.7
        return {"bytes": it * (2 * nnz * 8 + 16 * n * 8), "flops": it * (4 * nnz + 22 * n)}
    it = min(case["maxits"], 1.2 * it)
    basis = 0.5 * min(case["basis"], it)
    return {"bytes": it * (nnz * 8 + (basis + 4) * n * 8), "flops": it * (2 * nnz + 4 * basis * n)}


def tolerance(case):
    """About four times the largest difference from `exact` that 100 listed and drawn cases showed.  A solve's
    difference is that of its stopping test (it moves by as much when rounding makes it stop one iteration
    earlier or later): up to 0.2 rtol for the PCGs, 0.7 rtol for BiCGSTAB."""
    op = case["op"]
    f32 = case.get("dtype") == F32
    if op in ("spmv", "coo"):  # seen: 9e-8 and 2.9e-6; 2.5e-16 and 1.5e-14 (rows whose terms cancel)
        return {"rel": 4e-7, "max": 1.2e-5} if f32 else {"rel": 1e-15, "max": 6e-14}
    if op == "lmp":  # seen: 5.5e-15 and 4.1e-14
        return {"rel": 2.2e-14, "max": 1.6e-13}
    if op == "jacobi":  # seen: 4.9e-8 and 2.1e-7; 1.2e-16 and 5.4e-16
        return {"rel": 2e-7, "max": 1e-6} if f32 else {"rel": 5e-16, "max": 2.5e-15}
    if op in ("bicgstab", "gmres"):
        return {"rel": 3 * case["rtol"], "max": 6 * case["rtol"]}
    return {"rel": 0.8 * case["rtol"], "max": 4 * case["rtol"]}


# ------------------------------------------------------------------ the same in 64 bits, in torch
def _csr(rows, cols, vals, n):
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(rows.long(), minlength=n), 0)
    return torch.sparse_csr_tensor(rowptr, cols.long(), vals, (n, n))


def _diag(rows, cols, vals, n):
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    on = rows == cols
    d[rows[on].long()] = vals[on]
    return d


def _pcg(A, dinv, b, lengths, its=6000):
    """Jacobi-PCG on independent systems that lie one behind the other, until each stops getting better."""
    if lengths is None:
        def dot(u, v):
            return torch.dot(u, v).reshape(1)

        def wide(s):
            return s
    else:
        seg = torch.repeat_interleave(torch.arange(len(lengths), device=DEV), lengths)

        def dot(u, v):
            return torch.segment_reduce(u * v, "sum", lengths=lengths)

        def wide(s):
            return s[seg]
    x = torch.zeros_like(b)
    r = b.clone()
    z = r * dinv
    p = z.clone()
    rz = dot(r, z)
    end = 1e-28 * dot(r, r)
    for k in range(its):
        q = A @ p
        pq = dot(p, q)
        live = rz > 0 if k == 0 else live & (dot(r, r) > end)
        if k % 16 == 0 and not bool(live.any()):
            break
        alpha = torch.where(live, rz / pq, torch.zeros_like(rz))
        aw = wide(alpha)
        x += aw * p
        r -= aw * q
        z = r * dinv
        new = dot(r, z)
        p = z + wide(torch.where(live, new / rz, torch.zeros_like(rz))) * p
        rz = torch.where(live, new, rz)
    return x


def _bicgstab(A, dinv, b, its=6000):
    """Until the true residual is 1e-13 of b's norm; started again from the last x when it stalls."""
    x = torch.zeros_like(b)
    goal = 1e-13 * torch.linalg.vector_norm(b)
    done = 0
    while done < its:
        r = b - A @ x
        if torch.linalg.vector_norm(r) <= goal:
            break
        r0, p, rho = r.clone(), r.clone(), torch.dot(r, r)
        for _ in range(400):
            done += 1
            ph = p * dinv
            v = A @ ph
            alpha = rho / torch.dot(r0, v)
            s = r - alpha * v
            sh = s * dinv
            t = A @ sh
            om = torch.dot(t, s) / torch.dot(t, t)
            x = x + alpha * ph + om * sh
            r = s - om * t
            new = torch.dot(r0, r)
            if torch.linalg.vector_norm(r) <= 0.1 * goal or not torch.isfinite(new):
                break
            p = r + (new / rho) * (alpha / om) * (p - om * v)
            rho = new
    return x


def _gmres(A, dinv, b, basis, maxits, rtol):
    """Right-preconditioned GMRES(basis), a restart scaled by the last residual of the recurrence."""
    x = torch.zeros_like(b)
    first = float(torch.linalg.vector_norm(b))
    res, it = first, 0
    basis = min(basis, maxits)
    while True:
        V = [(b - A @ x) / res]
        H = np.zeros((basis + 1, basis))
        g = np.zeros(basis + 1)
        g[0] = res
        cs, sn = np.zeros(basis), np.zeros(basis)
        for j in range(basis):
            w = A @ (V[j] * dinv)
            hs = []
            for v in V:
                hj = torch.dot(w, v)
                hs.append(hj)
                w = w - hj * v
            nw = torch.linalg.vector_norm(w)
            H[:j + 2, j] = torch.stack(hs + [nw]).cpu().numpy()
            V.append(w / nw)
            for k in range(j):
                H[k, j], H[k + 1, j] = cs[k] * H[k, j] + sn[k] * H[k + 1, j], -sn[k] * H[k, j] + cs[k] * H[k + 1, j]
            rad = math.hypot(H[j, j], H[j + 1, j])
            cs[j], sn[j] = H[j, j] / rad, H[j + 1, j] / rad
            H[j, j], H[j + 1, j] = rad, 0.0
            g[j], g[j + 1] = cs[j] * g[j], -sn[j] * g[j]
            res = abs(g[j + 1])
            it += 1
            if res < rtol * first or it >= maxits:
                break
        y = np.linalg.solve(H[:j + 1, :j + 1], g[:j + 1])
        z = torch.zeros_like(b)
        for k in range(j + 1):
            z += float(y[k]) * V[k]
        x = x + z * dinv
        if res < rtol * first or it >= maxits:
            return x


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        systems = _batch_systems(case, seed)
        rows, cols, vals, bs, at = [], [], [], [], 0
        for rowptr, col, val, b in systems:
            rows.append(_rows(rowptr) + at)
            cols.append(col + at)
            vals.append(val)
            bs.append(b)
            at += b.numel()
        rows, cols, vals, b = (torch.cat(v) for v in (rows, cols, vals, bs))
        A = _csr(rows, cols, vals, at)
        dinv = 1.0 / _diag(rows, cols, vals, at)
        lengths = torch.tensor([v.numel() for v in bs], device=DEV)
        return {"x": _pcg(A, dinv, b, lengths, its=3000), "state": None}
    rows, cols, vals, b = _system(case, seed)
    n = b.numel()
    if op == "coo":
        g = _gen(seed, 1)
        torch.randperm(rows.numel(), device=DEV, generator=g)
        x = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
        vt = _torch(case["dtype"])
        return _csr(rows, cols, vals.to(vt).double(), n) @ x.to(vt).double()
    vt = _torch(case.get("dtype", F64))
    start = torch.rand(n, dtype=torch.float64, device=DEV, generator=_gen(seed, 2)).to(vt).double()
    vals, b = vals.to(vt).double(), b.to(vt).double()
    A = _csr(rows, cols, vals, n)
    if op == "spmv":
        return A @ start
    dinv = 1.0 / _diag(rows, cols, vals, n)
    if op == "jacobi":
        x = start
        for _ in range(case["sweeps"]):
            x = x + 0.8 * dinv * (b - A @ x)
        return {"x": x, "state": None}
    if op == "lmp":
        x, r = torch.zeros_like(b), b.clone()
        z = r * dinv
        p, rho, out = z.clone(), torch.dot(r, z), []
        for _ in range(case["steps"]):
            q = A @ p
            alpha = rho / torch.dot(p, q)
            x = x + alpha * p
            r = r - alpha * q
            z = r * dinv
            new = torch.dot(r, z)
            p = z + (new / rho) * p
            rho = new
            out += [alpha, rho, torch.linalg.vector_norm(r)]
        return {"x": x, "r": r, "p": p, "scalars": torch.stack(out).cpu().numpy()}
    if op == "gmres":
        return {"x": _gmres(A, dinv, b, case["basis"], case["maxits"], case["rtol"]), "state": None}
    if op == "bicgstab":
        return {"x": _bicgstab(A, dinv, b), "state": None}
    return {"x": _pcg(A, dinv, b, None), "state": None}
