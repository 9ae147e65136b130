"""The work that programs have the library do, as timed cases.

Two sorts of program stand behind them.  Most call the eigensolver: one solve
of A x = lambda B x for the smallest pairs, with everything resident on the
GPU, from batches of small 2D problems to the variable-coefficient operators
of the serving workload.  The others drive the OPS slots themselves (their own
outer iteration, the reference's front ends, a linear solver for time steps):
products with a sparse matrix, projections, linear combinations,
orthogonalisation, block CG, the projected eigenproblem.

Inputs are made on the GPU from the seed alone: finite-difference operators on
structured grids (the operators of gcge_gb300.problems, with grids that need
not be cubes) and normally distributed blocks.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gcge_gb300 as G
from gcge_gb300.problems import CSRMatrix, gcge_block_rule

F64 = torch.float64


# --------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------
def listed():
    return [
        # MatDotMultiVec on the 128 x 128 Laplacian, 20 columns: the smallest
        # call, a launch and little else
        dict(name="spmm_2d", kind="spmm", op="aniso", nx=128, ny=128, nz=1, k=20),
        # MatDotMultiVec on the 128^3 operator, a full block of 40 columns
        dict(name="spmm_3d", kind="spmm", op="diffusion", nx=128, ny=128, nz=128, k=40),
        # MultiVecQtAP: [X P W]^T A W of a Rayleigh-Ritz step in FP64, 64^3
        dict(name="qtap", kind="qtap", op="kron", nx=64, ny=64, nz=64, m=180, k=20),
        # MultiVecLinearComb: a block of Ritz vectors from the basis, 64^3
        dict(name="lincomb", kind="lincomb", op="kron", nx=64, ny=64, nz=64, m=180, k=20),
        # MultiVecOrth: a new block against a B-orthonormal basis, B with 27
        # entries per row, a grid that fills no tile evenly
        dict(name="orth", kind="orth", op="kron", nx=33, ny=33, nz=33, m=60, k=20),
        # block CG in FP32, 40 right-hand sides of a diffusion time step: the
        # inner solve's size on 128^3
        dict(name="pcg32_3d", kind="pcg", op="diffusion", nx=128, ny=128, nz=128, k=40, fp32=True),
        # block CG in FP64 through MultiLinearSolver: a diffusion time step
        # with a 27-point operator, 64^3
        dict(name="pcg64_27pt", kind="pcg", op="kron", nx=64, ny=64, nz=64, k=20, fp32=False),
        # the projected eigenproblem of a solve with nev = 100
        dict(name="eig", kind="eig", s=180),
        # one problem of a batch: anisotropic 2D Laplacian, diagonal B
        dict(name="solve_2d", kind="solve", op="aniso", nx=64, ny=65, nz=1, nev=13, b=True,
             mixed=True),
        # the 2D Laplacian, B = I, in FP64 (the default precision)
        dict(name="solve_2d_fp64", kind="solve", op="aniso", nx=128, ny=128, nz=1, nev=20, b=False,
             mixed=False),
        # generalized problem with a consistent mass matrix, 100 pairs
        dict(name="solve_mass_64", kind="solve", op="kron", nx=64, ny=64, nz=64, nev=100, b=True,
             mixed=True),
        # variable-coefficient diffusion, a large request of the serving
        # workload, 100 pairs
        dict(name="solve_diffusion_72", kind="solve", op="diffusion", nx=72, ny=72, nz=72, nev=100,
             b=True, mixed=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _grid(rng, op, most):
    """Grid sides of one operator, at most `most` points: 2D sides of the batch
    workload (40 to 220), 3D grids from 16^3 up, their sides up to 1.5 : 1."""
    if op == "aniso":
        nx = _log_int(rng, 40, 220)
        return nx, _log_int(rng, 40, max(40, min(220, most // nx))), 1
    side = _log_int(rng, 16 ** 3, most) ** (1.0 / 3.0)
    nx, ny = (max(16, int(side * rng.uniform(0.8, 1.2))) for _ in range(2))
    return nx, ny, max(16, int(side ** 3 / (nx * ny)))


def draw(rng):
    kind = rng.choice(["spmm", "qtap", "lincomb", "orth", "pcg", "pcg", "eig", "solve", "solve",
                       "solve"])
    if kind == "eig":
        return dict(kind=kind, s=_log_int(rng, 16, 400))
    op = rng.choice(["aniso", "diffusion", "kron"])
    if kind == "spmm":
        nx, ny, nz = _grid(rng, op, 128 ** 3 if op == "diffusion" else 64 ** 3)
        return dict(kind=kind, op=op, nx=nx, ny=ny, nz=nz, k=_log_int(rng, 1, 60))
    if kind in ("qtap", "lincomb"):
        nx, ny, nz = _grid(rng, op, 64 ** 3)
        return dict(kind=kind, op=op, nx=nx, ny=ny, nz=nz, m=_log_int(rng, 20, 200),
                    k=_log_int(rng, 2, 40))
    if kind == "orth":
        nx, ny, nz = _grid(rng, op, 48 ** 3)
        m = rng.choice([0, _log_int(rng, 10, 160)])
        return dict(kind=kind, op=op, nx=nx, ny=ny, nz=nz, m=m, k=_log_int(rng, 2, 40))
    if kind == "pcg":
        fp32 = rng.random() < 0.5
        nx, ny, nz = _grid(rng, op, 128 ** 3 if fp32 and op == "diffusion" else 64 ** 3)
        return dict(kind=kind, op=op, nx=nx, ny=ny, nz=nz, k=_log_int(rng, 1, 40), fp32=fp32)
    mixed = rng.random() < 0.75
    nx, ny, nz = _grid(rng, op, (64 if mixed else 40) ** 3)
    nev = _log_int(rng, 8, 64)
    return dict(kind="solve", op=op, nx=nx, ny=ny, nz=nz, nev=min(nev, nx * ny * nz // 40),
                b=op != "aniso" or rng.random() < 0.75, mixed=mixed)


# --------------------------------------------------------------------------
# Operators
# --------------------------------------------------------------------------
def _rng(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + stream)


def _uniform(seed, stream, *shape):
    return torch.rand(*shape, generator=_rng(seed, stream), device="cuda", dtype=F64)


def _normal(seed, stream, *shape):
    return torch.randn(*shape, generator=_rng(seed, stream), device="cuda", dtype=F64)


def _scale(seed):
    """A material constant between 0.5 and 2 that the seed decides."""
    return 0.5 * 4.0 ** float(_uniform(seed, 90, 1)[0])


def _stencil(dims, entries):
    """CSR arrays (row pointers, columns, values; on the GPU) of a grid operator:
    entries maps an offset (dz, dy, dx) to its coefficients, a number or a
    tensor over the grid [nz, ny, nx]; entries that leave the grid are dropped."""
    nx, ny, nz = dims
    z, y, x = (torch.arange(s, device="cuda") for s in (nz, ny, nx))
    idx = (z.view(-1, 1, 1) * ny + y.view(1, -1, 1)) * nx + x.view(1, 1, -1)
    vals, cols, keep = [], [], []
    for (dz, dy, dx) in sorted(entries):
        c = entries[(dz, dy, dx)]
        if not torch.is_tensor(c):
            c = torch.full((nz, ny, nx), c, device="cuda", dtype=F64)
        vals.append(c)
        cols.append(idx + (dz * ny + dy) * nx + dx)
        keep.append(((z + dz >= 0) & (z + dz < nz)).view(-1, 1, 1)
                    & ((y + dy >= 0) & (y + dy < ny)).view(1, -1, 1)
                    & ((x + dx >= 0) & (x + dx < nx)).view(1, 1, -1))
    n = nx * ny * nz
    vals, cols, keep = (torch.stack([t.reshape(n) for t in ts], dim=1) for ts in (vals, cols, keep))
    ptr = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    ptr[1:] = torch.cumsum(keep.sum(dim=1), 0)
    return ptr, cols[keep], vals[keep]


def _diag(d):
    i = torch.arange(d.numel() + 1, device="cuda")
    return i, i[:-1], d


def _diffusion(dims, seed):
    """Cell-centred diffusion, log-normal coefficient per cell, harmonic face
    means, Dirichlet faces; lumped mass."""
    nx, ny, nz = dims
    h = 1.0 / max(dims)
    kap = torch.exp(_normal(seed, 1, nz, ny, nx))
    diag = torch.zeros_like(kap)
    ent = {}
    for axis in range(3):
        size = kap.shape[axis]
        lo, hi = kap.narrow(axis, 0, size - 1), kap.narrow(axis, 1, size - 1)
        face = 2.0 * lo * hi / (lo + hi)
        up, down = torch.zeros_like(kap), torch.zeros_like(kap)
        up.narrow(axis, 0, size - 1).copy_(face)
        down.narrow(axis, 1, size - 1).copy_(face)
        diag += up + down
        diag.narrow(axis, 0, 1).add_(2.0 * kap.narrow(axis, 0, 1))
        diag.narrow(axis, size - 1, 1).add_(2.0 * kap.narrow(axis, size - 1, 1))
        step = [0, 0, 0]
        step[axis] = 1
        ent[tuple(step)] = -h * up
        ent[tuple(-s for s in step)] = -h * down
    ent[(0, 0, 0)] = h * diag
    return _stencil(dims, ent), _diag(h ** 3 * (1.0 + 0.1 * _uniform(seed, 2, nx * ny * nz)))


def _aniso(dims, seed):
    """Anisotropic 5-point Laplacian: -eps on x faces, -1 on y faces, eps from 1
    to 100 as the seed decides; a random diagonal mass."""
    eps = 100.0 ** float(_uniform(seed, 3, 1)[0])
    ent = {(0, 0, 0): 2.0 * eps + 2.0, (0, 0, 1): -eps, (0, 0, -1): -eps, (0, 1, 0): -1.0,
           (0, -1, 0): -1.0}
    return _stencil(dims, ent), _diag(0.5 + 1.5 * _uniform(seed, 4, dims[0] * dims[1]))


def _mass_1d(size):
    """Diagonal and off-diagonal of the 1D consistent mass on `size` points."""
    h = 1.0 / (size + 1)
    return 4.0 * h / 6.0, h / 6.0


def _kron_entries(dims):
    m = [_mass_1d(s) for s in (dims[2], dims[1], dims[0])]
    return {(dz, dy, dx): m[0][dz != 0] * m[1][dy != 0] * m[2][dx != 0]
            for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)}


def _kron(dims, seed):
    """7-point stiffness times a material constant; consistent mass M x M x M
    (27 entries per row)."""
    c = _scale(seed)
    w = [c * (s + 1) ** 2 for s in dims]
    ent = {(0, 0, 0): 2.0 * sum(w)}
    for s in (-1, 1):
        ent[(0, 0, s)], ent[(0, s, 0)], ent[(s, 0, 0)] = -w[0], -w[1], -w[2]
    return _stencil(dims, ent), _stencil(dims, _kron_entries(dims))


def _step_operator(case, seed):
    """The operator of an implicit time step, mass plus dt times stiffness,
    condition in the hundreds.  diffusion and aniso: the shifted stiffness on
    its own pattern; kron: 27 entries per row."""
    dims = (case["nx"], case["ny"], case["nz"])
    if case["op"] == "kron":
        ent = _kron_entries(dims)
        vol = math.prod(1.0 / (s + 1) for s in dims)
        dt = 20.0 * _scale(seed) / max(s + 1 for s in dims) ** 2
        w = [dt * vol * (s + 1) ** 2 for s in dims]
        ent[(0, 0, 0)] += 2.0 * sum(w)
        for s in (-1, 1):
            ent[(0, 0, s)] -= w[0]
            ent[(0, s, 0)] -= w[1]
            ent[(s, 0, 0)] -= w[2]
        return _stencil(dims, ent)
    (ptr, col, val), mass = _pencil(case, seed)
    if case["op"] == "diffusion":
        shift = 10.0 * max(dims) ** 2
    else:
        shift = 0.05 * float(val.max())
    row = torch.repeat_interleave(torch.arange(ptr.numel() - 1, device="cuda"), ptr.diff())
    return ptr, col, val + torch.where(row == col, shift * mass[2][row], 0.0)


def _pencil(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    return {"diffusion": _diffusion, "aniso": _aniso, "kron": _kron}[case["op"]](dims, seed)


def _host(m):
    ptr, col, val = m
    return CSRMatrix(ptr.numel() - 1, ptr.to(torch.int32).cpu().numpy(),
                     col.to(torch.int32).cpu().numpy(), val.cpu().numpy())


def _sparse(m):
    ptr, col, val = m
    n = ptr.numel() - 1
    return torch.sparse_csr_tensor(ptr, col, val, size=(n, n))


def _points(case):
    return case["nx"] * case["ny"] * case["nz"]


def _entries(case, mass=False):
    """Stored entries of the operator (of its mass matrix)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["op"] == "kron" and mass:
        return (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)
    if mass:
        return nx * ny * nz
    return nx * ny * nz + 2 * ((nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1))


# --------------------------------------------------------------------------
# Inputs of a call
# --------------------------------------------------------------------------
class _Ops:
    """An OPS object with its matrices and multivectors, freed together."""

    def __init__(self):
        self.ops = G.CudaOps()

    def __del__(self):
        try:
            self.ops.close()
        except Exception:
            pass

    def mat(self, m):
        return self.ops.mat(_host(m))

    def multivec(self, mat, host):
        """A multivector holding the rows of `host` (k x n) as its columns, and
        a tensor over its memory."""
        k, n = host.shape
        handle = self.ops.multivec(mat, k)
        torch.cuda.synchronize()
        t = torch.as_tensor(_Memory(self, handle, n, k), device="cuda")
        t.copy_(host)
        torch.cuda.synchronize()
        return handle, t


class _Memory:
    """The device memory of a multivector, column by column, for torch.  The
    handle points to its record: tag, rows, columns, leading dimension (32 bits
    each) and the address of column 0.  Keeps the OPS object alive."""

    class _Record(ctypes.Structure):
        _fields_ = [("tag", ctypes.c_uint32), ("nrows", ctypes.c_int), ("ncols", ctypes.c_int),
                    ("ld", ctypes.c_int), ("data", ctypes.c_void_p)]

    def __init__(self, owner, handle, n, k):
        r = self._Record.from_address(handle.value)
        if r.nrows != n or r.ncols != k or r.ld < n or not r.data:
            raise RuntimeError("multivector record has another layout")
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(k, n), typestr="<f8", data=(r.data, False),
                                             strides=(8 * r.ld, 8), version=3)


def _block(case, seed, stream, k):
    return _normal(seed, stream, k, _points(case))


def _b_apply(case, b):
    """X -> B X for blocks stored by rows (k x n)."""
    if case["op"] != "kron":
        d = b[2]
        return lambda x: x * d
    dims = (case["nx"], case["ny"], case["nz"])

    def apply(x):
        y = x.reshape(-1, dims[2], dims[1], dims[0])
        for axis, size in ((1, dims[2]), (2, dims[1]), (3, dims[0])):
            d, o = _mass_1d(size)
            t = d * y
            t.narrow(axis, 0, size - 1).add_(y.narrow(axis, 1, size - 1), alpha=o)
            t.narrow(axis, 1, size - 1).add_(y.narrow(axis, 0, size - 1), alpha=o)
            y = t
        return y.reshape(x.shape)

    return apply


def _b_orthonormal(x, apply):
    """The rows of x (k x n) B-orthonormalised by Cholesky factors, twice."""
    for _ in range(2):
        low = torch.linalg.cholesky(x @ apply(x).T)
        x = torch.linalg.solve_triangular(low, x, upper=False)
    return x


def _orth_blocks(case, seed, apply):
    """A B-orthonormal basis (m rows) and a new block of k directions that
    partly lie in its span, as the corrections of an iteration do."""
    m, k = case["m"], case["k"]
    w = _block(case, seed, 6, k)
    if m == 0:
        return None, w
    basis = _b_orthonormal(_block(case, seed, 5, m), apply)
    return basis, w + _normal(seed, 7, k, m) @ basis * 10.0


def _projected(case, seed):
    """A projected matrix as Rayleigh-Ritz meets it: Ritz values on the leading
    part, a dense block for P, and the new directions coupled to all."""
    s = case["s"]
    x = max(1, 3 * s // 4)
    ritz = torch.cumsum(0.5 + _uniform(seed, 8, s), 0)
    a = _normal(seed, 9, s, s) * 0.05
    a = a + a.T
    p = (s - x) // 2
    a[:x, :x + p] = 0.0
    a[:x + p, :x] = 0.0
    return a + torch.diag(ritz * (1.0 + 2.0 * (torch.arange(s, device="cuda") >= x)))


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def _setup_block_pcg(ops, max_iter, rate, tol):
    ops.lib.MultiLinearSolverSetup_BlockPCG(
        ctypes.c_int(max_iter), ctypes.c_double(rate), ctypes.c_double(tol), b"abs", None, None,
        None, None, None, ops.ptr)
    ops.check("MultiLinearSolverSetup_BlockPCG")
    proto = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                             ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int),
                             ctypes.c_void_p)
    return ctypes.cast(ops.ptr.contents.MultiLinearSolver, proto)


# a time step's solve: the eigensolver's cap and absolute tolerance, and a
# reduction to what FP32 resolves (some 20 steps)
PCG_ITERS, PCG_RATE, PCG_TOL = 30, 1e-5, 1e-14
PCG_STEPS = 20


def prepare(case, seed):
    kind = case["kind"]
    if kind == "eig":
        return _State(kind=kind, m=np.asfortranarray(_projected(case, seed).cpu().numpy()))
    if kind == "solve":
        a, b = _pencil(case, seed)
        nev = case["nev"]
        bs, ni, nm = gcge_block_rule(nev)
        x0 = _block(case, seed, 10, ni).cpu().numpy().T
        prep = G.Prepared(_host(a), _host(b) if case["b"] else None, nev, bs, ni, nm, X0=x0,
                          precision=G.PREC_MIXED if case["mixed"] else G.PREC_FP64)
        return _State(kind=kind, prep=prep, nev=nev)
    o = _Ops()
    k = case["k"]
    if kind == "pcg":
        mat = o.mat(_step_operator(case, seed))
        b, bt = o.multivec(mat, _block(case, seed, 11, k))
        x0, x0t = o.multivec(mat, torch.zeros_like(bt))
        x, xt = o.multivec(mat, x0t)
        s = _State(kind=kind, owner=o, ops=o.ops, mat=mat, b=b, x0=x0, x=x, xt=xt, k=k,
                   fp32=case["fp32"], two=(ctypes.c_int * 2))
        if not case["fp32"]:
            s.solver = _setup_block_pcg(o.ops, PCG_ITERS, PCG_RATE, PCG_TOL)
        return s
    a, b = _pencil(case, seed)
    if kind == "orth":
        mat = o.mat(b)
        basis, w = _orth_blocks(case, seed, _b_apply(case, b))
        src, _ = o.multivec(mat, w)
        x, xt = o.multivec(mat, w if basis is None else torch.cat([basis, w]))
        o.ops.orth_setup("mgs")
        return _State(kind=kind, owner=o, ops=o.ops, mat=mat, src=src, x=x, xt=xt, m=case["m"], k=k)
    mat = o.mat(a)
    p, pt = o.multivec(mat, _block(case, seed, 12, k))
    if kind == "spmm":
        y, yt = o.multivec(mat, torch.zeros_like(pt))
        return _State(kind=kind, owner=o, ops=o.ops, mat=mat, p=p, y=y, yt=yt, k=k)
    m = case["m"]
    q, _ = o.multivec(mat, _block(case, seed, 13, m))
    if kind == "qtap":
        ws, _ = o.multivec(mat, torch.zeros_like(pt))
        return _State(kind=kind, owner=o, ops=o.ops, mat=mat, q=q, p=p, ws=ws, m=m, k=k)
    coef = np.asfortranarray(_normal(seed, 14, m, k).cpu().numpy())
    return _State(kind=kind, owner=o, ops=o.ops, q=q, y=p, yt=pt, coef=coef, m=m, k=k)


def run(state):
    s = state
    if s.kind == "eig":
        return G.dense_eig(s.m)
    if s.kind == "solve":
        # the nev pairs asked for; the entries behind them are the iteration's
        return s.prep.solve().eval[:s.nev]
    ops, k = s.ops, s.k
    if s.kind == "spmm":
        ops.mat_dot(s.mat, s.p, s.y, (0, 0), (k, k))
        return s.yt
    if s.kind == "qtap":
        return ops.qtap("S", "N", s.q, s.mat, s.p, (0, 0), (s.m, k), s.ws)
    if s.kind == "lincomb":
        ops.linear_comb(s.q, s.y, (0, 0), (s.m, k), s.coef, s.m)
        return s.yt
    if s.kind == "orth":
        ops.axpby(1.0, s.src, 0.0, s.x, (0, s.m), (k, s.m + k))
        end = ops.orth(s.x, s.m, s.m + k, s.mat)
        return end, s.xt
    ops.axpby(1.0, s.x0, 0.0, s.x, (0, 0), (k, k))
    if not s.fp32:
        s.solver(s.mat, s.b, s.x, s.two(0, 0), s.two(k, k), ctypes.cast(ops.ptr, ctypes.c_void_p))
        ops.check("MultiLinearSolver")
        return s.xt
    it = ctypes.c_int()
    st = ops.lib.GCGE_BlockPCG(s.mat, None, ctypes.c_double(0.0), s.b, s.x, ctypes.c_int(k),
                               ctypes.c_int(PCG_ITERS), ctypes.c_double(PCG_RATE),
                               ctypes.c_double(PCG_TOL), ctypes.c_int(1), ctypes.byref(it))
    if st != G.GCGE_OK:
        raise G.GCGEError(st, "GCGE_BlockPCG")
    return s.xt.to(torch.float32)  # an FP32 solve: x holds FP32 values


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _product(case, k, v, mass=False):
    """Bytes and flops of one sparse product with k columns, v bytes a value."""
    nnz, n = _entries(case, mass), _points(case)
    return nnz * (v + 4) + 4.0 * (n + 1) + 2.0 * n * k * v, 2.0 * nnz * k


def work(case):
    kind = case["kind"]
    if kind == "eig":
        s = case["s"]
        return dict(bytes=8.0 * (2 * s * s + s), flops=9.0 * s ** 3)
    n = _points(case)
    if kind == "solve":
        # about ten outer steps per block of pairs, whatever the size: each the
        # inner solve's thirty steps, three passes of the basis in both
        # directions (projection, Ritz vectors, projected matrix)
        bs, ni, nm = gcge_block_rule(case["nev"])
        steps = 10.0 * math.ceil(case["nev"] / bs)
        v = 4 if case["mixed"] else 8
        pb, pf = _product(case, bs, v)
        if case["op"] == "kron":
            pb, pf = _product(case, bs, v, mass=True)
        basis = (ni + nm) / 2.0 + 2 * bs
        return dict(bytes=steps * (30 * (pb + 7.0 * n * bs * v) + 4 * 8.0 * n * (basis + bs)),
                    flops=steps * (30 * (pf + 10.0 * n * bs) + 8 * n * basis * bs))
    k = case["k"]
    if kind == "spmm":
        b, f = _product(case, k, 8)
        return dict(bytes=b, flops=f)
    if kind == "qtap":
        b, f = _product(case, k, 8)
        return dict(bytes=b + 8.0 * n * case["m"], flops=f + 2.0 * n * case["m"] * k)
    if kind == "lincomb":
        m = case["m"]
        return dict(bytes=8.0 * (n * (m + k) + m * k), flops=2.0 * n * m * k)
    if kind == "orth":
        m = case["m"]
        b, f = _product(case, k, 8, mass=True)
        # two projections (coefficients, update) and two factorisations
        return dict(bytes=4 * b + 8.0 * n * (4 * m + 6 * k),
                    flops=4 * f + 8.0 * n * m * k + 8.0 * n * k * k)
    v = 4 if case["fp32"] else 8
    b, f = _product(case, k, v, mass=case["op"] == "kron")
    return dict(bytes=PCG_STEPS * (b + 7.0 * n * k * v), flops=PCG_STEPS * (f + 10.0 * n * k))


# --------------------------------------------------------------------------
# The same results in 64 bits
# --------------------------------------------------------------------------
def _exact_pcg(case, seed):
    a = _sparse(_step_operator(case, seed))
    b = _block(case, seed, 11, case["k"]).T.contiguous()
    x, p = torch.zeros_like(b), torch.zeros_like(b)
    r = b.clone()
    rho = (r * r).sum(0)
    init = rho.sqrt()
    active = init > PCG_TOL
    beta = torch.zeros_like(rho)
    for _ in range(PCG_ITERS):
        if not bool(active.any()):
            break
        p = torch.where(active, r + beta * p, p)
        w = a @ p
        alpha = torch.where(active, rho / (p * w).sum(0), 0.0)
        x += alpha * p
        r -= alpha * w
        new = (r * r).sum(0)
        beta = torch.where(active, new / rho, beta)
        rho = torch.where(active, new, rho)
        active &= (rho.sqrt() > PCG_RATE * init) & (rho.sqrt() > PCG_TOL)
    return x.T.contiguous()


def _exact_solve(case, seed):
    nx, ny, nz, nev = case["nx"], case["ny"], case["nz"], case["nev"]

    def lap(size):
        i = torch.arange(1, size + 1, device="cuda", dtype=F64)
        return 4.0 * torch.sin(0.5 * math.pi * i / (size + 1)) ** 2

    if case["op"] == "kron":
        def mass(size):
            return (1.0 - lap(size) / 6.0) / (size + 1)

        sides = ((nz, (-1, 1, 1)), (ny, (1, -1, 1)), (nx, (1, 1, -1)))
        c = _scale(seed)
        num = sum((c * (s + 1) ** 2 * lap(s)).view(v) for s, v in sides)
        one = torch.ones((), device="cuda", dtype=F64)
        den = math.prod((mass(s).view(v) for s, v in sides), start=one)
        return torch.sort((num / den).reshape(-1)).values[:nev].cpu().numpy()
    if case["op"] == "aniso" and not case["b"]:
        eps = 100.0 ** float(_uniform(seed, 3, 1)[0])
        lam = (eps * lap(nx)).view(1, -1) + lap(ny).view(-1, 1)
        return torch.sort(lam.reshape(-1)).values[:nev].cpu().numpy()
    if nx * ny * nz > 5000:
        return None
    a, b = _pencil(case, seed)
    d = b[2].rsqrt()
    dense = d.view(-1, 1) * _sparse(a).to_dense() * d
    return torch.linalg.eigvalsh(dense)[:nev].cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "eig":
        # (the vectors are unique up to sign only)
        return torch.linalg.eigvalsh(_projected(case, seed)).cpu().numpy(), None
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "pcg":
        return _exact_pcg(case, seed)
    a, b = _pencil(case, seed)
    k = case["k"]
    if kind == "orth":
        apply = _b_apply(case, b)
        basis, w = _orth_blocks(case, seed, apply)
        for _ in range(2):
            if basis is not None:
                w = w - (w @ apply(basis).T) @ basis
        w = _b_orthonormal(w, apply)
        return case["m"] + k, w if basis is None else torch.cat([basis, w])
    p = _block(case, seed, 12, k)
    if kind == "spmm":
        return (_sparse(a) @ p.T.contiguous()).T.contiguous()
    q = _block(case, seed, 13, case["m"])
    if kind == "qtap":
        return (q @ (_sparse(a) @ p.T.contiguous())).cpu().numpy()
    return _normal(seed, 14, case["m"], k).T @ q
