"""Performance cases of the GPU path: what is timed, on which inputs, and what the results are in 64-bit arithmetic.

Every case goes through the public entry points of ``sparkit_b200.gpu`` as a user's program calls them: handles
(``Device_matrix``, preconditioners, ``Batch``, ``Net``, ``Pairs``) are made once in ``prepare``, the vectors live on the
device, and ``run`` is one product, one solve, one apply or one gradient.

The sizes are those of the repository's benchmark configurations (256^2 Poisson, 128^3 Laplacian and diffusion, the
million-row Zipf matrix, 512^2 convection-diffusion, uneven batches of 1k to 64k rows) and odd or smaller ones beside them.
"""
import math

import numpy as np
import torch

from sparkit_b200 import gpu
from sparkit_b200.formats import Compressed_row_matrix

# ------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------


def listed():
    return [
        # one product with a small operator, as an application's own loop calls it: launch latency
        dict(name="spmv_csr_small", kind="spmv", form="csr", pattern="lap2d", nx=67, ny=61, nz=1, dtype="f64"),
        # the headline product: 3-D stencil, FP64 CSR
        dict(name="spmv_csr_lap3d", kind="spmv", form="csr", pattern="lap3d", nx=128, ny=128, nz=128, dtype="f64"),
        # the skewed matrix of the format sweep: power-law row lengths, random columns
        dict(name="spmv_csr_zipf", kind="spmv", form="csr", pattern="zipf", nx=1000000, ny=1, nz=1, dtype="f64"),
        # a single-precision product of a ragged grid in the ELLPACK format
        dict(name="spmv_ell_f32", kind="spmv", form="ell", pattern="lap3d", nx=131, ny=113, nz=97, dtype="f32"),
        # a small symmetric solve: the 256^2 Poisson problem, Jacobi-CG to 1e-10
        dict(name="cg_poisson_256", kind="cg", pattern="lap2d", nx=256, ny=256, nz=1, precond="jacobi",
             tol=1e-10),
        # a large one: variable-coefficient diffusion in 3-D, plain FP64
        dict(name="cg_diffusion_128", kind="cg", pattern="grf3d", nx=128, ny=128, nz=128, precond="jacobi", tol=1e-11),
        # the same problem in mixed precision (FP32 inner CG, FP64 refinement)
        dict(name="mixed_cg_diffusion_128", kind="mixed_cg", pattern="grf3d", nx=128, ny=128, nz=128),
        # a small nonsymmetric solve: an implicit time step of upwind convection-diffusion, Jacobi-BiCGSTAB
        dict(name="bicgstab_convdiff_200", kind="bicgstab", pattern="convdiff", nx=201, ny=187, nz=1, peclet=4.0,
             shift=0.01),
        # FGMRES(30) with the two-level preconditioner on variable-coefficient convection-diffusion
        dict(name="fgmres_twolevel_512", kind="fgmres", pattern="convdiff", nx=512, ny=512, nz=1, peclet=10.0, agg=8),
        # many uneven SPD systems solved together
        dict(name="batched_1024", kind="batched", count=1024, nmin=1000, nmax=65536),
        # the learned preconditioner's apply inside FGMRES: the network's forward pass at the configured grid
        dict(name="learned_apply_512", kind="learned_apply", nx=512, ny=512),
        # one training step's loss and gradient: forward and backward on a batch of the training grid
        dict(name="learned_grad_128", kind="learned_grad", nx=128, ny=128, batch=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "cg", "cg", "mixed_cg", "bicgstab", "fgmres", "gmres", "batched",
                       "learned_apply", "learned_grad"])
    if kind == "spmv":
        pattern = rng.choice(["lap2d", "lap3d", "grf3d", "convdiff", "vec3", "zipf"])
        # 3x3 blocks for the vector problem; no ELLPACK of 2048 slots a row
        form = rng.choice({"vec3": ["csr", "bsr", "bsr"], "zipf": ["csr", "csr", "jad"]}.get(pattern, ["csr", "csr", "ell", "jad"]))
        dims = {"lap2d": (_log(rng, 24, 1200), _log(rng, 24, 1200), 1),
                "convdiff": (_log(rng, 24, 1000), _log(rng, 24, 1000), 1),
                "zipf": (_log(rng, 3000, 1000000), 1, 1)}.get(pattern)
        if dims is None:
            top = 64 if pattern == "vec3" else 128
            dims = (_log(rng, 9, top), _log(rng, 9, top), _log(rng, 9, top))
        c = dict(kind=kind, form=form, pattern=pattern, nx=dims[0], ny=dims[1], nz=dims[2],
                 dtype=rng.choice(["f64", "f64", "f32"]))
        if pattern == "convdiff":
            c["peclet"] = round(math.exp(rng.uniform(0.0, math.log(30.0))), 2)
        return c
    if kind == "cg":
        if rng.random() < 0.5:
            return dict(kind=kind, pattern="lap2d", nx=_log(rng, 40, 500), ny=_log(rng, 40, 500), nz=1,
                        precond=rng.choice(["none", "jacobi"]), tol=1e-11)
        return dict(kind=kind, pattern=rng.choice(["lap3d", "grf3d"]), nx=_log(rng, 20, 128), ny=_log(rng, 20, 128),
                    nz=_log(rng, 20, 128), precond="jacobi", tol=1e-11)
    if kind == "mixed_cg":
        return dict(kind=kind, pattern=rng.choice(["lap3d", "grf3d"]), nx=_log(rng, 24, 128), ny=_log(rng, 24, 128),
                    nz=_log(rng, 24, 128))
    if kind in ("bicgstab", "gmres"):
        return dict(kind=kind, pattern="convdiff", nx=_log(rng, 40, 260), ny=_log(rng, 40, 260), nz=1,
                    peclet=round(math.exp(rng.uniform(0.0, math.log(10.0))), 2),
                    shift=round(math.exp(rng.uniform(math.log(0.003), math.log(0.03))), 5))
    if kind == "fgmres":
        agg = rng.choice([4, 8])
        top = 256 if agg == 4 else 512
        return dict(kind=kind, pattern="convdiff", nx=agg * _log(rng, 12, top // agg), ny=agg * _log(rng, 12, top // agg),
                    nz=1, peclet=round(math.exp(rng.uniform(0.0, math.log(15.0))), 2), agg=agg)
    if kind == "batched":
        lo = _log(rng, 300, 2000)
        return dict(kind=kind, count=_log(rng, 60, 1000), nmin=lo, nmax=_log(rng, 4 * lo, 60000))
    if kind == "learned_apply":
        return dict(kind=kind, nx=8 * _log(rng, 4, 64), ny=8 * _log(rng, 4, 64))
    return dict(kind=kind, nx=8 * _log(rng, 4, 16), ny=8 * _log(rng, 4, 16), batch=rng.randint(1, 8))


# ------------------------------------------------------------------
# Matrices, made on the GPU from a seed
# ------------------------------------------------------------------
_CUDA = "cuda"
_F64 = torch.float64


def _gen(seed, salt=0):
    return torch.Generator(device=_CUDA).manual_seed((int(seed) * 7919 + salt) % (1 << 62))


def _uniform(n, seed, salt=0, dtype=_F64):
    return (torch.rand(n, dtype=_F64, device=_CUDA, generator=_gen(seed, salt)) * 2.0 - 1.0).to(dtype)


def _field(shape, sigma, corr, seed, salt):
    """A periodic Gaussian random field of standard deviation sigma and correlation length corr cells."""
    w = torch.randn(shape, dtype=_F64, device=_CUDA, generator=_gen(seed, salt))
    k2 = 0.0
    for d, s in enumerate(shape):
        k = 2.0 * math.pi * torch.fft.fftfreq(s, dtype=_F64, device=_CUDA)
        k2 = k2 + (k * k).reshape([-1 if e == d else 1 for e in range(len(shape))])
    g = torch.fft.ifftn(torch.fft.fftn(w) * torch.exp(-0.5 * k2 * corr * corr)).real
    g = g - g.mean()
    return g * (sigma / g.std())


def _neighbours(dims):
    """(offsets, inside masks) of the 5- or 7-point stencil in column order; the diagonal is in the middle."""
    nx, ny, nz = dims
    node = torch.arange(nx * ny * nz, device=_CUDA)
    i, j, k = node % nx, (node // nx) % ny, node // (nx * ny)
    lo = [(-1, i > 0), (-nx, j > 0), (-nx * ny, k > 0)][: 3 if nz > 1 else 2]
    hi = [(1, i + 1 < nx), (nx, j + 1 < ny), (nx * ny, k + 1 < nz)][: 3 if nz > 1 else 2]
    side = lo[::-1] + [(0, torch.ones_like(i, dtype=torch.bool))] + hi
    return [o for o, _ in side], [m for _, m in side]


class _Rows:
    """A square matrix as candidate entries per row: columns, values and a mask, each [rows, candidates], columns ascending."""

    def __init__(self, cols, vals, mask):
        self.cols, self.vals, self.mask = cols, vals, mask
        self.n = cols.shape[0]

    def csr(self):
        rp = torch.zeros(self.n + 1, dtype=torch.int64, device=_CUDA)
        torch.cumsum(self.mask.sum(1), 0, out=rp[1:])
        return rp, self.cols[self.mask], self.vals[self.mask]

    def times(self, x):
        """A x in the order of the columns, in 64 bits."""
        y = torch.zeros(self.n, dtype=_F64, device=_CUDA)
        for k in range(self.cols.shape[1]):
            t = self.vals[:, k].to(_F64) * x[self.cols[:, k].clamp(0, self.n - 1)]
            y += torch.where(self.mask[:, k], t, torch.zeros_like(t))
        return y


def _stencil(dims, offs, masks, vals):
    n = dims[0] * dims[1] * dims[2]
    node = torch.arange(n, device=_CUDA)
    return _Rows(torch.stack([node + o for o in offs], 1), torch.stack(vals, 1), torch.stack(masks, 1))


def _laplacian(dims, diag=None):
    offs, masks = _neighbours(dims)
    one = torch.ones(dims[0] * dims[1] * dims[2], dtype=_F64, device=_CUDA)
    d = float(len(offs) - 1) if diag is None else diag
    return _stencil(dims, offs, masks, [d * one if o == 0 else -one for o in offs])


def _diffusion(dims, seed):
    """Finite-volume diffusion, coefficients exp(g) with g of standard deviation 2 and correlation length 8 cells:
    harmonic means on the faces, Dirichlet boundary."""
    offs, masks = _neighbours(dims)
    kc = torch.exp(_field(dims[::-1], 2.0, 8.0, seed, 3)).reshape(-1)
    node = torch.arange(kc.numel(), device=_CUDA)
    face = [None if o == 0 else torch.where(m, 2.0 * kc * kc[(node + o).clamp(0, kc.numel() - 1)]
                                            / (kc + kc[(node + o).clamp(0, kc.numel() - 1)]), kc)
            for o, m in zip(offs, masks)]
    diag = sum(f for f in face if f is not None)
    return _stencil(dims, offs, masks, [diag if f is None else -f for f in face])


def _convection(nx, ny, peclet, seed, shift=0.0):
    """Upwind finite-volume convection-diffusion: diffusion exp(g), a divergence-free velocity from a random stream
    function, median cell Peclet number `peclet`, Dirichlet boundary.  With a shift, the implicit time step whose
    inverse length is `shift` times the operator's mean diagonal."""
    m = max(nx, ny)
    kc = torch.exp(_field((ny, nx), 1.0, max(m / 32.0, 1.0), seed, 5))
    psi = _field((ny + 1, nx + 1), 1.0, max(m / 8.0, 1.0), seed, 6)
    psi = psi * torch.sin(math.pi * torch.arange(ny + 1, dtype=_F64, device=_CUDA) / ny)[:, None]
    psi = psi * torch.sin(math.pi * torch.arange(nx + 1, dtype=_F64, device=_CUDA) / nx)[None, :]
    u, v = psi[1:, :] - psi[:-1, :], -(psi[:, 1:] - psi[:, :-1])
    kx = 2.0 * kc[:, :-1] * kc[:, 1:] / (kc[:, :-1] + kc[:, 1:])
    ky = 2.0 * kc[:-1, :] * kc[1:, :] / (kc[:-1, :] + kc[1:, :])
    pe = torch.cat([(u[:, 1:-1].abs() / kx).reshape(-1), (v[1:-1, :].abs() / ky).reshape(-1)])
    scale = peclet / pe.median()
    fx, fy = u[:, 1:-1] * scale, v[1:-1, :] * scale
    z = torch.zeros((ny, nx), dtype=_F64, device=_CUDA)
    diag, w, e, s, n = z.clone(), z.clone(), z.clone(), z.clone(), z.clone()
    diag[:, :-1] += kx + fx.clamp(min=0.0)
    e[:, :-1] = -kx + fx.clamp(max=0.0)
    diag[:, 1:] += kx + (-fx).clamp(min=0.0)
    w[:, 1:] = -kx + (-fx).clamp(max=0.0)
    diag[:-1, :] += ky + fy.clamp(min=0.0)
    n[:-1, :] = -ky + fy.clamp(max=0.0)
    diag[1:, :] += ky + (-fy).clamp(min=0.0)
    s[1:, :] = -ky + (-fy).clamp(max=0.0)
    diag[:, 0] += kc[:, 0]
    diag[:, -1] += kc[:, -1]
    diag[0, :] += kc[0, :]
    diag[-1, :] += kc[-1, :]
    diag = diag + shift * diag.mean()
    offs, masks = _neighbours((nx, ny, 1))
    return _stencil((nx, ny, 1), offs, masks, [t.reshape(-1) for t in (s, w, diag, e, n)])


def _vector_laplacian(dims, seed):
    """Three unknowns a cell: the Laplacian in each, and a dense 3x3 coupling U[-0.1, 0.1] in the diagonal block."""
    offs, masks = _neighbours(dims)
    cells = dims[0] * dims[1] * dims[2]
    coup = (torch.rand((cells, 3, 3), dtype=_F64, device=_CUDA, generator=_gen(seed, 7)) * 2 - 1) * 0.1
    coup[:, [0, 1, 2], [0, 1, 2]] = float(len(offs) - 1)
    cell = torch.arange(cells, device=_CUDA)[:, None].expand(cells, 3)
    comp = torch.arange(3, device=_CUDA)[None, :].expand(cells, 3)
    cols, vals, mask = [], [], []
    for o, m in zip(offs, masks):
        mm = m[:, None].expand(cells, 3)
        for c in range(3) if o == 0 else (None,):
            cols.append((3 * (cell + o) + (comp if c is None else c)).reshape(-1))
            vals.append((-torch.ones((cells, 3), dtype=_F64, device=_CUDA) if c is None else coup[:, :, c]).reshape(-1))
            mask.append(mm.reshape(-1))
    return _Rows(torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(mask, 1))


def _zipf(n, seed):
    """Row lengths Zipf(1.5) capped at 2048, columns uniform (duplicates dropped), values N(0, 1): (rows, cols, values)."""
    cap = min(2048, n // 2)
    p = torch.arange(1, 400001, dtype=_F64, device=_CUDA) ** -1.5
    cdf = torch.cumsum(p, 0) / 2.6123753486854883
    lens = (torch.searchsorted(cdf, torch.rand(n, dtype=_F64, device=_CUDA, generator=_gen(seed, 1))) + 1).clamp(max=cap)
    rows = torch.repeat_interleave(torch.arange(n, device=_CUDA), lens)
    key = torch.unique(rows * n + torch.randint(0, n, (rows.numel(),), device=_CUDA, generator=_gen(seed, 2)))
    return key // n, key % n, torch.randn(key.numel(), dtype=_F64, device=_CUDA, generator=_gen(seed, 4))


def _rows_of(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    if case["pattern"] in ("lap2d", "lap3d"):
        return _laplacian(dims)
    if case["pattern"] == "grf3d":
        return _diffusion(dims, seed)
    if case["pattern"] == "vec3":
        return _vector_laplacian(dims, seed)
    return _convection(case["nx"], case["ny"], case["peclet"], seed, case.get("shift", 0.0))


def _host_csr(n, rp, ci, va):
    return Compressed_row_matrix((n, n), rp.cpu().numpy(), ci.cpu().numpy(), va.cpu().numpy())


def _sizes(case):
    """(rows, stored entries) without building the matrix; expected ones for the random patterns."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["pattern"] == "zipf":
        cap = min(2048, nx // 2)
        k = np.arange(1, cap, dtype=np.float64)
        inside = float(np.sum(k ** -0.5)) / 2.6123753486854883
        return nx, int(nx * (inside + cap * (1.0 - float(np.sum(k ** -1.5)) / 2.6123753486854883)))
    n = nx * ny * nz
    nnz = n + 2 * ((nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1))
    return (3 * n, 3 * nnz + 6 * n) if case["pattern"] == "vec3" else (n, nnz)


# ------------------------------------------------------------------
# The network of the learned preconditioner
# ------------------------------------------------------------------
_LAYERS = [(8, 16), (16, 32), (32, 64), (64, 64), (64, 64), (64, 32), (32, 16), (16, 16), (16, 1)]


def _parameters(seed):
    """Flat FP32 parameters in layer order, weights [out][tap][in] then biases, He-initialised."""
    g = np.random.default_rng(seed + 17)
    return np.concatenate([np.concatenate([(g.standard_normal(co * 9 * ci) * math.sqrt(2.0 / (9 * ci))).astype(np.float32),
                                           (0.05 * g.standard_normal(co)).astype(np.float32)]) for ci, co in _LAYERS])


def _planes(A):
    """The coefficient planes diag, west, east, south, north and the inverse diagonal, FP32 as the preconditioner keeps them."""
    v = torch.where(A.mask, A.vals, torch.zeros_like(A.vals))
    s, w, d, e, n = (v[:, k] for k in range(5))
    return [t.to(torch.float32).to(_F64) for t in (d, w, e, s, n, 1.0 / d)]


def _forward(params, x):
    """The network on features x [batch, 8, H, W], in 64 bits."""
    from torch.nn.functional import avg_pool2d, conv2d, interpolate, relu
    w, at = [], 0
    for ci, co in _LAYERS:
        k = params[at:at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        w.append((k, params[at + co * 9 * ci:at + co * 9 * ci + co]))
        at += co * 9 * ci + co

    def conv(t, i):
        return conv2d(t, w[i][0], w[i][1], padding=1)

    e0 = relu(conv(x, 0))
    e1 = relu(conv(avg_pool2d(e0, 2), 1))
    e2 = relu(conv(avg_pool2d(e1, 2), 2))
    b3 = relu(conv(relu(conv(avg_pool2d(e2, 2), 3)), 4))
    d2 = relu(conv(interpolate(b3, scale_factor=2) + e2, 5))
    d1 = relu(conv(interpolate(d2, scale_factor=2) + e1, 6))
    return conv(relu(conv(interpolate(d1, scale_factor=2) + e0, 7)), 8)


def _features(planes, r, ny, nx):
    d, w, e, s, n, inv = planes
    rt = r * inv
    scale = torch.sqrt((rt * rt).mean())
    z = torch.zeros_like(rt)
    return torch.stack([rt / scale, w * inv, e * inv, s * inv, n * inv, z, z, z]).reshape(8, ny, nx), scale


def _pair_data(case, seed):
    """The training pairs of one instance: errors, and their residuals r = A e."""
    A = _convection(case["nx"], case["ny"], 10.0, seed)
    es = [_uniform(A.n, seed, 20 + k) for k in range(case["batch"])]
    return A, es, [A.times(e) for e in es]


# ------------------------------------------------------------------
# Batches of SPD systems
# ------------------------------------------------------------------

def _systems(case, seed):
    """Per system: 2-D or 3-D Laplacian plus a shift U[0, 0.5], sizes log-uniform (the same ones for every seed)."""
    g, size = np.random.default_rng(seed + 31), np.random.default_rng(31)
    for _ in range(case["count"]):
        n = math.exp(size.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        shift = float(g.uniform(0.0, 0.5))
        if size.integers(0, 2):
            m = max(2, int(round(n ** (1.0 / 3.0))))
            yield (m, m, m), float(np.float32(6.0 + shift))
        else:
            m = max(2, int(round(n ** 0.5)))
            yield (m, m, 1), float(np.float32(4.0 + shift))


def _batch_arrays(case, seed):
    offs, rps, cols, vals, bs, xs = [0], [], [], [], [], []
    base = 0
    for k, (dims, diag) in enumerate(_systems(case, seed)):
        A = _laplacian(dims, diag)
        rp, ci, va = A.csr()
        x = _uniform(A.n, seed, 100 + k)
        rps.append(rp[:-1] + base)
        cols.append(ci + offs[-1])
        vals.append(va.to(torch.float32))
        bs.append(A.times(x))
        xs.append(x)
        base += int(ci.numel())
        offs.append(offs[-1] + A.n)
    rps.append(torch.tensor([base], device=_CUDA))
    return np.array(offs, dtype=np.int64), torch.cat(rps), torch.cat(cols), torch.cat(vals), torch.cat(bs), torch.cat(xs)


# ------------------------------------------------------------------
# prepare, run, work, exact
# ------------------------------------------------------------------

def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else _F64


def prepare(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        if case["pattern"] == "zipf":
            rows, cols, vals = _zipf(case["nx"], seed)
            n = case["nx"]
            rp = torch.zeros(n + 1, dtype=torch.int64, device=_CUDA)
            torch.cumsum(torch.bincount(rows, minlength=n), 0, out=rp[1:])
            host = _host_csr(n, rp, cols, vals.to(_dtype(case)))
        else:
            A = _rows_of(case, seed)
            n = A.n
            rp, ci, va = A.csr()
            host = _host_csr(n, rp, ci, va.to(_dtype(case)))
        Ad = gpu.Device_matrix(host)
        if case["form"] == "ell":
            Ad = gpu.to_ellpack(Ad)
        elif case["form"] == "jad":
            Ad = gpu.to_jagged_diagonal(Ad)
        elif case["form"] == "bsr":
            Ad = gpu.to_block_sparse_row(Ad, 3, 3)
        x = _uniform(n, seed, 9, _dtype(case))
        return dict(case=case, A=Ad, x=x, y=torch.empty_like(x))
    if kind == "batched":
        offs, rp, ci, va, b, _ = _batch_arrays(case, seed)
        batch = gpu.Batch(offs, rp.cpu().numpy(), ci.cpu().numpy(), va.cpu().numpy())
        return dict(case=case, batch=batch, b=b, x=torch.zeros_like(b), cfg=gpu.Batch_config(tolerance=1e-10))
    if kind == "learned_apply":
        A = _convection(case["nx"], case["ny"], 10.0, seed)
        Ad = gpu.Device_matrix(_host_csr(A.n, *A.csr()))
        net = gpu.Net(seed=1)
        net.set_params(_parameters(seed))
        M = gpu.learned_preconditioner(Ad, net, case["nx"], case["ny"])
        r = _uniform(A.n, seed, 9)
        return dict(case=case, A=Ad, M=M, r=r, z=torch.empty_like(r))
    if kind == "learned_grad":
        A, es, rs = _pair_data(case, seed)
        Ad = gpu.Device_matrix(_host_csr(A.n, *A.csr()))
        pairs = gpu.Pairs(case["nx"], case["ny"], case["batch"], 1)
        inst = pairs.add_instance(Ad)
        for e, r in zip(es, rs):
            pairs.add(inst, r, e)
        net = gpu.Net(seed=1)
        net.set_params(_parameters(seed))
        return dict(case=case, net=net, pairs=pairs, idx=np.arange(case["batch"], dtype=np.int32))
    # the solvers: b = A x*, x* ~ U[-1, 1], from a zero guess
    A = _rows_of(case, seed)
    b = A.times(_uniform(A.n, seed, 9))
    Ad = gpu.Device_matrix(_host_csr(A.n, *A.csr()))
    M = None
    if kind == "fgmres":
        M = gpu.twolevel(Ad, gpu.jacobi(Ad), case["nx"], case["ny"], case["agg"])
    elif kind != "mixed_cg" and case.get("precond", "jacobi") == "jacobi":
        M = gpu.jacobi(Ad)
    return dict(case=case, A=Ad, M=M, b=b, x=torch.zeros_like(b))


def run(state):
    kind = state["case"]["kind"]
    if kind == "spmv":
        state["A"].spmv(state["x"], state["y"])
        return state["y"]
    if kind == "learned_apply":
        state["M"].apply(state["r"], state["z"])
        return state["z"]
    if kind == "learned_grad":
        loss, grad = state["net"].loss_grad(state["pairs"], state["idx"], 0.5)
        return dict(loss=loss, grad=grad)
    b, x = state["b"], state["x"]
    x.zero_()
    if kind == "batched":
        _, _, _, converged = state["batch"].solve(b, x, state["cfg"])
        return dict(x=x, converged=converged)
    op = gpu.spmv(state["A"])
    if kind == "cg":
        s = gpu.conjugate_gradient(b, x, gpu.CGConfig(state["case"]["tol"], 1000000, 6000), op, state["M"])
    elif kind == "mixed_cg":
        s = gpu.mixed_cg(b, x, gpu.Mixed_config(tolerance=1e-10), op)
    elif kind == "bicgstab":
        s = gpu.bicgstab(b, x, gpu.Bicgstab_config(1e-12, 6000), op, state["M"])
    elif kind == "gmres":
        s = gpu.gmres(b, x, gpu.Gmres_config(1e-11, 30, 6000), op, state["M"])
    else:
        s = gpu.fgmres(b, x, gpu.Fgmres_config(1e-11, 30, 6000), op, state["M"])
    return dict(x=x, converged=s.converged)


def work(case):
    kind = case["kind"]
    if kind == "spmv":
        # values, 4-byte indices, row pointers, x and y, each once
        n, nnz = _sizes(case)
        v = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=nnz * (v + 4) + 4 * (n + 1) + 2 * n * v, flops=2 * nnz)
    if kind == "batched":
        # each system's matrix and right-hand side read once, its solution written once
        n = case["count"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        return dict(bytes=int(n * (6 * 8 + 4 + 16)), flops=int(n * 12))
    if kind in ("learned_apply", "learned_grad"):
        p = case["nx"] * case["ny"] * case.get("batch", 1)
        level = [0, 1, 2, 3, 3, 2, 1, 0, 0]
        f = sum(18 * ci * co * p / 4 ** lv for (ci, co), lv in zip(_LAYERS, level))
        return dict(bytes=int(p * (16 + 16)), flops=int(f * (3 if kind == "learned_grad" else 1)))
    # a solve: the matrix and b read once, x written once, whatever the method does in between
    n, nnz = _sizes(case)
    return dict(bytes=nnz * 12 + 4 * (n + 1) + 2 * n * 8, flops=2 * nnz)


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        x = _uniform(_sizes(case)[0], seed, 9, _dtype(case)).to(_F64)
        if case["pattern"] == "zipf":
            rows, cols, vals = _zipf(case["nx"], seed)
            return torch.zeros_like(x).index_add_(0, rows, vals.to(_dtype(case)).to(_F64) * x[cols])
        A = _rows_of(case, seed)
        A.vals = A.vals.to(_dtype(case)).to(_F64)
        return A.times(x)
    if kind == "batched":
        return dict(x=_batch_arrays(case, seed)[5], converged=None)
    if kind in ("learned_apply", "learned_grad"):
        params = torch.from_numpy(_parameters(seed)).to(_CUDA).to(_F64)
        ny, nx = case["ny"], case["nx"]
        if kind == "learned_apply":
            A = _convection(nx, ny, 10.0, seed)
            x, s = _features(_planes(A), _uniform(A.n, seed, 9), ny, nx)
            return s * _forward(params, x[None]).reshape(-1)
        A, es, rs = _pair_data(case, seed)
        planes = _planes(A)
        params.requires_grad_(True)
        S = _stencil((nx, ny, 1), *_neighbours((nx, ny, 1)), [planes[k] for k in (3, 1, 0, 2, 4)])
        loss = 0.0
        for e, r in zip(es, rs):
            x, s = _features(planes, r, ny, nx)
            dif = _forward(params, x[None]).reshape(-1) - e / s
            loss = loss + (S.times(dif) ** 2).sum() / ((r / s) ** 2).sum() + 0.5 * (dif ** 2).sum() / ((e / s) ** 2).sum()
        loss = loss / len(es)
        grad, = torch.autograd.grad(loss, params)
        return dict(loss=float(loss.detach()), grad=grad.to(torch.float64))
    # the solvers: the right-hand side was made from this solution
    return dict(x=_uniform(_sizes(case)[0], seed, 9), converged=None)
