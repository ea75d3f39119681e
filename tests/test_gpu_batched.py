"""The batched solver (FP32 Jacobi-CG inside FP64 refinement per system) against the oracle's per-system FP64 Jacobi-CG: every
system reaches the FP64 tolerance on its true residual, with a comparable
number of CG iterations."""
import numpy as np
import pytest

from sparkit_b200 import _lib, gpu, matgen
from sparkit_b200.formats import Compressed_row_matrix

pytestmark = pytest.mark.gpu


def small_batch(count=48, seed=1):
    return matgen.batched_spd_systems(count, nmin=100, nmax=3000, seed=seed)


def system(offs, rp, ci, v, s):
    a, e = offs[s], offs[s + 1]
    rows = rp[a:e + 1] - rp[a]
    return Compressed_row_matrix((e - a, e - a), rows, ci[rp[a]:rp[e]] - a, v[rp[a]:rp[e]].astype(np.float64))


def test_batched_solves_every_system(gpu_lib, oracle):
    import torch
    offs, rp, ci, v, kinds = small_batch()
    B = gpu.Batch(offs, rp, ci, v)
    n = int(offs[-1])
    b = matgen.uniform_vector(n, seed=2)
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    inner, outer, rel, conv = B.solve(bd, xd, gpu.Batch_config())
    x = xd.cpu().numpy()
    assert conv.all() and (rel < 1e-10).all()
    for s in range(len(offs) - 1):
        A = system(offs, rp, ci, v, s)
        a, e = offs[s], offs[s + 1]
        r = b[a:e] - oracle.spmv(A, x[a:e])
        assert np.linalg.norm(r) / np.linalg.norm(b[a:e]) < 1e-10, s
        if s % 8 == 0:
            _, sr = oracle.cg(A, b[a:e], np.zeros(e - a), 1e-10, 10 ** 6, 100000, left="jacobi")
            assert inner[s] <= 1.6 * sr["computed_iterations"] + 20, (s, inner[s], sr["computed_iterations"])


def test_autotune_and_graph_replay(gpu_lib):
    import torch
    offs, rp, ci, v, _ = small_batch(32, seed=3)
    B = gpu.Batch(offs, rp, ci, v)
    bd = torch.from_numpy(matgen.uniform_vector(int(offs[-1]), seed=4)).cuda()
    xd = torch.zeros_like(bd)
    g, t, ms = B.autotune(bd, xd, sample=16)
    assert g in (1, 2, 4, 8) and t in (256, 512, 1024) and (ms > 0).all()
    cfg = gpu.Batch_config(lanes_per_row=g, threads_per_cta=t)
    B.solve(bd, xd, cfg)
    x1 = xd.clone()
    xd.zero_()
    B.solve(bd, xd, cfg)  # replays the captured graph
    torch.cuda.synchronize()
    assert torch.equal(xd, x1)
    for lanes in (1, 4, 8):
        xd.zero_()
        _, _, rel, conv = B.solve(bd, xd, gpu.Batch_config(lanes_per_row=lanes, threads_per_cta=256))
        assert conv.all() and (rel < 1e-10).all()


def test_batch_rejects_coupled_systems(gpu_lib):
    offs = np.array([0, 2, 4], np.int64)
    rp = np.array([0, 1, 3, 4, 5], np.int64)
    ci = np.array([0, 1, 2, 2, 3], np.int64)  # row 1 reaches column 2 of the second system
    with pytest.raises(_lib.SkError):
        gpu.Batch(offs, rp, ci, np.ones(5, np.float32))


def test_cluster_classes_and_their_edges(gpu_lib):
    """One lane per row solves a system on a cluster of 1 to 7 CTAs by its
    size: systems at the classes' limits and one row beside them, with rows
    and slices that do not fill, an empty one, one whose columns are spread
    over the whole system (every gather crosses CTAs), and the two kinds that
    stay with the general kernel (more than 65,536 rows, a row of more than
    64 entries).  Each reaches the FP64 tolerance on its true residual."""
    import scipy.sparse as sp
    import torch
    rng = np.random.default_rng(7)

    def chain(n):
        return sp.diags([np.full(n - 1, -1.0), np.full(n, 2.5), np.full(n - 1, -1.0)], [-1, 0, 1]) if n > 1 else \
            sp.csr_matrix([[2.5]])

    mats = [chain(n) for n in (1, 31, 32, 33, 1000, 5376, 5377, 10848, 10849, 21696, 21697, 32544, 32545, 43392,
                               43393, 54240, 54241, 65088, 65089, 65536, 65537)]
    g = matgen.laplacian_2d_dirichlet(171)
    L = sp.csr_matrix((g.values(), g.col_ind(), g.row_ptr()), g.shape()) + 0.1 * sp.identity(171 * 171)
    perm = rng.permutation(171 * 171)
    mats.append(L.tocsr()[perm][:, perm])
    arrow = sp.identity(300).tolil()
    arrow[0, :70] = 0.01
    arrow[:70, 0] = 0.01
    arrow[0, 0] = 2.0
    mats += [arrow, sp.csr_matrix((0, 0)), chain(17)]
    offs, rps, cols, vals, nnz = [0], [], [], [], 0
    for m in mats:
        m = sp.csr_matrix(m).astype(np.float32)
        m.sort_indices()
        rps.append(m.indptr[:-1].astype(np.int64) + nnz)
        cols.append(m.indices.astype(np.int64) + offs[-1])
        vals.append(m.data)
        nnz += m.nnz
        offs.append(offs[-1] + m.shape[0])
    rp = np.concatenate(rps + [[nnz]])
    ci, va = np.concatenate(cols), np.concatenate(vals)
    B = gpu.Batch(np.array(offs), rp, ci, va)
    b = rng.uniform(-1, 1, offs[-1])
    bd = torch.from_numpy(b).cuda()
    full = sp.csr_matrix((va.astype(np.float64), ci, rp), (offs[-1], offs[-1]))
    for threads in (512, 1024):
        xd = torch.zeros_like(bd)
        _, _, rel, conv = B.solve(bd, xd, gpu.Batch_config(threads_per_cta=threads))
        assert conv.all() and (rel < 1e-10).all()
        r = b - full @ xd.cpu().numpy()
        for s in range(len(mats)):
            a, e = offs[s], offs[s + 1]
            assert np.linalg.norm(r[a:e]) <= 1.0001e-10 * np.linalg.norm(b[a:e]), (s, e - a)


def chains(sizes, seed):
    """Tridiagonal SPD systems of these sizes as one batch, and a right-hand side."""
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    total = int(offs[-1])
    i = np.arange(total)
    cols = np.stack([i - 1, i, i + 1], 1)
    keep = np.ones((total, 3), bool)
    keep[offs[:-1], 0] = False
    keep[offs[1:] - 1, 2] = False
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))])
    va = np.tile(np.float32([-1.0, 2.5, -1.0]), (total, 1))[keep]
    return offs, rp, cols[keep], va, np.random.default_rng(seed).uniform(-1, 1, total)


def test_clusters_start_beside_other_work(gpu_lib):
    """The CTAs of a cluster start one after another where other work holds
    SMs: every solve of systems on clusters of 2 to 7 CTAs gives the same bits,
    and the systems are solved."""
    import torch
    offs, rp, ci, va, b = chains([11000, 22000, 33000, 44000, 55000, 65200] * 8, seed=3)
    B = gpu.Batch(offs, rp, ci, va)
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    _, _, rel, conv = B.solve(bd, xd)
    first = xd.clone()
    assert conv.all() and (rel < 1e-10).all()
    other, m = torch.cuda.Stream(), torch.randn(2048, 2048, device="cuda")
    for _ in range(20):
        xd.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            for _ in range(20):
                m = torch.tanh(m @ m)
        _, _, rel, conv = B.solve(bd, xd)
        assert conv.all() and torch.equal(xd, first)


@pytest.mark.parametrize("changed", range(4))
def test_results_go_to_the_arrays_of_the_call(gpu_lib, changed):
    """Another array for any one of the four results: this call writes to it, and
    to the former one no more."""
    import ctypes

    import torch
    offs, rp, ci, va, b = chains([100, 700, 12000], seed=5)
    B = gpu.Batch(offs, rp, ci, va)
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    L, cfg = _lib.lib(), B._cfg(gpu.Batch_config())

    def solve(arrays):
        xd.zero_()
        torch.cuda.synchronize()
        res = _lib.BatchResults(*[ctypes.c_void_p(a.data_ptr()) for a in arrays])
        _lib.check(L.sk_batched_cg_solve(B.handle, ctypes.c_void_p(bd.data_ptr()), ctypes.c_void_p(xd.data_ptr()),
                                         ctypes.byref(cfg), ctypes.byref(res), None))

    types = [torch.int32, torch.int32, torch.float64, torch.int32]
    old = [torch.full((3,), -1, dtype=t, device="cuda") for t in types]
    solve(old)
    want = [a.clone() for a in old]
    new = list(old)
    new[changed] = torch.full_like(old[changed], -1)
    old[changed].fill_(-7)
    solve(new)
    for a, w in zip(new, want):
        assert torch.equal(a, w)
    assert (old[changed] == -7).all()


def test_autotune_times_a_launch_once(gpu_lib):
    """threads_per_cta does not apply to systems on clusters: the three one-lane
    variants are one launch and one time, unless a sampled system stays with
    the general kernel."""
    import torch
    for last, once in ((9000, True), (65600, False)):
        offs, rp, ci, va, b = chains([300, 5000, last], seed=6)
        B = gpu.Batch(offs, rp, ci, va)
        bd = torch.from_numpy(b).cuda()
        _, _, ms = B.autotune(bd, torch.zeros_like(bd), sample=3)
        one_lane = ms.reshape(3, 4)[:, 0]
        assert (ms > 0).all() and (np.unique(one_lane).size == 1) == once, ms


def test_no_room_for_the_sliced_copy(gpu_lib):
    """A device with room for the matrices and half of their sliced copy: the
    batch gives that half back and its systems are solved without it."""
    import gc

    import torch
    small = chains([100], seed=1)
    gpu.Batch(*small[:4]).solve(torch.from_numpy(small[4]).cuda(), torch.zeros(100, dtype=torch.float64, device="cuda"))
    offs, rp, ci, va, b = chains([60000] * 128, seed=7)
    csr, copy = 8 * ci.size + 4 * rp.size, 6 * ci.size
    gc.collect()  # no batch of another test is given back in between
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - csr - copy // 2 - (8 << 20), dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    B = gpu.Batch(offs, rp, ci, va)
    taken = before - torch.cuda.mem_get_info()[0]
    del held
    torch.cuda.empty_cache()
    assert taken <= csr + (16 << 20), (taken, csr, copy)
    bd = torch.from_numpy(b).cuda()
    _, _, rel, conv = B.solve(bd, torch.zeros_like(bd))
    assert conv.all() and (rel < 1e-10).all()
