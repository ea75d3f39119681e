"""The stencil copy of a large CSR handle on 5 or 7 diagonals (half of them when
the matrix is symmetric bit for bit): every product keeps the CSR row's bits."""
import numpy as np
import pytest

from sparkit_b200 import formats, gpu, matgen

pytestmark = pytest.mark.gpu


def grid(dims, symmetric, seed):
    """A stencil of random entries on a ragged grid, two of its pairs removed."""
    nx, ny, nz = dims
    n = nx * ny * nz
    node = np.arange(n)
    i, j, k = node % nx, (node // nx) % ny, node // (nx * ny)
    hi = [(1, i + 1 < nx), (nx, j + 1 < ny)] + ([(nx * ny, k + 1 < nz)] if nz > 1 else [])
    rng = np.random.default_rng(seed)
    rows, cols, vals = [node], [node], [rng.uniform(4, 8, n)]
    for off, ok in hi:
        a = node[ok]
        if a.size == 0:
            continue
        a = np.delete(a, [3, a.size // 2])
        v = rng.standard_normal(a.size)
        rows += [a, a + off]
        cols += [a + off, a]
        vals += [v, v if symmetric else rng.standard_normal(a.size)]
    return formats.Compressed_row_matrix.from_entries((n, n), np.concatenate(rows), np.concatenate(cols),
                                                      np.concatenate(vals))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("dims", [(331, 337, 1), (1, 409, 431), (43, 47, 53), (2, 300, 260), (96, 32, 32)])
@pytest.mark.parametrize("kind", ["symmetric", "one bit off", "nonsymmetric"])
def test_products_keep_their_bits(gpu_lib, oracle, dtype, dims, kind):
    import torch
    A = grid(dims, kind != "nonsymmetric", 3).astype(dtype)
    if kind == "one bit off":
        v = A.values()
        at = A.row_ptr()[A.shape()[0] // 3]
        v[at] = np.nextafter(v[at], dtype(np.inf))
    Ad = gpu.Device_matrix(A)
    width = 1 + 2 * sum(d > 1 for d in dims)
    assert Ad.layout() == ("stencil" if width in (5, 7) and A.size() >= 1 << 19 else "sell")
    n = A.shape()[0]
    x = matgen.uniform_vector(n, seed=5, dtype=dtype)
    x[n // 2] = np.inf  # reaches the rows that store it and no other
    x[7] = np.nan
    buf = torch.empty(n + 1, dtype=torch.float64 if dtype == np.float64 else torch.float32, device="cuda")
    for shift in (0, 1):  # aligned to 16 bytes, and not
        xd = buf[shift:shift + n]
        xd.copy_(torch.from_numpy(x))
        yd = torch.empty(n, dtype=buf.dtype, device="cuda")
        Ad.spmv(xd, yd)
        assert np.array_equal(yd.cpu().numpy(), oracle.spmv(A, x), equal_nan=True)


def test_solver_over_the_copy(gpu_lib, oracle):
    """A fused product (its dot product in the epilogue) on a grid too large
    for the one-launch solve."""
    A = matgen.laplacian_3d_dirichlet(65, 63, 66)
    n = A.shape()[0]
    b = oracle.spmv(A, matgen.uniform_vector(n, seed=2))
    Ad = gpu.Device_matrix(A)
    assert Ad.layout() == "stencil"
    x = np.zeros(n)
    s = gpu.conjugate_gradient(b, x, gpu.CGConfig(1e-10, 1000, 1000), gpu.spmv(Ad), gpu.jacobi(Ad))
    _, sr = oracle.cg(A, b, np.zeros(n), 1e-10, 1000, 1000, left="jacobi")
    assert s.converged and abs(s.computed_iterations - sr["computed_iterations"]) <= max(
        2, sr["computed_iterations"] // 50)
    assert np.linalg.norm(b - oracle.spmv(A, x)) <= 1e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("symmetric", [True, False])
def test_diagonal_copy_beside_it(gpu_lib, oracle, symmetric):
    """sk_matrix_add_diagonals on a handle with a stencil copy: its products
    stay on that copy, whose bytes the handle reports before and after, and
    every entry point keeps its bits."""
    import torch
    A = grid((43, 47, 53), symmetric, 4)
    n = A.shape()[0]
    Ad = gpu.Device_matrix(A)
    moved = n * (8 * (4 if symmetric else 7) + 2 + 16)
    assert Ad.info()["spmv_bytes"] == moved
    x = matgen.uniform_vector(n, seed=6)
    want = oracle.spmv(A, x)
    assert Ad.add_diagonals()
    assert Ad.layout() == "stencil" and Ad.info()["spmv_bytes"] == moved
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    Ad.spmv(xd, yd)
    assert np.array_equal(yd.cpu().numpy(), want)
    assert np.array_equal(gpu.multiply(Ad, x), want)
    Ad.add_f32_values()
    y32 = torch.empty(n, dtype=torch.float32, device="cuda")
    Ad.spmv_f32(xd.float(), y32)
    assert np.array_equal(y32.cpu().numpy(), oracle.spmv(A.astype(np.float32), x.astype(np.float32)))


def test_no_room_for_the_copy(gpu_lib, oracle):
    """A device with room for the handle and half of its stencil copy: the handle
    is made without it, holds nothing of it, and multiplies as before."""
    import gc

    import torch
    A = matgen.laplacian_3d_dirichlet(128)
    n = A.shape()[0]
    full = gpu.Device_matrix(A)
    assert full.layout() == "stencil"
    size, copy = full.info()["device_bytes"], n * (4 * 8 + 2) + 64 + 128
    full.close()
    gc.collect()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - size + copy // 2, dtype=torch.uint8, device="cuda")
    Ad = gpu.Device_matrix(A)
    del held
    torch.cuda.empty_cache()
    assert Ad.layout() == "sell" and Ad.info()["device_bytes"] == size - copy
    x = matgen.uniform_vector(n, seed=2)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    Ad.spmv(xd, yd)
    assert np.array_equal(yd.cpu().numpy(), oracle.spmv(A, x))
