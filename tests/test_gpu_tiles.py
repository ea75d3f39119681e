"""The panel-major copy of a skewed handle's long rows (x panels in shared
memory, partial sums added by the kernel of the short rows): short rows keep
the CSR bits, long rows stay within the split product's bars."""
import numpy as np
import pytest
import scipy.sparse as sp

from sparkit_b200 import _lib, formats, gpu, matgen

pytestmark = pytest.mark.gpu


def skewed(n, m, seed, dtype):
    """n x m: Zipf(1.5) row lengths up to min(2048, m), sorted columns."""
    rng = np.random.default_rng(seed)
    lens = np.minimum(rng.zipf(1.5, size=n), min(2048, m))
    rows = np.repeat(np.arange(n), lens)
    return formats.Compressed_row_matrix.from_entries((n, m), rows, rng.integers(0, m, rows.size),
                                                      rng.standard_normal(rows.size), dtype=dtype)


def launches(fn):
    before = _lib.launch_count()
    fn()
    return _lib.launch_count() - before


def held(A, x, y, oracle):
    S = sp.csr_matrix((A.values().astype(np.float64), A.col_ind(), A.row_ptr()), A.shape())
    ref = S @ x.astype(np.float64)
    scale = np.max(abs(S) @ np.abs(x.astype(np.float64)))
    assert np.max(np.abs(y - ref)) <= (1e-14 if x.dtype == np.float64 else 1e-6) * scale
    short = A.row_lengths() <= 32
    assert np.array_equal(y[short], oracle.spmv(A, x)[short])


@pytest.mark.parametrize("dtype,n,m", [(np.float64, 150_000, 24_576), (np.float64, 150_001, 24_577),
                                       (np.float64, 150_000, 300_007), (np.float32, 300_000, 49_153)])
def test_long_rows_by_panels(gpu_lib, oracle, dtype, n, m):
    import torch
    A = skewed(n, m, 3, dtype)
    Ad = gpu.Device_matrix(A)
    x = matgen.uniform_vector(m, seed=5, dtype=dtype)
    buf = torch.empty(m + 1, dtype=torch.float64 if dtype == np.float64 else torch.float32, device="cuda")
    for shift in (0, 1):  # aligned to 16 bytes, and not
        xd = buf[shift:shift + m]
        xd.copy_(torch.from_numpy(x))
        yd = torch.full((n,), float("nan"), dtype=buf.dtype, device="cuda")
        assert launches(lambda: Ad.spmv(xd, yd)) == 2
        y = yd.cpu().numpy()
        held(A, x, y, oracle)
    # an infinity reaches the rows that store its column and no other
    xd[m // 2] = float("inf")
    Ad.spmv(xd, yd)
    col = sp.csr_matrix((np.ones(A.size()), A.col_ind(), A.row_ptr()), A.shape())[:, m // 2].toarray().ravel() > 0
    assert np.array_equal(~np.isfinite(yd.cpu().numpy()), col)


def test_streams_and_capture(gpu_lib, oracle):
    """Products of one handle on two streams share its partial sums and give
    the bits of one alone; a captured one does not use them."""
    import torch
    A = skewed(150_000, 150_000, 4, np.float64)
    Ad = gpu.Device_matrix(A)
    xs = [torch.from_numpy(matgen.uniform_vector(150_000, seed=s)).cuda() for s in (1, 2)]
    ref = []
    for x in xs:
        y = torch.empty_like(x)
        Ad.spmv(x, y)
        ref.append(y.clone())
    ys = [torch.empty_like(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for x, y, s in zip(xs, ys, streams):
            with torch.cuda.stream(s):
                Ad.spmv(x, y)
    torch.cuda.synchronize()
    for y, r in zip(ys, ref):
        assert torch.equal(y, r)
    g = torch.cuda.CUDAGraph()
    y = torch.zeros_like(xs[0])
    with torch.cuda.graph(g):
        Ad.spmv(xs[0], y)
    g.replay()
    torch.cuda.synchronize()
    held(A, xs[0].cpu().numpy(), y.cpu().numpy(), oracle)


@pytest.mark.parametrize("dtype,n", [(np.float64, 150_000), (np.float32, 300_000)])
@pytest.mark.parametrize("spread", [1, 3])
def test_long_rows_round_no_worse_than_split(gpu_lib, dtype, n, spread):
    """The long rows' error against wider arithmetic (80 bits for FP64, 64 for
    FP32) beside that of the split product, which a captured call runs: rows
    spread over all panels, and rows crowded into a third of them.  A lane
    adds eight trees of eight entries one after another and up to six such runs,
    the split product 16 entries of a row of 2048; rows of a few hundred
    crowded entries may come 10% higher, which the bar leaves them."""
    import torch
    m = 1_000_003
    A = skewed(n, m // spread, 8, dtype)
    A = formats.Compressed_row_matrix((n, m), A.row_ptr(), A.col_ind(), A.values())
    Ad = gpu.Device_matrix(A)
    x = matgen.uniform_vector(m, seed=9, dtype=dtype)
    xd = torch.from_numpy(x).cuda()
    direct, split = torch.empty(n, dtype=xd.dtype, device="cuda"), torch.empty(n, dtype=xd.dtype, device="cuda")
    assert launches(lambda: Ad.spmv(xd, direct)) == 2
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        Ad.spmv(xd, split)
    g.replay()
    torch.cuda.synchronize()
    wide = np.longdouble if dtype == np.float64 else np.float64
    long = A.row_lengths() > 32
    terms = A.values().astype(wide) * x[A.col_ind()].astype(wide)
    exact = np.add.reduceat(terms, A.row_ptr()[:-1])  # every row holds at least one entry
    err = [np.linalg.norm((y.cpu().numpy().astype(wide) - exact)[long].astype(np.float64)) for y in (direct, split)]
    assert err[0] <= 1.1 * err[1], err


def test_where_the_copy_is_not_built(gpu_lib, oracle):
    """Few long-row entries, or a long row whose columns do not ascend: one
    launch, as before."""
    import torch
    small = skewed(40_000, 40_000, 5, np.float64)
    A = skewed(150_000, 150_000, 6, np.float64)
    i = int(np.argmax(A.row_lengths()))
    a, e = A.row_ptr()[i], A.row_ptr()[i + 1]
    ci, va = A.col_ind().copy(), A.values().copy()
    ci[a:e], va[a:e] = ci[a:e][::-1].copy(), va[a:e][::-1].copy()
    for M in (small, formats.Compressed_row_matrix(A.shape(), A.row_ptr(), ci, va)):
        Md = gpu.Device_matrix(M)
        x = matgen.uniform_vector(M.shape()[1], seed=1)
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty(M.shape()[0], dtype=torch.float64, device="cuda")
        assert launches(lambda: Md.spmv(xd, yd)) == 1
        held(M, x, yd.cpu().numpy(), oracle)
