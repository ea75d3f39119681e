// sk_tile.cu -- the panel-major copy of the long rows of a skewed CSR handle
// (tile_part_kernel and the long rows of hyb_spmv_kernel in sk_kernels.cuh).
//
// No reference counterpart: it is a second device layout of the long rows of
// Compressed_row_matrix (Compressed_row_matrix.hpp:20-132).
//
// The split product gathers x once per entry from L2 and is bound by the
// rate of those requests.  Here the columns are cut into panels of x that fit
// one CTA's shared memory, and the entries of the long rows are stored panel
// after panel, so that a CTA loads the panel it works on once and gathers
// from shared memory.  The entries a row has in one panel are a segment; the
// segments of a panel are sorted by decreasing length and packed 32 to a
// slice, a lane each, entry j of lane l at off + 32 j + l with a 16-bit column
// inside the panel.  A lane sums its segment, eight entries at a time as a
// tree; the row's partial sums are stored together in panel order and added by
// the kernel that takes the short rows.
//
// Built on the device: a search per (row, panel), a radix sort of the
// segments by (panel, decreasing length), a scan of the slices' sizes and one
// pass that writes them.
#include <climits>

#include "sk_kernels.cuh"
#include "sk_sort.cuh"

namespace sk {
namespace {

// bad = 1 unless the columns of every listed row ascend strictly
__global__ void tile_sorted_kernel(const int* __restrict__ rp, const int* __restrict__ ci,
                                   const int* __restrict__ rows, int nrows, int* bad) {
  const int lane = threadIdx.x & 31;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nrows; w += (gridDim.x * blockDim.x) >> 5) {
    const int b = rp[rows[w]], e = rp[rows[w] + 1];
    for (int k = b + 1 + lane; k < e; k += 32)
      if (ci[k] <= ci[k - 1]) *bad = 1;
  }
}

__device__ __forceinline__ int tile_lower(const int* __restrict__ ci, int b, int e, long long col) {
  while (b < e) {
    const int m = b + ((e - b) >> 1);
    if (ci[m] < col) b = m + 1;
    else e = m;
  }
  return b;
}

// Segment (row i, panel p) at i * panels + p: its first entry, whether it
// has any, and its sort key: panel, then decreasing length; empty ones last.
__global__ void tile_segments_kernel(const int* __restrict__ rp, const int* __restrict__ ci,
                                     const int* __restrict__ rows, i64 nseg, int panels, int width,
                                     int* __restrict__ start, unsigned char* __restrict__ any,
                                     unsigned* __restrict__ key) {
  for (i64 t = blockIdx.x * static_cast<i64>(blockDim.x) + threadIdx.x; t < nseg;
       t += static_cast<i64>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(t % panels), row = rows[t / panels];
    const int b = rp[row], e = rp[row + 1];
    const int s = tile_lower(ci, b, e, static_cast<long long>(p) * width);
    const int len = tile_lower(ci, s, e, static_cast<long long>(p + 1) * width) - s;
    start[t] = s;
    any[t] = len > 0;
    key[t] = len > 0 ? (static_cast<unsigned>(p) << 16) | (65535u - static_cast<unsigned>(len)) : 0xffffffffu;
  }
}

// first[p] = sorted segments before panel p, p = 0 .. panels (the last: all
// that are not empty)
__global__ void tile_panel_first_kernel(const unsigned* __restrict__ key, i64 nseg, int panels, int* first) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p <= panels; p += gridDim.x * blockDim.x) {
    const unsigned long long k = p == panels ? 0xffffffffull : static_cast<unsigned long long>(p) << 16;
    i64 b = 0, e = nseg;
    while (b < e) {
      const i64 m = b + ((e - b) >> 1);
      if (key[m] < k) b = m + 1;
      else e = m;
    }
    first[p] = static_cast<int>(b);
  }
}

// Panel of slice s and its first sorted segment; slices_of[p] = slices before
// panel p.
__device__ __forceinline__ int tile_panel_of(const int* __restrict__ slices_of, int panels, int s) {
  int b = 0, e = panels;
  while (b + 1 < e) {
    const int m = (b + e) >> 1;
    if (slices_of[m] <= s) b = m;
    else e = m;
  }
  return b;
}

// Entries (padded) of each slice: 32 times its longest segment, the first.
__global__ void tile_sizes_kernel(const unsigned* __restrict__ key, const int* __restrict__ first,
                                  const int* __restrict__ slices_of, int panels, int nslice, int* size) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nslice; s += gridDim.x * blockDim.x) {
    const int p = tile_panel_of(slices_of, panels, s);
    size[s] = 32 * static_cast<int>(65535u - (key[first[p] + 32 * (s - slices_of[p])] & 65535u));
  }
}

template <typename T>
__global__ void tile_fill_kernel(const unsigned* __restrict__ key, const int* __restrict__ order,
                                 const int* __restrict__ first, const int* __restrict__ slices_of, int panels,
                                 int nslice, int width, const int* __restrict__ start, const i64* __restrict__ out,
                                 const int* __restrict__ ci, const T* __restrict__ va, const int* __restrict__ off,
                                 unsigned short* __restrict__ len, int* __restrict__ dst,
                                 unsigned short* __restrict__ col, T* __restrict__ val) {
  const int lane = threadIdx.x & 31;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslice; s += (gridDim.x * blockDim.x) >> 5) {
    const int p = tile_panel_of(slices_of, panels, s);
    const int q = first[p] + 32 * (s - slices_of[p]) + lane;
    int n = 0, b = 0, o = -1;
    if (q < first[p + 1]) {
      n = static_cast<int>(65535u - (key[q] & 65535u));
      b = start[order[q]];
      o = static_cast<int>(out[order[q]]);
    }
    len[static_cast<i64>(s) * 32 + lane] = static_cast<unsigned short>(n);
    dst[static_cast<i64>(s) * 32 + lane] = o;
    const i64 at = static_cast<i64>(off[s]) + lane;
    for (int k = 0; k < n; ++k) {
      col[at + 32 * k] = static_cast<unsigned short>(ci[b + k] - p * width);
      val[at + 32 * k] = va[b + k];
    }
  }
}

__global__ void tile_row_first_kernel(const i64* __restrict__ out, int nrows, int panels, int* first) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= nrows; i += gridDim.x * blockDim.x)
    first[i] = static_cast<int>(out[static_cast<i64>(i) * panels]);
}

}  // namespace

sk_status build_tiles(sk_matrix A, i64 long_nnz, i64 longest, cudaStream_t st) {
  auto& C = A->csr;
  if (!C.hyb || C.hyb_nlong == 0 || long_nnz < (A->dtype == SK_F64 ? kTileMinEntries64 : kTileMinEntries32))
    return SK_OK;
  const size_t V = vbytes(A->dtype);
  // as many panels as shared memory asks for, and so many that a row's
  // segments stay short when its columns are spread: a segment is one lane's
  // chain (one panel of 2048-entry rows took 120 us however few)
  const i64 least = std::max((A->ncol * static_cast<i64>(V) + kTileSmem - 1) / kTileSmem,
                             (longest + kTileSegment - 1) / kTileSegment);
  const int width = static_cast<int>(((A->ncol + least - 1) / least + 31) / 32 * 32);
  const i64 panels = (A->ncol + width - 1) / width;
  const i64 nseg = static_cast<i64>(C.hyb_nlong) * panels;
  if (panels > 65535 || nseg > (i64(1) << 28)) return SK_OK;
  // the largest size any handle uses, per device
  const cudaError_t attr = A->dtype == SK_F64
                               ? cudaFuncSetAttribute(tile_part_kernel<double>,
                                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      static_cast<int>(kTileSmem))
                               : cudaFuncSetAttribute(tile_part_kernel<float>,
                                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      static_cast<int>(kTileSmem));
  if (attr != cudaSuccess) {
    cudaGetLastError();
    return SK_OK;
  }
  Temps tmp(st);
  sk_status s;
  int *bad = nullptr, *start = nullptr, *idx = nullptr, *idx2 = nullptr, *first = nullptr, *order = nullptr;
  unsigned *key = nullptr, *key2 = nullptr, *sorted = nullptr;
  unsigned char* any = nullptr;
  i64* out = nullptr;
  if ((s = tmp.get(&bad, 1)) != SK_OK) return s;
  SK_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), st));
  SK_LAUNCH(tile_sorted_kernel, grid_for(static_cast<i64>(C.hyb_nlong) * 32), kThreads, 0, st, C.row_ptr, C.col_ind,
            C.hyb_long, C.hyb_nlong, bad);
  int hbad = 0;
  SK_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
  SK_CUDA(cudaStreamSynchronize(st));
  if (hbad) return SK_OK;  // a row whose columns do not ascend: segments would not keep its order
  if ((s = tmp.get(&start, nseg)) != SK_OK || (s = tmp.get(&any, nseg)) != SK_OK ||
      (s = tmp.get(&key, nseg)) != SK_OK || (s = tmp.get(&key2, nseg)) != SK_OK ||
      (s = tmp.get(&idx, nseg)) != SK_OK || (s = tmp.get(&idx2, nseg)) != SK_OK ||
      (s = tmp.get(&out, nseg + 1)) != SK_OK || (s = tmp.get(&first, panels + 1)) != SK_OK)
    return s;
  SK_LAUNCH(tile_segments_kernel, grid_for(nseg), kThreads, 0, st, C.row_ptr, C.col_ind, C.hyb_long, nseg,
            static_cast<int>(panels), width, start, any, key);
  SK_CUDA(cudaGetLastError());
  if ((s = exclusive_scan(any, nseg, out, tmp, st)) != SK_OK) return s;
  if ((s = stable_radix_sort(key, key2, idx, idx2, nseg, 0xffffffffu, tmp, st, &sorted, &order)) != SK_OK) return s;
  SK_LAUNCH(tile_panel_first_kernel, ceil_div(panels + 1, kThreads), kThreads, 0, st, sorted, nseg,
            static_cast<int>(panels), first);
  std::vector<int> hfirst(static_cast<size_t>(panels) + 1), hslices(static_cast<size_t>(panels) + 1, 0);
  SK_CUDA(cudaMemcpyAsync(hfirst.data(), first, hfirst.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  SK_CUDA(cudaStreamSynchronize(st));
  for (i64 p = 0; p < panels; ++p)
    hslices[static_cast<size_t>(p) + 1] =
        hslices[static_cast<size_t>(p)] + (hfirst[static_cast<size_t>(p) + 1] - hfirst[static_cast<size_t>(p)] + 31) / 32;
  const int nslice = hslices.back(), nparts = hfirst.back();
  if (nslice == 0) return SK_OK;
  int *slices_of = nullptr, *size = nullptr, *off = nullptr;
  i64* off64 = nullptr;
  if ((s = upload_vector(A, hslices, &slices_of, st)) != SK_OK) return s;
  if ((s = tmp.get(&size, nslice)) != SK_OK || (s = tmp.get(&off64, nslice + 1)) != SK_OK) return s;
  SK_LAUNCH(tile_sizes_kernel, grid_for(nslice), kThreads, 0, st, sorted, first, slices_of, static_cast<int>(panels),
            nslice, size);
  SK_CUDA(cudaGetLastError());
  if ((s = exclusive_scan(size, nslice, off64, tmp, st)) != SK_OK) return s;
  std::vector<i64> hoff(static_cast<size_t>(nslice) + 1);
  SK_CUDA(cudaMemcpyAsync(hoff.data(), off64, hoff.size() * sizeof(i64), cudaMemcpyDeviceToHost, st));
  SK_CUDA(cudaStreamSynchronize(st));
  const i64 entries = hoff.back();
  // the padding stays small (segments of like length meet in a slice) unless
  // the panels hold few segments
  if (entries >= (i64(1) << 31) - 64 || entries > long_nnz + long_nnz / 4) return SK_OK;
  // columns that crowd into few panels make long segments after all
  for (int t = 0; t < nslice; ++t)
    if (hoff[static_cast<size_t>(t) + 1] - hoff[static_cast<size_t>(t)] > 32 * 4 * kTileSegment) return SK_OK;
  // each CTA a run of slices of about equal work: its entries, and what a
  // slice costs whatever its length
  const int grid = A->sm_count;
  constexpr double kSliceCost = 128;
  std::vector<int> unit(static_cast<size_t>(grid) + 1, nslice);
  const double total = static_cast<double>(entries) + kSliceCost * nslice;
  unit[0] = 0;
  for (int b = 1, t = 0; b < grid; ++b) {
    while (t < nslice && static_cast<double>(hoff[static_cast<size_t>(t)]) + kSliceCost * t < total * b / grid) ++t;
    unit[static_cast<size_t>(b)] = t;
  }
  void *len = nullptr, *dst = nullptr, *col = nullptr, *val = nullptr, *rowf = nullptr, *part = nullptr,
       *offp = nullptr;
  if ((s = upload_vector(A, unit, &C.tl_unit, st)) != SK_OK ||
      (s = dev_alloc(A, &offp, (nslice + 1) * sizeof(int))) != SK_OK ||
      (s = dev_alloc(A, &len, static_cast<size_t>(nslice) * 64)) != SK_OK ||
      (s = dev_alloc(A, &dst, static_cast<size_t>(nslice) * 128)) != SK_OK ||
      (s = dev_alloc(A, &col, static_cast<size_t>(entries) * 2 + 64)) != SK_OK ||
      (s = dev_alloc(A, &val, static_cast<size_t>(entries) * V + 64)) != SK_OK ||
      (s = dev_alloc(A, &rowf, (static_cast<size_t>(C.hyb_nlong) + 1) * sizeof(int))) != SK_OK ||
      (s = dev_alloc(A, &part, static_cast<size_t>(nparts) * V + 64)) != SK_OK)
    return s;
  off = static_cast<int*>(offp);
  SK_LAUNCH(narrow_i64_kernel, grid_for(nslice + 1), kThreads, 0, st, off64, nslice + 1, off);
  const int fill_grid = grid_for(static_cast<i64>(nslice) * 32);
  if (A->dtype == SK_F64)
    SK_LAUNCH(tile_fill_kernel<double>, fill_grid, kThreads, 0, st, sorted, order, first, slices_of,
              static_cast<int>(panels), nslice, width, start, out, C.col_ind, static_cast<const double*>(C.vals), off,
              static_cast<unsigned short*>(len), static_cast<int*>(dst), static_cast<unsigned short*>(col),
              static_cast<double*>(val));
  else
    SK_LAUNCH(tile_fill_kernel<float>, fill_grid, kThreads, 0, st, sorted, order, first, slices_of,
              static_cast<int>(panels), nslice, width, start, out, C.col_ind, static_cast<const float*>(C.vals), off,
              static_cast<unsigned short*>(len), static_cast<int*>(dst), static_cast<unsigned short*>(col),
              static_cast<float*>(val));
  SK_LAUNCH(tile_row_first_kernel, grid_for(C.hyb_nlong + 1), kThreads, 0, st, out, C.hyb_nlong,
            static_cast<int>(panels), static_cast<int*>(rowf));
  SK_CUDA(cudaGetLastError());
  auto* lock = new TileLock;
  if (cudaEventCreateWithFlags(&lock->used, cudaEventDisableTiming) != cudaSuccess) {
    delete lock;
    return fail(SK_CUDA_ERROR, "cudaEventCreate");
  }
  C.tl_lock = lock;
  SK_CUDA(cudaStreamSynchronize(st));
  C.tl_panels = static_cast<int>(panels);
  C.tl_width = width;
  C.tl_slices_of = slices_of;
  C.tl_off = off;
  C.tl_len = static_cast<unsigned short*>(len);
  C.tl_dst = static_cast<int*>(dst);
  C.tl_col = static_cast<unsigned short*>(col);
  C.tl_vals = val;
  C.tl_row_first = static_cast<int*>(rowf);
  C.tl_part = part;
  // the second kernel's CTAs by what its rows read: a long row its partial
  // sums, a short row its entries, each with a gather of x
  C.tl_long_frac = static_cast<double>(nparts) / (static_cast<double>(nparts) + 4.0 * static_cast<double>(A->nnz - long_nnz));
  C.tile = true;
  return SK_OK;
}

void destroy_tiles(sk_matrix A) {
  if (!A->csr.tl_lock) return;
  cudaEventDestroy(A->csr.tl_lock->used);
  delete A->csr.tl_lock;
  A->csr.tl_lock = nullptr;
}

}  // namespace sk
