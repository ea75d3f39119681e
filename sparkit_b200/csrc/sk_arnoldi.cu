// sk_arnoldi.cu -- the modified Gram-Schmidt of one Arnoldi step of
// GMRES(m) / FGMRES(m) as one cooperative launch.
//
// The reference orthogonalizes w = A z_j against v_0 .. v_j one vector at
// a time (fgmres.hpp:259-281, gmres.hpp:259-281): h_ij = <v_i, w>, w -= h_ij
// v_i, and then h_{j+1,j} = ||w||, v_{j+1} = w / h_{j+1,j} (:283-285,
// scale_vector :403-408).  As separate launches that is j + 1 passes each
// reading and writing w.  Here each CTA keeps its rows of w in shared
// memory for the whole step, so w is read once and written once, each v_i
// is read once, and each h is one grid-wide sum behind a bounded grid
// barrier.  The arithmetic of every element is that of the per-vector
// kernels (OpFgMgs, OpFgScale: w - h v in the value type, dot terms summed
// in double); only the order in which the dot products' partial sums meet
// differs.
#include <algorithm>
#include <climits>

#include "sk_arnoldi.cuh"
#include "sk_gridsum.cuh"

namespace sk {
namespace {

constexpr int kAT = 512;  // threads per CTA (two CTAs per SM where w fits)
constexpr int kAW = kAT / 32;

__device__ __forceinline__ unsigned long long arn_ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long arn_now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits (one thread) until `target` arrivals were counted; false when the
// wait ran out here or in another CTA (the error word is set).
__device__ __forceinline__ bool arn_wait(const unsigned long long* arrived, unsigned long long target, int* err,
                                         unsigned long long wait_ns) {
  unsigned long long t0 = 0;
  for (unsigned spins = 0; arn_ld_acquire(arrived) < target; ++spins) {
    if ((spins & 255u) == 255u) {
      if (*reinterpret_cast<volatile int*>(err) != 0) return false;
      const unsigned long long t = arn_now_ns();
      if (t0 == 0) {
        t0 = t;
      } else if (t - t0 > wait_ns) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
  return true;
}

// Barrier number `epoch` (from 1) of this launch: passed when the arrival
// counter reaches epoch * gridDim.x (+ bias, which only the timeout tests
// set).  False when a wait ran out here or in another CTA (the error word
// is set); the caller then returns.
__device__ bool arn_barrier(ArnoldiSync* s, unsigned& epoch, unsigned long long wait_ns, unsigned bias) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    epoch += 1;
    const unsigned long long target = static_cast<unsigned long long>(epoch) * gridDim.x + bias;
    asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&s->arrived) : "memory");
    s_ok = arn_wait(&s->arrived, target, &s->err, wait_ns);
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ double arn_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The grid-wide sum of v, the same bits in every thread of every CTA: a
// block tree, one slot per CTA, a barrier, then every CTA sums the slots in
// CTA order with the same tree.  Consecutive sums alternate slot sets.
__device__ bool arn_allreduce(double& v, double* slots, int set, ArnoldiSync* s, unsigned& epoch,
                              unsigned long long wait_ns, unsigned bias) {
  __shared__ double s_part[kAW];
  __shared__ double s_tot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  v = arn_warp_sum(v);
  if (lane == 0) s_part[warp] = v;
  __syncthreads();
  double* slot = slots + static_cast<size_t>(set) * gridDim.x;
  if (warp == 0) {
    double t = arn_warp_sum(lane < kAW ? s_part[lane] : 0.0);
    if (lane == 0) slot[blockIdx.x] = t;
  }
  if (!arn_barrier(s, epoch, wait_ns, bias)) return false;
  double t = threadIdx.x < gridDim.x ? __ldcg(slot + threadIdx.x) : 0.0;
  t = arn_warp_sum(t);
  if (lane == 0) s_part[warp] = t;
  __syncthreads();
  if (warp == 0) {
    t = arn_warp_sum(lane < kAW ? s_part[lane] : 0.0);
    if (lane == 0) s_tot = t;
  }
  __syncthreads();
  v = s_tot;
  return true;
}

template <typename T>
__global__ void __launch_bounds__(kAT, 2) arnoldi_mgs_kernel(ArnoldiArgs<T> a) {
  extern __shared__ __align__(16) unsigned char arn_smem[];
  T* wt = reinterpret_cast<T*>(arn_smem);
  if (solve_done(a.sc)) return;  // the same flag for every CTA
  const i64 r0 = static_cast<i64>(blockIdx.x) * a.rows_per_cta;
  const i64 r1 = a.n < r0 + a.rows_per_cta ? a.n : r0 + a.rows_per_cta;
  const int cnt = r1 > r0 ? static_cast<int>(r1 - r0) : 0;
  for (int k = threadIdx.x; k < cnt; k += kAT) wt[k] = a.w[r0 + k];
  __syncthreads();
  unsigned epoch = 0;
  double hd = *a.hcol;  // h_{0j}, from the product's epilogue
  for (int i = 0; i <= a.j; ++i) {
    // w -= h_ij v_i; then h_{i+1,j} = <v_{i+1}, w>, or ||w|| at i = j
    const T h = static_cast<T>(hd);
    const T* vi = a.V + static_cast<i64>(i) * a.ldv + r0;
    const T* vn = i < a.j ? a.V + static_cast<i64>(i + 1) * a.ldv + r0 : nullptr;
    double red = 0.0;
    for (int k = threadIdx.x; k < cnt; k += kAT) {
      const T wk = sub(wt[k], mul(h, vi[k]));
      wt[k] = wk;
      red += static_cast<double>(mul(vn ? vn[k] : wk, wk));
    }
    if (!arn_allreduce(red, a.slots, i & 1, a.sync, epoch, a.wait_ns, a.bias)) return;
    const T d = static_cast<T>(red);
    const T hn = vn ? d : sqrt(d);
    hd = static_cast<double>(hn);
    if (blockIdx.x == 0 && threadIdx.x == 0) a.hcol[i + 1] = hd;
  }
  // v_{j+1} = w / h_{j+1,j}, skipped when h_{j+1,j} is not positive
  const T h = static_cast<T>(hd);
  const bool scale = h > T(0);
  const T f = a.divide ? h : T(1) / h;
  for (int k = threadIdx.x; k < cnt; k += kAT) {
    const T wk = wt[k];
    a.w[r0 + k] = scale ? (a.divide ? dvd(wk, f) : mul(wk, f)) : wk;
  }
}

template <typename T>
int arnoldi_grid(const sk_matrix_s* A, i64 n, size_t* smem_out, i64* rows_out) {
  if (n <= 0 || n > INT_MAX) return 0;
  int coop = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, A->device) != cudaSuccess || !coop) return 0;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, A->device) != cudaSuccess) return 0;
  // two CTAs per SM when both fit (twice the warps and half the rows per
  // thread to hide the loads of each basis vector), else one
  for (int per : {2, 1}) {
    const int grid = static_cast<int>(std::min<i64>(static_cast<i64>(per) * A->sm_count, (n + kAT - 1) / kAT));
    const i64 rows = (n + grid - 1) / grid;
    const size_t smem = static_cast<size_t>(rows) * sizeof(T);
    if (smem + 2048 > static_cast<size_t>(optin) || grid > kAT) continue;  // w does not fit on chip
    // The attribute is process-wide: it is always set to the largest size
    // any plan can use, so a plan made on another thread never lowers it
    // below this plan's size between this call and the launch.
    if (cudaFuncSetAttribute(arnoldi_mgs_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - 2048) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, arnoldi_mgs_kernel<T>, kAT, smem) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (per_sm < 1 || grid > per_sm * A->sm_count) continue;
    *smem_out = smem;
    *rows_out = rows;
    return grid;
  }
  return 0;
}

// ------------------------------------------------------------------
// The same step behind two grid-wide sums instead of j + 2.
//
// What bounds the kernel above is its j + 2 dependent sums, 3 us each.  The
// coefficients of modified Gram-Schmidt, h_i = <v_i, w - sum_{k<i} h_k v_k>,
// are the solution of (I + L) h = c with c = V^T w and L the strictly lower
// triangle of V^T V (Swirydowicz, Langou, Ananthan, Yang, Thomas, "Low
// synchronization Gram-Schmidt and generalized minimal residual algorithms",
// Numer. Linear Algebra Appl. 28, 2021): the same projector, product by
// product, with the same loss of orthogonality.  So one pass over V takes
// c and the new row of L (<v_j, v_k>, k < j) in one exchange of 2j + 1 sums,
// h = (I + L)^-1 c comes from the inverse kept in `tri` and one row more, and
// a second pass (L2 and L1 hold it) takes w -= h_i v_i vector after vector in
// the element arithmetic of OpFgMgs; the second exchange is the norm's.
//
// Layout: one 1024-thread CTA per SM holds its rows of w and v_j in shared
// memory; pass 1 gives each warp one basis vector (several warps share one
// while there are fewer than 32), four 16-byte loads a lane in flight.
// (Keeping pass 1's vectors on chip for pass 2 changed nothing: L2 holds them.)
// The step's Givens rotations run in its tail, on one thread of CTA 0, instead
// of a kernel of their own (6.5 us).
//
// GMRES(30), 205 x 256 convection-diffusion: 50.7 ms with the kernel above and
// its rotations, 17.2 so; FGMRES(30) with the two-level preconditioner at
// 512^2: 96.9 and 56.0 ms (all else as it was).
// ------------------------------------------------------------------
constexpr int kLT = 1024;
constexpr int kLW = kLT / 32;
constexpr int kLMax = kArnLowCols;  // columns of one cycle: restart lengths above go on with the kernel above
constexpr int kLGrid = kArnLowGrid;

template <typename T>
struct Vec16;
template <>
struct Vec16<double> {
  static constexpr int kW = 2;
  double2 v;
  __device__ void load(const double* p) { v = *reinterpret_cast<const double2*>(p); }
  __device__ double get(int k) const { return k == 0 ? v.x : v.y; }
};
template <>
struct Vec16<float> {
  static constexpr int kW = 4;
  float4 v;
  __device__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ float get(int k) const { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
};

// apply_givens_rotations (fgmres.hpp:287-337), record_residual (:340-346) and
// check_convergence (:349-356) of column j by one thread, in the value type G
// and the arithmetic of FgGivens: h[0 .. j] and hn = h_{j+1,j}, the earlier
// rotations from shared memory.
template <typename G, typename T>
__device__ void arn_givens(ArnoldiArgs<T> const& a, const double* h, double hn, const double* cs_, const double* sn_) {
  Scalars* sc = a.sc_out;
  const int j = a.j, um1 = a.m + 1;
  const int hon = sc->hist_on;
  const long long it = sc->iters, hl = sc->hist_len;
  const double bnorm = sc->bnorm, tol = sc->tol;
  const double g0 = a.sm.g[j], g1 = a.sm.g[j + 1];
  double* H = a.sm.H + static_cast<i64>(j) * um1;
  G hi = static_cast<G>(h[0]);
  for (int i = 0; i < j; ++i) {
    const G cs = static_cast<G>(cs_[i]), sn = static_cast<G>(sn_[i]), hi1 = static_cast<G>(h[i + 1]);
    H[i] = static_cast<double>(add(mul(cs, hi), mul(sn, hi1)));
    hi = add(mul(-sn, hi), mul(cs, hi1));
  }
  const G aa = hi, bb = static_cast<G>(hn);
  G cs, sn;
  if (bb == G(0)) {
    cs = G(1);
    sn = G(0);
  } else if (aa == G(0)) {
    cs = G(0);
    sn = G(1);
  } else {
    const G rr = sqrt(add(mul(aa, aa), mul(bb, bb)));
    cs = dvd(aa, rr);
    sn = dvd(bb, rr);
  }
  a.sm.cs[j] = static_cast<double>(cs);
  a.sm.sn[j] = static_cast<double>(sn);
  H[j] = static_cast<double>(add(mul(cs, aa), mul(sn, bb)));
  H[j + 1] = 0.0;
  const G gj = static_cast<G>(g0), gj1 = static_cast<G>(g1);
  const double gn = static_cast<double>(add(mul(-sn, gj), mul(cs, gj1)));
  a.sm.g[j + 1] = gn;
  a.sm.g[j] = static_cast<double>(add(mul(cs, gj), mul(sn, gj1)));
  sc->iters = it + 1;
  sc->jfinal = j;
  const G absres = fabs(static_cast<G>(gn));
  sc->rnorm = static_cast<double>(absres);
  if (hon) {
    a.hist[hl] = static_cast<double>(absres);
    sc->hist_len = hl + 1;
  }
  if (absres / static_cast<G>(bnorm) < static_cast<G>(tol)) {
    sc->converged = 1;
    sc->done = 1;
  }
}

template <typename T>
__global__ void __launch_bounds__(kLT, 1) arnoldi_low_kernel(ArnoldiArgs<T> a) {
  extern __shared__ __align__(16) unsigned char arn_smem[];
  __shared__ double s_part[kLW][2];        // pass 1: per task {<v_i, w>, <v_i, v_j>}
  __shared__ double s_tot[2 * kLMax];      // the sums, in every CTA
  __shared__ double s_h[kLMax + 1];
  __shared__ double s_rot[2][kLMax];       // CTA 0: the earlier rotations
  __shared__ double s_tri[kLMax * (kLMax - 1) / 2 + 1];  // rows 1 .. j - 1 of (I + L)^-1 below the diagonal
  constexpr int W = Vec16<T>::kW;
  if (solve_done(a.sc)) return;  // the same flag for every CTA
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = a.j, grid = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
  const i64 r0 = static_cast<i64>(me) * a.rows_per_cta;
  const i64 r1 = a.n < r0 + a.rows_per_cta ? a.n : r0 + a.rows_per_cta;
  const int cnt = r1 > r0 ? static_cast<int>(r1 - r0) : 0;
  T* wt = reinterpret_cast<T*>(arn_smem);
  T* vt = wt + a.rows_per_cta;  // v_j (rows_per_cta is a multiple of 32)
  const unsigned tag = a.sync->step + 1;  // CTA 0 advances it after the last sum of this launch
  const GridWait wait{&a.sync->err, a.wait_ns, a.bias};
  {
    const T* vj = a.V + static_cast<i64>(j) * a.ldv + r0;
    for (int k = tid; k < cnt; k += kLT) {
      wt[k] = a.w[r0 + k];
      vt[k] = vj[k];
    }
    const int tri = j * (j - 1) / 2;  // rows below j, packed
    for (int k = tid; k < tri; k += kLT) s_tri[k] = a.tri[k];
    if (me == 0 && tid < j) {
      s_rot[0][tid] = a.sm.cs[tid];
      s_rot[1][tid] = a.sm.sn[tid];
    }
  }
  __syncthreads();
  // pass 1: task t = (vector i = t % (j + 1), segment t / (j + 1) of the rows)
  const int nvec = j + 1;
  const int segs = nvec >= kLW ? 1 : kLW / nvec;
  const int seglen = ((cnt + segs - 1) / segs + 4 * W - 1) / (4 * W) * (4 * W);
  const int nv = 2 * j + 1;  // the sums: c_0 .. c_j, then l_0 .. l_{j-1}
  for (int t0 = 0; t0 < nvec * segs; t0 += kLW) {
    const int t = t0 + warp;
    if (t < nvec * segs) {
      const int i = t % nvec;
      const int b = min(cnt, (t / nvec) * seglen), e = min(cnt, b + seglen);
      double dw = 0.0, dv = 0.0;
      if (i < j) {
        const T* vi = a.V + static_cast<i64>(i) * a.ldv + r0;
        const int full = b + (e - b) / W * W;
        int k = b + lane * W;
        for (; k + 3 * 32 * W < full; k += 4 * 32 * W) {
          Vec16<T> x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u].load(vi + k + u * 32 * W);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            Vec16<T> y, z;
            y.load(wt + k + u * 32 * W);
            z.load(vt + k + u * 32 * W);
#pragma unroll
            for (int c = 0; c < W; ++c) {
              dw += static_cast<double>(mul(x[u].get(c), y.get(c)));
              dv += static_cast<double>(mul(x[u].get(c), z.get(c)));
            }
          }
        }
        for (; k < full; k += 32 * W) {
          Vec16<T> x, y, z;
          x.load(vi + k);
          y.load(wt + k);
          z.load(vt + k);
#pragma unroll
          for (int c = 0; c < W; ++c) {
            dw += static_cast<double>(mul(x.get(c), y.get(c)));
            dv += static_cast<double>(mul(x.get(c), z.get(c)));
          }
        }
        for (int q = full + lane; q < e; q += 32) {
          dw += static_cast<double>(mul(vi[q], wt[q]));
          dv += static_cast<double>(mul(vi[q], vt[q]));
        }
      } else {
        for (int q = b + lane; q < e; q += 32) dw += static_cast<double>(mul(vt[q], wt[q]));
      }
      dw = arn_warp_sum(dw);
      dv = arn_warp_sum(dv);
      if (lane == 0) {
        if (segs == 1) {  // more vectors than warps: straight to the vector's own place
          s_tot[i] = dw;
          if (i < j) s_tot[nvec + i] = dv;
        } else {
          s_part[t][0] = dw;
          s_part[t][1] = dv;
        }
      }
    }
  }
  __syncthreads();
  // each sum's partials go to its own CTA, which adds them in CTA order and
  // sends the total to every CTA
  if (tid < nv) {
    const int i = tid < nvec ? tid : tid - nvec, which = tid < nvec ? 0 : 1;
    double p = 0.0;
    if (segs == 1) {
      p = s_tot[tid];
    } else {
      for (int sg = 0; sg < segs; ++sg) p += s_part[sg * nvec + i][which];
    }
    mail_send(a.box1 + static_cast<size_t>(tid) * kLGrid + me, p, tag);
  }
  bool ok = true;
  for (int v = me + warp * grid; v < nv; v += kLW * grid) {
    double p[kLGrid / 32];
    ok = mail_wait<kLGrid / 32>(a.box1 + static_cast<size_t>(v) * kLGrid + lane, 32, (grid - lane + 31) / 32, tag,
                                wait, p) && ok;
    double t = p[0];
#pragma unroll
    for (int q = 1; q < kLGrid / 32; ++q) t += p[q];
    t = arn_warp_sum(t);
    if (__all_sync(0xffffffffu, ok))
      for (int q = lane; q < grid; q += 32) mail_send(a.box2 + static_cast<size_t>(q) * (2 * kLMax) + v, t, tag);
  }
  double tot[1] = {0.0};
  if (ok && tid < nv) ok = mail_wait<1>(a.box2 + static_cast<size_t>(me) * (2 * kLMax) + tid, 0, 1, tag, wait, tot);
  if (__syncthreads_or(!ok)) return;  // s_tot's partials read above
  if (tid < nv) s_tot[tid] = tot[0];
  __syncthreads();
  // h = (I + L)^-1 c: rows below j from `tri`, row j from the rows above it
  for (int i = warp; i < j; i += kLW) {
    double t = 0.0;
    for (int k = lane; k < i; k += 32) t += s_tri[i * (i - 1) / 2 + k] * s_tot[k];
    t = arn_warp_sum(t);
    if (lane == 0) s_h[i] = s_tot[i] + t;
  }
  __syncthreads();
  if (warp == 0) {
    double t = 0.0;
    for (int k = lane; k < j; k += 32) t += s_tot[nvec + k] * s_h[k];
    t = arn_warp_sum(t);
    if (lane == 0) s_h[j] = s_tot[j] - t;
  }
  __syncthreads();
  // pass 2: w -= h_i v_i in order, from the last rows (still in cache) up
  double red = 0.0;
  for (int k = cnt - 1 - tid; k >= 0; k -= kLT) {
    const T* vk = a.V + r0 + k;
    T wk = wt[k];
    int i = 0;
    for (; i + 8 <= j; i += 8) {
      T x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = vk[static_cast<i64>(i + u) * a.ldv];
#pragma unroll
      for (int u = 0; u < 8; ++u) wk = sub(wk, mul(static_cast<T>(s_h[i + u]), x[u]));
    }
    {
      T x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i + u < j) x[u] = vk[static_cast<i64>(i + u) * a.ldv];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i + u < j) wk = sub(wk, mul(static_cast<T>(s_h[i + u]), x[u]));
    }
    wk = sub(wk, mul(static_cast<T>(s_h[j]), vt[k]));
    wt[k] = wk;
    red += static_cast<double>(mul(wk, wk));
  }
  red = arn_warp_sum(red);
  if (lane == 0) s_part[warp][0] = red;
  __syncthreads();
  // one slot per CTA and an arrival, all in warp 0 (a mailbox exchange, which
  // every CTA would poll in every other's stead, is 1 us slower)
  double nrm = 0.0;
  if (warp == 0) {
    const double part = arn_warp_sum(s_part[lane][0]);
    double* slot = a.slots + static_cast<size_t>(tag & 1) * 512;
    if (lane == 0) {
      __stcg(slot + me, part);
      asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&a.sync->low_arrived)
                   : "memory");
      ok = arn_wait(&a.sync->low_arrived, static_cast<unsigned long long>(tag) * grid + a.bias, &a.sync->err,
                    a.wait_ns);
    }
    __syncwarp();
    double p[kLGrid / 32];
#pragma unroll
    for (int q = 0; q < kLGrid / 32; ++q) p[q] = lane + 32 * q < grid ? __ldcg(slot + lane + 32 * q) : 0.0;
#pragma unroll
    for (int q = 0; q < kLGrid / 32; ++q) nrm += p[q];
    nrm = arn_warp_sum(nrm);
    if (lane == 0) s_tot[0] = nrm;
  }
  // while the norm travels: row j of (I + L)^-1
  if (me == 0 && tid >= kLT / 2 && tid - kLT / 2 < j) {
    const int k = tid - kLT / 2;
    double t = s_tot[nvec + k];  // (s_tot[0] is not read here)
    for (int i = k + 1; i < j; ++i) t += s_tot[nvec + i] * s_tri[i * (i - 1) / 2 + k];
    a.tri[j * (j - 1) / 2 + k] = -t;
  }
  if (__syncthreads_or(!ok)) return;
  nrm = s_tot[0];
  const T h = sqrt(static_cast<T>(nrm));
  // v_{j+1} = w / h_{j+1,j}, skipped when h_{j+1,j} is not positive
  const bool scale = h > T(0);
  const T f = a.divide ? h : T(1) / h;
  for (int k = cnt - 1 - tid; k >= 0; k -= kLT) {
    const T wk = wt[k];
    a.w[r0 + k] = scale ? (a.divide ? dvd(wk, f) : mul(wk, f)) : wk;
  }
  if (me == 0 && tid == kLT - 1) {
    for (int i = 0; i <= j; ++i) s_h[i] = static_cast<double>(static_cast<T>(s_h[i]));
    if (a.hess64)
      arn_givens<double>(a, s_h, static_cast<double>(h), s_rot[0], s_rot[1]);
    else
      arn_givens<T>(a, s_h, static_cast<double>(h), s_rot[0], s_rot[1]);
    a.sync->step = tag;
  }
}

// One CTA per SM whose shared memory holds its rows of w and v_j.
template <typename T>
bool arnoldi_low_plan(const sk_matrix_s* A, i64 n, ArnoldiPlan* p) {
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, A->device) != cudaSuccess) return false;
  const int grid = static_cast<int>(
      std::min<i64>(std::min(A->sm_count, kLGrid), std::max<i64>(1, (n + kArnLowRows - 1) / kArnLowRows)));
  const i64 rows = ((n + grid - 1) / grid + 31) / 32 * 32;
  const size_t smem = static_cast<size_t>(rows) * 2 * sizeof(T);
  const size_t fixed = sizeof(double) * (kLMax * (kLMax - 1) / 2 + 1 + 5 * kLMax + 1 + 2 * kLW) + 1024;
  if (smem + fixed > static_cast<size_t>(optin)) return false;
  int per_sm = 0;
  // process-wide, so always the largest size any plan can use
  if (cudaFuncSetAttribute(arnoldi_low_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(optin - fixed)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, arnoldi_low_kernel<T>, kLT, smem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (per_sm < 1) return false;
  p->low_grid = grid;
  p->low_smem = smem;
  p->low_rows = rows;
  return true;
}

}  // namespace

template <typename T>
bool arnoldi_plan(const sk_matrix_s* A, i64 n, ArnoldiPlan* p) {
  *p = ArnoldiPlan{};
  p->grid = arnoldi_grid<T>(A, n, &p->smem, &p->rows_per_cta);
  if (p->grid > 0 && !arnoldi_low_plan<T>(A, n, p)) p->low_grid = 0;
  return p->grid > 0;
}

template <typename T>
sk_status arnoldi_launch(const ArnoldiPlan& p, ArnoldiArgs<T> a, cudaStream_t st) {
  const bool low = p.low(a.j);
  a.rows_per_cta = low ? p.low_rows : p.rows_per_cta;
  a.wait_ns = wait_limit_ns();
  a.bias = wait_target_bias();
  // the barriers of the one-sum-per-vector kernel count from 0; the error
  // word and the step count stay for the solve
  if (!low) SK_CUDA(cudaMemsetAsync(&a.sync->arrived, 0, sizeof(unsigned long long), st));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(low ? p.low_grid : p.grid));
  cfg.blockDim = dim3(low ? kLT : kAT);
  cfg.dynamicSmemBytes = low ? p.low_smem : p.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  SK_CUDA(cudaLaunchKernelEx(&cfg, low ? arnoldi_low_kernel<T> : arnoldi_mgs_kernel<T>, a));
  return SK_OK;
}

template bool arnoldi_plan<double>(const sk_matrix_s*, i64, ArnoldiPlan*);
template bool arnoldi_plan<float>(const sk_matrix_s*, i64, ArnoldiPlan*);
template sk_status arnoldi_launch<double>(const ArnoldiPlan&, ArnoldiArgs<double>, cudaStream_t);
template sk_status arnoldi_launch<float>(const ArnoldiPlan&, ArnoldiArgs<float>, cudaStream_t);

}  // namespace sk
