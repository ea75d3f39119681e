// sk_arnoldi.cuh -- the modified Gram-Schmidt of one GMRES / FGMRES Arnoldi
// step as one cooperative launch (sk_arnoldi.cu).
#pragma once

#include "sk_kernels.cuh"

namespace sk {

// Barrier words of the launch: `arrived` is zeroed before every launch; a
// barrier wait that runs out sets `err`, which stays set for the solve.
struct ArnoldiSync {
  unsigned long long arrived;
  int err;
  unsigned step;  // two-sum kernel: launches done since the solve began, the tag of their sums
  unsigned long long low_arrived;  // its arrivals, counted over the solve
};

// The two-sum form of the step (arnoldi_low_kernel): columns it takes, its
// largest grid, and the fewest rows worth a CTA of their own.
constexpr int kArnLowCols = 64;
constexpr int kArnLowGrid = 160;
constexpr int kArnLowRows = 64;
// Its workspace: the mailboxes of its first exchange and the packed inverse.
constexpr size_t kArnLowBytes =
    static_cast<size_t>(2 * kArnLowCols) * kArnLowGrid * 32 +
    static_cast<size_t>(kArnLowCols) * kArnLowCols * 8;

struct FgSmall {  // device arrays of one restart cycle
  double* H;   // (m+1) x m, column-major, leading dimension m+1
  double* cs;
  double* sn;
  double* g;   // m+1
  double* y;   // m
  double* zero;  // a constant 0 (the h of an MGS pass that only takes a dot)
};

// w (= v_{j+1}) holds A z_j and hcol[0] = h_{0j} (the product's epilogue);
// the launch writes hcol[1 .. j+1] and leaves v_{j+1} = w / h_{j+1,j}.
// slots: 2 * grid doubles.
template <typename T>
struct ArnoldiArgs {
  i64 n;
  T* w;
  const T* V;
  i64 ldv;
  int j;
  double* hcol;
  bool divide;  // GMRES divides by h, FGMRES multiplies by 1 / h
  const Scalars* sc;
  ArnoldiSync* sync;
  double* slots;
  // two-sum form: mailboxes {sum, sending CTA} and {receiving CTA, sum}, and
  // (I + L)^-1 below its diagonal by rows
  ulonglong2* box1;
  ulonglong2* box2;
  double* tri;
  // two-sum form: the step's Givens rotations and convergence test
  Scalars* sc_out;
  double* hist;
  FgSmall sm;
  int m;
  bool hess64;  // the least-squares problem in FP64 whatever T is
  i64 rows_per_cta;             // set by arnoldi_launch
  unsigned long long wait_ns;   // bound of each barrier wait, set by arnoldi_launch
  unsigned bias;                // extra arrivals a barrier waits for (timeout tests)
};

struct ArnoldiPlan {
  int grid = 0;
  size_t smem = 0;
  i64 rows_per_cta = 0;
  int low_grid = 0;  // two-sum form: its grid, or 0 when it does not fit
  size_t low_smem = 0;
  i64 low_rows = 0;
  // whether step j runs in it
  bool low(int j) const { return low_grid > 0 && j < kArnLowCols; }
};

// Whether the step fits: a cooperative grid of at most one CTA per SM whose
// CTAs hold their rows of w in shared memory.
template <typename T>
bool arnoldi_plan(const sk_matrix_s* A, i64 n, ArnoldiPlan* p);

// Enqueues the step on st (capturable: a cooperative kernel launch, after a
// memset of the barrier counter in the one-sum-per-vector form).  In the
// two-sum form the product need not make hcol[0], and the column is rotated
// (apply_givens_rotations, record_residual, check_convergence).
template <typename T>
sk_status arnoldi_launch(const ArnoldiPlan& p, ArnoldiArgs<T> a, cudaStream_t st);

}  // namespace sk
