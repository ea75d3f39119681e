// sk_gridsum.cuh -- values sent between the CTAs of a cooperative grid that
// carry their own arrival.
//
// A value is stored as two 8-byte words of 32 data bits and a 32-bit tag
// (8-byte stores are single-copy atomic) in a mailbox slot that its receiver
// polls until both words hold the tag of this exchange: no counter, no fence,
// and no clearing between exchanges.  It suits an exchange of many sums at
// once, each added by a CTA of its own and sent on to all (2j + 1 sums over 148
// CTAs: 2.6 us for both hops).  For one sum an arrival counter and a slot per
// CTA are faster (1.87 us, grid_allreduce in sk_mixed.cu): 148 CTAs that each
// poll 148 slots take 3.
//
// Waits are bounded: a poll that runs out sets the error word, every other
// CTA sees it within 256 polls, and the caller returns.
#pragma once

#include "sk_kernels.cuh"

namespace sk {

struct GridWait {
  int* err;
  unsigned long long wait_ns;
  unsigned bias;  // 1: the polls wait for a tag that nobody sends (timeout tests)
};

// One mailbox slot: two words of (tag << 32 | data).
using MailSlot = ulonglong2;

__device__ __forceinline__ unsigned long long mail_now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mail_send(MailSlot* slot, double v, unsigned tag) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
  const unsigned long long a = t | (u & 0xffffffffull), b = t | (u >> 32);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(a), "l"(b) : "memory");
}

// Waits for N values with this tag (slot k at k * stride, k < n of them), all
// N polls in flight together; v[k] of the others is 0.  False when the wait
// ran out.
template <int N>
__device__ __forceinline__ bool mail_wait(const MailSlot* slot, int stride, int n, unsigned tag, GridWait const& w,
                                          double (&v)[N]) {
  const unsigned want = tag + w.bias;
  unsigned long long t0 = 0;
  for (unsigned spins = 0;; ++spins) {
    unsigned long long a[N], b[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      a[k] = b[k] = static_cast<unsigned long long>(want) << 32;
      if (k < n)
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(a[k]), "=l"(b[k])
                     : "l"(slot + static_cast<size_t>(k) * stride)
                     : "memory");
    }
    bool all = true;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      all = all && static_cast<unsigned>(a[k] >> 32) == want && static_cast<unsigned>(b[k] >> 32) == want;
      v[k] = __longlong_as_double(static_cast<long long>((a[k] & 0xffffffffull) | (b[k] << 32)));
    }
    if (all) return true;
    if ((spins & 255u) == 255u) {
      if (*reinterpret_cast<volatile int*>(w.err) != 0) return false;
      const unsigned long long t = mail_now_ns();
      if (t0 == 0) {
        t0 = t;
      } else if (t - t0 > w.wait_ns) {
        atomicExch(w.err, 1);
        return false;
      }
    }
  }
}

}  // namespace sk
