// evp_resident_mail.cuh -- mailboxes between the blocks of a resident launch
// (evp_kernels_resident.cu explains them).
#pragma once

#include <cuda_runtime.h>

namespace evp {

constexpr unsigned long long kResWaitNs = 2000000000ull;  // 2 s
constexpr int kResCode = 15;
constexpr int kMailProbeCode = 19;  // evp1d_debug_mail_wait_timeout

// Two doubles of one point, each 32-bit half beside the message's number.
__device__ __forceinline__ void mail_put(double4 *box, double u, double v, unsigned seq) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(u);
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned long long n = (unsigned long long)seq << 32;
  const unsigned long long m = 0xffffffffull;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(box), "l"((a & m) | n),
               "l"((a >> 32) | n)
               : "memory");
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0+16], {%1, %2};" ::"l"(box), "l"((b & m) | n),
               "l"((b >> 32) | n)
               : "memory");
}

struct Mail {
  unsigned long long a0, a1, b0, b1;
};

__device__ __forceinline__ Mail mail_get(const double4 *box) {
  Mail w;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
               : "=l"(w.a0), "=l"(w.a1)
               : "l"(box)
               : "memory");
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2+16];"
               : "=l"(w.b0), "=l"(w.b1)
               : "l"(box)
               : "memory");
  return w;
}

__device__ __forceinline__ bool mail_is(const Mail &w, unsigned seq) {
  return (unsigned)(w.a0 >> 32) == seq && (unsigned)(w.a1 >> 32) == seq &&
         (unsigned)(w.b0 >> 32) == seq && (unsigned)(w.b1 >> 32) == seq;
}

__device__ __forceinline__ double2 mail_value(const Mail &w) {
  const unsigned long long m = 0xffffffffull;
  return make_double2(__longlong_as_double((long long)((w.a0 & m) | (w.a1 << 32))),
                      __longlong_as_double((long long)((w.b0 & m) | (w.b1 << 32))));
}

__device__ __forceinline__ unsigned long long res_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The whole warp waits (bounded) for message `seq` of the corners in each
// lane's `polled` (bit k: corner k, whose point's slot is ~ref[k]; 0: none).
// The corners are polled together, so that a round of reads costs one trip to
// L2; the words stay as they came until every corner has its own (fewer
// registers than the values beside them).  The lanes leave the loop together:
// a warp whose lanes left one by one would go through what follows in as many
// parts.  Returns false in every lane when the wait ran out.
__device__ __forceinline__ bool mail_wait(Mail (&m)[4], const double4 *box, const int (&ref)[4],
                                          unsigned polled, unsigned seq,
                                          unsigned long long limit_ns = kResWaitNs) {
  unsigned left = polled;
  unsigned long long t0 = 0;
  for (unsigned tries = 1; __any_sync(0xffffffffu, left != 0); tries++) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (left >> k & 1) m[k] = mail_get(box + ~ref[k]);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if ((left >> k & 1) && mail_is(m[k], seq)) left &= ~(1u << k);
    if ((tries & 63u) == 0) {
      const unsigned long long t = res_ns();
      if (t0 == 0) t0 = t;
      if (__any_sync(0xffffffffu, t - t0 > limit_ns)) return false;
    }
  }
  return true;
}

// The same for at most one mailbox a lane (`left`: it waits for its own, whose
// velocity goes to `w`).  Returns true in the lanes whose wait ran out.
__device__ __forceinline__ bool mail_wait_one(double2 &w, const double4 *box, bool left,
                                              unsigned seq,
                                              unsigned long long limit_ns = kResWaitNs) {
  unsigned long long t0 = 0;
  for (unsigned tries = 1; __any_sync(0xffffffffu, left); tries++) {
    if (left) {
      const Mail m = mail_get(box);
      if (mail_is(m, seq)) {
        w = mail_value(m);
        left = false;
      }
    }
    if ((tries & 63u) == 0) {
      const unsigned long long t = res_ns();
      if (t0 == 0) t0 = t;
      if (__any_sync(0xffffffffu, t - t0 > limit_ns)) break;
    }
  }
  return left;
}

}  // namespace evp
