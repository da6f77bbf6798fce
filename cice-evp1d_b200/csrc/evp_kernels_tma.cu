// evp_kernels_tma.cu -- the fused EVP subcycle as a TMA-fed producer/consumer
// kernel (sm_100a), one CTA per SM.
//
// CTA b works through the tiles of its run, t = run_off[b] .. run_off[b+1]-1,
// in order.  A tile's stress inputs (geometry, strength, packed index words,
// the 12 stresses, u and v of the owned points and of the stencil's extra
// points, and the recomputed forward halo) are staged in shared memory in a
// two-slot ring.  The owned points of a tile are contiguous slots and its
// per-call constants one contiguous block, so the owned data arrive by
// cp.async.bulk (TMA) copies completing on the slot's mbarrier (complete_tx);
// the halo and the extra velocities are gathered with 4/8-byte cp.async, whose
// completion arrives on the same mbarrier (cp.async.mbarrier.arrive).
//
// Three roles, each a number of warpgroups with registers of its own:
//   producers (4 warps): the bulk warp writes the slot's header, arms its
//     barrier and copies the constants, u and v; three gather warps copy four
//     stresses each and gather a third of the halo.  Each waits for the slot
//     and the record by itself.  (One warp issuing all 15 bulk copies took
//     1.3 us a tile, of a period of 2.5; four take 0.5.)  Their own inputs,
//     the tile's slot range and gather lists, are one 1.3 KB record per tile
//     that a bulk copy brings up to kRecRing tiles ahead.
//   stress (8 warps, one thread per compute-set point: the tile's owned points,
//     then its forward halo, 256 at most): all inputs to registers, which
//     frees the slot for the tile after next; the new stresses to the other
//     ping-pong buffer; str to the tile's table, and what stepu needs of the
//     point itself (old velocity, packed word) beside it.
//   stepu (8 warps, the owned points): its 13 inputs (the second part of the
//     constant block) straight to registers while stress runs (the bulk warp
//     has prefetched them into L2), then str from the tile's own table and from
//     the previous tile's, which stays alive: three tables rotate (six of the
//     eight str, in pairs read together; str1 and str5 are read by their own
//     point alone).  Where every Tbu of the call is +0, every uinit and vinit
//     finite and revp == 0, the last three inputs are not read: Tbu is +0, and
//     revp*uinit a signed zero whose sign comes from the packed word.
// What bounds it: up to about 500k points stress, 2.1 us a tile: 1.45 in the
// arithmetic, at 85 % of the FP64 pipe with stepu beside it, 0.65 in moving
// its inputs and results, when the pipe idles (three warps per scheduler do
// not fit the registers); above that HBM (1.18M points: 81 % of the measured
// copy rate).  us a subcycle, against eight warps that did stress and stepu one
// after the other with a shared-memory slot for stepu's inputs: 124k points
// 12.4 -> 11.25, 190k 17.1 -> 15.6, 296k 25.9 -> 23.3, 460k 36.5 -> 33.1, 1.18M
// 91.5 -> 83.  (With a single slot for stepu's inputs, freed when stepu began,
// the copies' latency of 2 us a tile set the pace: 12.0, 25.0, 86.)
// Consecutive one-subcycle launches overlap: each CTA lets the next launch
// start at once (griddepcontrol.launch_dependents), and a launch started that
// way loads its first tile's records, constants and stepu inputs while the
// previous one finishes, reading the state only after griddepcontrol.wait.
//
// Every mbarrier wait is bounded by %globaltimer (kWaitNs): on expiry the warp
// records an error code and leaves; the waits for its arrivals run out in turn.
// Every producer warp waits (bounded) for the slots it has issued copies into
// before it exits, so nothing is left in flight.
#include <cstddef>
#include <cstdint>

#include "evp_kernels.cuh"
#include "evp_resident_mail.cuh"
#include "evp_tiles.h"

namespace evp {

namespace {

constexpr int kSSlots = 2;                          // stress-part ring
constexpr int kRecRing = 4;                         // producer records in flight
constexpr int kStressThreads = kTileCompute;        // 256 = 8 warps, two per scheduler
constexpr int kStepuThreads = kTileCompute;         // 8 more
constexpr int kGatherWarps = 3;                     // producer warps issuing cp.async gathers
constexpr int kStageWarps = 1 + kGatherWarps;       // bulk warp + gather warps: a warpgroup
constexpr int kThreads = kStressThreads + kStepuThreads + 32 * kStageWarps;
// Registers: the launch gives each of 640 threads kLaunchRegs; the roles share
// the same sum out again (setmaxnreg; its inc would wait for ever for more than
// the launch's sum, which tma_prepare checks against the compiled kernels).
constexpr int kLaunchRegs = 96;
constexpr int kStressRegs = 144, kStepuRegs = 72, kStageRegs = 48;
static_assert(kStressThreads * kStressRegs + kStepuThreads * kStepuRegs +
                      32 * kStageWarps * kStageRegs <=
                  kThreads * kLaunchRegs,
              "the roles' registers are the launch's");
static_assert(kStageWarps == 4, "setmaxnreg goes by warpgroups of four warps");
constexpr int kUV = kTileOwned + kTileUvx;
constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s

// Stress part of a tile.
struct SSlot {
  double cs[kConstStressFields][kTileOwned];  // constant block fields 0..7 (one bulk copy)
  double s12[12][kTileOwned];                 // the 12 stresses
  double u[kUV];
  double v[kUV];
  double hf[kTmaStressFields][kTileHalo];  // halo: 6 geometry, strength, 12 stresses
  uint32_t hmeta[kTileHalo];
  uint32_t hlcc[kTileHalo];
  uint32_t hlcor[kTileHalo];
  int hdr[4];  // tile offset, owned count, halo count (written by the bulk warp)
};

static_assert(kConstTileSlots == kTileOwned, "constant blocks hold one tile");
static_assert(kConstFields == kConstStressFields + kTmaStepuFields, "constant block layout");

struct Smem {
  SSlot ss[kSSlots];
  // rotating str tables of what other points read: (str2, str7), (str3, str6),
  // (str4, str8); position kZeroSlot holds 0
  double2 str[3][3][kStrRow];
  // what stepu needs of its own point, from stress: (str1, str5); the old
  // velocity, the packed word with uinit's and vinit's signs, the slot offset
  double2 own_str[2][kTileOwned];
  double2 old[3][kTileOwned];
  uint2 word[3][kTileOwned];
  int off[3];
  alignas(16) int32_t rec[kRecRing][kRecInts];  // bulk copies' destination
  unsigned long long sfull[kSSlots];
  unsigned long long sempty[kSSlots];
  unsigned long long rec_full[kRecRing], rec_empty[kRecRing];
  unsigned long long strfull[2];  // stress of a step is in the str tables (even, odd steps)
  unsigned long long strread[2];  // stepu of a step has read them
  volatile int done[kStepuThreads / 32];  // several subcycles: steps each stepu warp has stored
  volatile int prod_ok;  // several subcycles: no producer warp's wait has run out
};

static_assert(sizeof(SSlot) % 16 == 0, "slots must keep 16-byte alignment");
static_assert((kRecInts * 4) % 16 == 0, "records are bulk-copied");
static_assert(offsetof(Smem, rec) % 16 == 0 && offsetof(Smem, ss) % 16 == 0 &&
                  offsetof(Smem, str) % 16 == 0 && offsetof(Smem, own_str) % 16 == 0 &&
                  offsetof(Smem, old) % 16 == 0 && offsetof(Smem, word) % 8 == 0 &&
                  offsetof(Smem, sfull) % 8 == 0,
              "alignment of bulk copies' destinations, 16-byte and mbarrier accesses");
static_assert(offsetof(SSlot, s12) % 16 == 0 && offsetof(SSlot, u) % 16 == 0 &&
                  offsetof(SSlot, v) % 16 == 0 && sizeof(double[kTileOwned]) % 16 == 0,
              "bulk copies' destinations within a slot");
static_assert(sizeof(Smem) <= 227 * 1024, "shared memory per block");

// ---------------- PTX helpers -------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait for the phase of parity `parity` to complete; on expiry the
// wait's code goes into the error word.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity,
                                          int *err, int code,
                                          unsigned long long limit_ns = kWaitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > limit_ns) {
      atomicMax(err, code);
      return false;
    }
  }
  return true;
}

// TMA bulk copy global -> shared, completing `bytes` on `bar` (no multicast).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Bulk prefetch of global memory into L2 (no shared memory, no completion).
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}

__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}

// The barrier's pending count drops by one once this thread's earlier
// cp.async copies have landed.
__device__ __forceinline__ void cp_async_arrive(unsigned long long *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

// Order this thread's generic-proxy shared-memory accesses before later
// async-proxy (bulk copy) accesses to the same memory.
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// This warpgroup's registers per thread from here on.
template <int kRegs>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// The bulk warp and the gather warps.
__device__ __forceinline__ void stage_sync() {
  asm volatile("bar.sync 2, %0;" ::"r"(32 * kStageWarps) : "memory");
}

__device__ __forceinline__ void trace_stamp(const TmaArgs &a, int it, int slot) {
  if (a.trace && blockIdx.x == 0 && it < kTraceTiles) a.trace[it * 8 + slot] = (long long)global_ns();
}

// Acquire load of a counter another CTA raises (gpu scope).
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Order this thread's generic-proxy global accesses with its async-proxy
// (bulk copy) accesses of global memory.
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ void fence_acq_rel_gpu() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

// Bounded wait until the counter *e, which other CTAs raise, reaches `need`
// (acquire); on expiry the wait's code goes into the error word.
__device__ __forceinline__ bool wait_counter(const unsigned *e, unsigned need, int *err,
                                             int code, unsigned long long limit_ns) {
  if (ld_acquire(e) >= need) return true;
  const unsigned long long t0 = global_ns();
  while (ld_acquire(e) < need) {
    if (global_ns() - t0 > limit_ns) {
      atomicMax(err, code);
      return false;
    }
  }
  return true;
}

// Relaxed load of a counter another CTA raises (gpu scope, past L1).
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Load of a constant of the call, read once (volatile: issued where it stands,
// ahead of the waits that follow).
__device__ __forceinline__ double ld_const(const double *p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// Coherent 8-byte load (at L2) of state other CTAs may have written.
__device__ __forceinline__ double ld_cg(const double *p) { return __ldcg(p); }

// ---------------- the kernel ---------------------------------------------------
// kStd: parameters with std_params(p) (stress_update_std).  The launch runs
// a.nsub subcycles; CTA b works through its run's tiles once per subcycle.
// kMulti: a launch of several subcycles (a.nsub > 1 with per-tile counters);
// otherwise one subcycle, whose last-subcycle outputs kLast selects.
template <bool kLast, bool kStd, bool kMulti>
__global__ void __launch_bounds__(kThreads, 1) k_tma(TmaArgs a, Params p) {
  // Indexed straight off the __shared__ symbol (no integer round trip), so
  // every access compiles to a shared-memory load or store, not a generic one.
  // The bulk copies need 16-byte alignment, which the dynamic shared memory
  // base has (checked: a misaligned base is refused, not faulted on).
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &S = *reinterpret_cast<Smem *>(smem_raw);
  const int tid = threadIdx.x;
  if (smem_addr(smem_raw) & 15u) {
    if (tid == 0) atomicMax(a.err, 8);
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < kSSlots; s++) {
      mbar_init(&S.sfull[s], 1 + 32 * kGatherWarps);  // expect_tx arrival + cp.async lanes
      mbar_init(&S.sempty[s], kStressThreads / 32);
      mbar_init(&S.strfull[s], kStressThreads / 32);
      mbar_init(&S.strread[s], kStepuThreads / 32);
    }
    for (int r = 0; r < kRecRing; r++) {
      mbar_init(&S.rec_full[r], 1);
      mbar_init(&S.rec_empty[r], kStageWarps);
    }
    for (int w = 0; w < kStepuThreads / 32; w++) S.done[w] = 0;
    S.prod_ok = 1;
    mbar_fence_init();
  }
  if (tid < 9) S.str[tid / 3][tid % 3][kZeroSlot] = make_double2(0.0, 0.0);
  __syncthreads();
  // A launch of one subcycle may be followed by the next subcycle's, launched
  // as a programmatic dependent (a.pdl there): it can start as soon as every
  // CTA here has started.  Its CTAs cannot share an SM with these (shared
  // memory), so they take the SMs these CTAs leave, and before their
  // griddep_wait they read only what no subcycle writes (tile records,
  // constant blocks).
  if (!kMulti) griddep_launch_dependents();
  // the short stepu part (kTmaStepuCompact fields) where the call allows it
  const bool cpt = a.compact && __ldg(a.cflags) == 0;

  const int T0 = a.run_off[blockIdx.x], T1 = a.run_off[blockIdx.x + 1];
  const int n = T1 - T0;             // tiles of the run
  const int nq = kMulti ? n * a.nsub : n;  // (subcycle, tile) steps of the launch
  constexpr bool multi = kMulti;
  constexpr uint32_t kCsBytes = kConstStressFields * kTileOwned * 8u;
  constexpr size_t kBlk = (size_t)kConstFields * kTileOwned;  // doubles per constant block
  if (n <= 0) return;

  if (tid >= kStressThreads + kStepuThreads) {
    reg_dec<kStageRegs>();
    // ======================= producers ===================================
    // Each warp waits (bounded) for the tile record and the free slot.  The bulk
    // warp (pw 0) writes the slot header, arms the slot's full barrier with the
    // bytes of all bulk copies (the others' may land before: the phase still
    // lacks the arrival) and issues the constants', u's and v's.  The gather
    // warps issue the stresses' and gather the forward halo and the extra
    // velocities (8-byte cp.async, or, in a launch of several subcycles,
    // coherent loads).  A record is refilled once all four are done with it.
    // Step q = (subcycle q / n, tile q % n).
    // A launch of several subcycles: step q's stress part goes out only when
    // every tile its tile depends on has finished the previous subcycle.  The
    // bulk warp's lanes read those tiles' counters (relaxed) at the end of
    // round q-1 and check them here, so the check usually costs no wait; the
    // acquire fence then orders the state reads after the counters, and a
    // barrier of the four warps the others' reads after that.  The bulk warp
    // also publishes this CTA's steps: once every stepu warp has stored a step
    // (S.done), it raises the tile's counter after a gpu-scope fence.  Stress
    // and stepu finish every earlier step without this round: no wait can
    // depend on itself.
    const int pw = (tid - kStressThreads - kStepuThreads) >> 5;
    const int lane = tid & 31;
    constexpr uint32_t kRecBytes = kRecInts * 4u;
    const uint32_t ubytes = (cpt ? kTmaStepuCompact : kTmaStepuFields) * kTileOwned * 8u;
    int pub = 0;  // steps whose counters are raised (multi-subcycle launches)
    // Lane 0: raise the counters of every step whose stepu has stored.
    auto publish = [&](int limit) {
      bool any = false;
      for (; pub < limit; pub++) {
        for (int w = 0; w < kStepuThreads / 32; w++)
          if (S.done[w] <= pub) return;
        if (!any) __threadfence();
        any = true;
        atomicAdd(a.epoch + T0 + (kMulti ? pub % n : pub), 1u);
      }
    };
    int nrec = 0;  // records issued (the bulk warp's lane 0 counts)
    auto issue_rec = [&]() {
      const int r = nrec % kRecRing;
      const int t = T0 + (kMulti ? nrec % n : nrec);
      mbar_arrive_expect_tx(&S.rec_full[r], kRecBytes);
      bulk_g2s(S.rec[r], a.tile_rec + (size_t)t * kRecInts, kRecBytes, &S.rec_full[r]);
      nrec++;
    };
    if (pw == 0 && lane == 0)
      while (nrec < kRecRing && nrec < nq) issue_rec();
    int issued = 0;
    bool ok = true;
    unsigned seen = 0u;  // per lane: the smallest counter polled for the next step
    for (int q = 0; q < nq; q++) {
      const int sub = kMulti ? q / n : 0, t = T0 + (kMulti ? q % n : q);
      const int from = sub & 1;
      const double *u_in = kMulti && a.uv_step ? a.u[0] + (size_t)sub * a.uv_step : a.u[from];
      const double *v_in = kMulti && a.uv_step ? a.v[0] + (size_t)sub * a.uv_step : a.v[from];
      const int r = issued % kRecRing;
      const int s = issued % kSSlots;
      const uint32_t use = (uint32_t)(issued / kSSlots);
      SSlot &st = S.ss[s];
      const int32_t *rec = S.rec[r];
      int w = 1;
      if (lane == 0) {
        w = mbar_wait(&S.rec_full[r], (uint32_t)(issued / kRecRing) & 1, a.err, 6) ? 1 : 0;
        if (pw == 0) trace_stamp(a, issued, 3);
        if (w && issued >= kSSlots)
          w = mbar_wait(&S.sempty[s], (use - 1) & 1, a.err, 2) ? 1 : 0;
      }
      w = __shfl_sync(0xffffffffu, w, 0);
      __syncwarp();
      if (pw == 0) {
        if constexpr (kMulti) {
          if (w && sub > 0) {
            // the tiles step q depends on have finished subcycle sub - 1; the
            // warp waits together, lane 0 publishing this CTA's finished steps
            // meanwhile (a tile may wait on its own run's steps)
            const unsigned need = (unsigned)sub;
            const int d0 = a.dep_off[t], d1 = a.dep_off[t + 1];
            const unsigned long long t0 = global_ns();
            for (bool first = true;; first = false) {
              bool mine = true;
              for (int d = d0 + lane; d < d1 && mine; d += 32) {
                if (first && d < d0 + 32 && seen >= need) continue;
                mine = ld_relaxed(a.epoch + a.dep_idx[d]) >= need;
              }
              if (__all_sync(0xffffffffu, mine)) break;
              if (lane == 0) publish(q);
              // one decision for the whole warp (lane 0's clock)
              if (__shfl_sync(0xffffffffu, global_ns() - t0 > kWaitNs ? 1 : 0, 0)) {
                if (lane == 0) atomicMax(a.err, 13);
                w = 0;
                break;
              }
            }
            // acquire: the neighbours' state is read after their counters, by
            // these bulk copies (async proxy) and by the gather warps
            fence_acq_rel_gpu();
            fence_proxy_async_global();
          }
        }
        if (lane == 0) trace_stamp(a, issued, 4);
        if (w) {
          const int nh = rec[3];
          for (int h = lane; h < nh; h += 32) {
            st.hlcor[h] = (uint32_t)rec[kRecHLcor + h];
            st.hlcc[h] = (uint32_t)rec[kRecHLcc + h];
          }
          if (lane == 0) {
            st.hdr[0] = rec[0];
            st.hdr[1] = rec[1];
            st.hdr[2] = nh;
          }
          __syncwarp();
          // release: the header and halo indices are visible to consumers
          // once the phase completes
          if (lane == 0) {
            const uint32_t b8 = (uint32_t)((rec[1] + 3) & ~3) * 8u;
            mbar_arrive_expect_tx(&S.sfull[s], kCsBytes + 14 * b8);
          }
        }
      }
      if constexpr (kMulti) {
        // one decision for all four warps, which meet again below
        if (!w && lane == 0) S.prod_ok = 0;
        stage_sync();
        w = S.prod_ok;
        fence_proxy_async_global();
      }
      if (!w) {
        ok = false;
        break;
      }
      const int off = rec[0], cnt = rec[1], nx = rec[2], nh = rec[3];
      if (pw == 0) {
        const uint32_t b8 = (uint32_t)((cnt + 3) & ~3) * 8u;
        if (lane == 0) {
          bulk_g2s(st.cs, a.cblk + (size_t)t * kBlk, kCsBytes, &S.sfull[s]);
          // (stepu's loads of its part find it in L2)
          bulk_prefetch_l2(a.cblk + (size_t)t * kBlk + kConstStressFields * kTileOwned, ubytes);
        }
        // the state the previous subcycle wrote
        if (issued == 0) griddep_wait();
        if (lane == 0) {
          bulk_g2s(st.u, u_in + off, b8, &S.sfull[s]);
          bulk_g2s(st.v, v_in + off, b8, &S.sfull[s]);
          trace_stamp(a, issued, 6);
        }
      } else {
        // gather warp gw takes the velocity extras u (first) / v (last) and
        // every kGatherWarps-th halo field; the last one also the halo meta
        const int gw = pw - 1;
        if (issued == 0) griddep_wait();
        if (lane < 12 / kGatherWarps) {
          const int k = gw * (12 / kGatherWarps) + lane;
          bulk_g2s(st.s12[k], a.s[from][k] + off, (uint32_t)((cnt + 3) & ~3) * 8u, &S.sfull[s]);
        }
        __syncwarp();
        if (!multi) {
          if (gw == 0)
            for (int x = lane; x < nx; x += 32)
              cp_async8(&st.u[kTileOwned + x], u_in + rec[kRecUvx + x]);
          if (gw == kGatherWarps - 1)
            for (int x = lane; x < nx; x += 32)
              cp_async8(&st.v[kTileOwned + x], v_in + rec[kRecUvx + x]);
          for (int h = lane; h < nh; h += 32) {
            const int g = rec[kRecHalo + h];
            for (int f = gw; f < kTmaStressFields; f += kGatherWarps)
              cp_async8(&st.hf[f][h], (f < 7 ? a.sg[f] : a.s[from][f - 7]) + g);
            if (gw == kGatherWarps - 1) cp_async4(&st.hmeta[h], a.meta + g);
          }
          cp_async_arrive(&S.sfull[s]);
        } else {
          // state written by other CTAs in this launch: loads at L2 (not a
          // copy that an earlier read may have left in this SM's L1)
          // Each lane issues a batch of loads before it stores any of them,
          // so that they overlap instead of taking one L2 round trip each.
          constexpr int kXPer = kTileUvx / 32;  // extras per lane at most
          for (int c = 0; c < 2; c++) {
            if (c == 0 ? gw != 0 : gw != kGatherWarps - 1) continue;
            const double *src = c == 0 ? u_in : v_in;
            double *dst = (c == 0 ? st.u : st.v) + kTileOwned;
            double xv[kXPer];
#pragma unroll
            for (int i = 0; i < kXPer; i++) {
              const int x = lane + 32 * i;
              xv[i] = x < nx ? ld_cg(src + rec[kRecUvx + x]) : 0.0;
            }
#pragma unroll
            for (int i = 0; i < kXPer; i++)
              if (lane + 32 * i < nx) dst[lane + 32 * i] = xv[i];
          }
          // halo: this warp's fields f = gw (mod kGatherWarps) of every halo
          // point, spread over the lanes by (point, field)
          const int nf = (kTmaStressFields - gw + kGatherWarps - 1) / kGatherWarps;
          const int items = nh * nf;
          constexpr int kBatch = 8;
          for (int j0 = 0; j0 < items; j0 += 32 * kBatch) {
            double hv[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
              const int j = j0 + lane + 32 * i;
              if (j < items) {
                const int h = j / nf, f = gw + kGatherWarps * (j - h * nf);
                hv[i] = ld_cg((f < 7 ? a.sg[f] : a.s[from][f - 7]) + rec[kRecHalo + h]);
              }
            }
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
              const int j = j0 + lane + 32 * i;
              if (j < items) {
                const int h = j / nf, f = gw + kGatherWarps * (j - h * nf);
                st.hf[f][h] = hv[i];
              }
            }
          }
          if (gw == kGatherWarps - 1)
            for (int h = lane; h < nh; h += 32) st.hmeta[h] = a.meta[rec[kRecHalo + h]];
          mbar_arrive(&S.sfull[s]);
        }
        if (gw == 0 && lane == 0) trace_stamp(a, issued, 7);
      }
      // the record's generic reads come before its async-proxy refill
      fence_proxy_async();
      if constexpr (kMulti) stage_sync();  // every warp is done with prod_ok
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.rec_empty[r]);
      if (pw == 0) {
        if (lane == 0) {
          trace_stamp(a, issued, 0);
          // the record every warp has finished with by now
          if (q >= 1 && nrec < nq) {
            if (mbar_wait(&S.rec_empty[(q - 1) % kRecRing], (uint32_t)((q - 1) / kRecRing) & 1,
                          a.err, 18))
              issue_rec();
          }
        }
        if (a.prefetch > 0 && !multi) {
          const int tp = t + a.prefetch;
          if (tp < T1 && lane < 15) {
            // what the stage load of a later tile copies: its constant block,
            // the owned ranges of the 12 stresses, u and v
            const int po = a.tile_meta[8 * tp], pc = a.tile_meta[8 * tp + 1];
            const uint32_t pb = (uint32_t)((pc + 3) & ~3) * 8u;
            if (lane == 0)
              bulk_prefetch_l2(a.cblk + (size_t)tp * kBlk, (uint32_t)(kBlk * 8u));
            else if (lane <= 12)
              bulk_prefetch_l2(a.s[from][lane - 1] + po, pb);
            else
              bulk_prefetch_l2((lane == 13 ? u_in : v_in) + po, pb);
          }
        }
        if (multi) {
          if (lane == 0) publish(q);
          // the counters of the next step's dependencies, read ahead
          const int q1 = q + 1;
          if (q1 < nq && q1 / n > 0) {
            const int t1 = T0 + q1 % n, d = a.dep_off[t1] + lane;
            seen = d < a.dep_off[t1 + 1] ? ld_relaxed(a.epoch + a.dep_idx[d]) : 0u;
          }
        }
      }
      issued++;
    }
    // No copy may target shared memory after the CTA exits: every warp waits
    // (bounded) for the slots it has issued copies into.  A wait that ran out
    // in one warp need not have in another: a gather warp can have issued into
    // a slot that the bulk warp never armed, which holds it here for the limit.
    // (Without such a failure these waits end before stress does.)
    for (int k = issued - kSSlots; k < issued; k++)
      if (k >= 0 && lane == 0)
        mbar_wait(&S.sfull[k % kSSlots], (uint32_t)(k / kSSlots) & 1, a.err, 3);
    if (pw == 0) {
      if (multi && lane == 0) {
        // the last steps' counters (a later launch zeroes them anyway)
        const unsigned long long t0 = global_ns();
        while (ok && pub < issued && global_ns() - t0 < kWaitNs) publish(issued);
      }
      // records issued ahead and never consumed must land before exit too
      if (lane == 0) {
        for (int k = issued; k < nrec; k++)
          mbar_wait(&S.rec_full[k % kRecRing], (uint32_t)(k / kRecRing) & 1, a.err, 7);
      }
    }
    __syncwarp();
    return;
  }

  const int lane = tid & 31;
  if (tid >= kStressThreads) {
    // ======================= stepu of the owned points =====================
    // Its 13 fields come to registers, straight from the constant block, while
    // stress of the same step runs; the rest is in the tables of strfull.
    reg_dec<kStepuRegs>();
    const int c = tid - kStressThreads;
    for (int q = 0; q < nq; q++) {
      const int b = q % 3;
      const int bp = (q + 2) % 3;  // the previous tile's table
      const int sub = kMulti ? q / n : 0;
      const int to = (sub & 1) ^ 1;
      const bool wlast = kMulti ? (a.last && sub == a.nsub - 1) : kLast;
      const double *cu = a.cblk + ((size_t)(T0 + (kMulti ? q % n : q)) * kConstFields +
                                   kConstStressFields) * kTileOwned + c;
      StepuIn in;
      in.kvrel = ld_const(cu);
      in.uocn = ld_const(cu + kTileOwned);
      in.vocn = ld_const(cu + 2 * kTileOwned);
      in.waterx = ld_const(cu + 3 * kTileOwned);
      in.watery = ld_const(cu + 4 * kTileOwned);
      in.forcex = ld_const(cu + 5 * kTileOwned);
      in.forcey = ld_const(cu + 6 * kTileOwned);
      in.umassdti = ld_const(cu + 7 * kTileOwned);
      in.fm = ld_const(cu + 8 * kTileOwned);
      in.uarear = ld_const(cu + 9 * kTileOwned);
      in.Tbu = 0.0;
      if (!cpt) {
        in.Tbu = ld_const(cu + 10 * kTileOwned);
        in.uinit = ld_const(cu + 11 * kTileOwned);
        in.vinit = ld_const(cu + 12 * kTileOwned);
      }
      if (q == 0) griddep_wait();
      const bool ok = mbar_wait(&S.strfull[q & 1], (uint32_t)(q >> 1) & 1, a.err, 16);
      const uint2 word = S.word[b][c];
      const uint32_t m = word.x;
      const bool act = ok && !((m >> 30) & kSkipU);
      const int at = S.off[b] + c;
      if (act) {
        const double2 old = S.old[b][c];
        in.uold = old.x;
        in.vold = old.y;
        if (cpt) {
          // Tbu is +0; revp == 0, so revp*uinit is a zero with uinit's sign
          in.uinit = (word.y >> 30 & 1u) ? -1.0 : 1.0;
          in.vinit = (word.y >> 31) ? -1.0 : 1.0;
        }
        // a neighbour's str: own table, or the previous tile's (kStrPrev)
        const uint32_t vnw = m & kLnbMask, vsw = (m >> kLnbBits) & kLnbMask;
        const uint32_t vsse = (m >> (2 * kLnbBits)) & kLnbMask;
        const double2 own = S.own_str[q & 1][c];
        const double2 nw = S.str[(vnw & kStrPrev) ? bp : b][0][vnw & (kStrPrev - 1)];
        const double2 sse = S.str[(vsse & kStrPrev) ? bp : b][1][vsse & (kStrPrev - 1)];
        const double2 sw = S.str[(vsw & kStrPrev) ? bp : b][2][vsw & (kStrPrev - 1)];
        in.s1 = own.x;
        in.s5 = own.y;
        in.s2nw = nw.x;
        in.s7nw = nw.y;
        in.s3sse = sse.x;
        in.s6sse = sse.y;
        in.s4sw = sw.x;
        in.s8sw = sw.y;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.strread[q & 1]);
      if (act) {
        const StepuOut o = stepu_point(in, p);
        double *u_out = kMulti && a.uv_step ? a.u[0] + (size_t)(sub + 1) * a.uv_step : a.u[to];
        double *v_out = kMulti && a.uv_step ? a.v[0] + (size_t)(sub + 1) * a.uv_step : a.v[to];
        u_out[at] = o.u;
        v_out[at] = o.v;
        if (wlast) {
          a.strintx[at] = o.strintx;
          a.strinty[at] = o.strinty;
          a.Cb[at] = o.Cb;
        }
      }
      if (kMulti) {
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          S.done[c >> 5] = q + 1;
        }
      }
      if (c == 0) trace_stamp(a, q, 5);
      if (__any_sync(0xffffffffu, !ok)) return;
    }
    return;
  }

  // ========================= stress ======================================
  // A warp goes from tile to tile by itself: its inputs are all in registers
  // before the arithmetic, so that the slot is free for the tile after next.
  // The three str tables: stepu of step q reads those of q and q-1 while
  // stress of q+1 writes the third; stress of q+2 writes over that of q-1, and
  // over the even/odd own_str of q, and waits until stepu of q has read them.
  // (The first tile of a run never reads the previous table, so nothing
  // crosses from one subcycle to the next there.)  A warp whose wait ran out
  // leaves; the waits for its arrivals run out in turn.
  reg_inc<kStressRegs>();
  const int c = tid;  // compute-set index: owned c < cnt, halo cnt + h
  // Writes the ping-pong set the previous subcycle read: only after it has
  // completed (the first tile cannot land before that anyway).
  griddep_wait();
  for (int q = 0; q < nq; q++) {
    const int s = q % kSSlots;
    const int b = q % 3;
    const int sub = kMulti ? q / n : 0;
    const int to = (sub & 1) ^ 1;
    const bool wlast = kMulti ? (a.last && sub == a.nsub - 1) : kLast;
    bool ok = mbar_wait(&S.sfull[s], (uint32_t)(q / kSSlots) & 1, a.err, 1);
    if (tid == 0) trace_stamp(a, q, 1);
    bool own = false, in = false, act = false;
    int at = 0;
    double geo[7], s12[12];
    Corners cr;
    uint2 word = make_uint2((uint32_t)kSkipU << 30, 0u);
    if (ok) {
      const SSlot &st = S.ss[s];
      const int cnt = st.hdr[1];
      at = st.hdr[0] + c;
      own = c < cnt;
      const int h = c - cnt;
      in = own || h < st.hdr[2];
      if (in) {
        uint32_t m, lc;
        if (own) {
          const unsigned long long ml = (unsigned long long)__double_as_longlong(st.cs[7][c]);
          m = (uint32_t)ml;
          lc = (uint32_t)(ml >> 32);
          word = make_uint2(m, lc);
          S.old[b][c] = make_double2(st.u[c], st.v[c]);
        } else {
          m = st.hmeta[h];
          lc = st.hlcor[h];
        }
        act = !((m >> 30) & kSkipT);
        if (act) {
          // geometry and strength (fields 0..6), then the 12 stresses
          const double *F = own ? &st.cs[0][c] : &st.hf[0][h];
          const double *F12 = own ? &st.s12[0][c] : &st.hf[7][h];
          const int fs = own ? kTileOwned : kTileHalo;
          const int cc = own ? c : (int)st.hlcc[h];
          const int iee = lc & kLnbMask, ine = (lc >> kLnbBits) & kLnbMask;
          const int ise = (lc >> (2 * kLnbBits)) & kLnbMask;
          cr.ucc = st.u[cc];
          cr.vcc = st.v[cc];
          cr.uee = st.u[iee];
          cr.vee = st.v[iee];
          cr.une = st.u[ine];
          cr.vne = st.v[ine];
          cr.use = st.u[ise];
          cr.vse = st.v[ise];
#pragma unroll
          for (int k = 0; k < 7; k++) geo[k] = F[k * fs];
#pragma unroll
          for (int k = 0; k < 12; k++) s12[k] = F12[k * fs];
        }
      }
    }
    S.word[b][c] = word;
    if (tid == 0) S.off[b] = at;
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.sempty[s]);
    double out[8];
    if (act) {
      const Geom gm = make_geom(geo[0], geo[1], geo[2], geo[3], geo[4], geo[5], p.deltaminEVP);
      stress_point<kStd>(cr, gm, geo[6], s12, out, p);
      if (own) {
#pragma unroll
        for (int k = 0; k < 12; k++) a.s[to][k][at] = s12[k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) out[k] = 0.0;
    }
    if (q >= 2) ok &= mbar_wait(&S.strread[q & 1], (uint32_t)((q >> 1) - 1) & 1, a.err, 17);
    if (ok && in) {
      S.str[b][0][c] = make_double2(out[1], out[6]);
      S.str[b][1][c] = make_double2(out[2], out[5]);
      S.str[b][2][c] = make_double2(out[3], out[7]);
      if (own) S.own_str[q & 1][c] = make_double2(out[0], out[4]);
      if (wlast && own) {
#pragma unroll
        for (int k = 0; k < 8; k++) a.str_out[k][at] = out[k];
      }
    }
    if (__any_sync(0xffffffffu, !ok)) return;
    __syncwarp();  // every lane's stores come before the arrival
    if (lane == 0) mbar_arrive(&S.strfull[q & 1]);
    if (tid == 0) trace_stamp(a, q, 2);
  }
}

size_t smem_bytes() { return sizeof(Smem); }

// One thread waits, through the kernel's own bounded wait, on an mbarrier at
// which nothing ever arrives: the wait runs out after limit_ns and records
// kProbeCode, as a timed-out wait of the subcycle kernel would.
constexpr int kProbeCode = 12;

__global__ void k_wait_probe(int *err, unsigned long long limit_ns) {
  __shared__ unsigned long long bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    mbar_wait(&bar, 0, err, kProbeCode, limit_ns);
  }
}

// The same for the dependency wait of a multi-subcycle launch: one thread
// waits on a counter that nothing raises.
constexpr int kDepProbeCode = 14;

__global__ void k_dep_probe(int *err, const unsigned *counter, unsigned long long limit_ns) {
  if (threadIdx.x == 0) wait_counter(counter, 1u, err, kDepProbeCode, limit_ns);
}

}  // namespace

const char *tma_wait_name(int code) {
  switch (code) {
    case 1: return "a consumer waited for a tile's stress inputs";
    case 2: return "the producer waited for a free stress slot";
    case 3: return "the producer waited for its copies to land before it ended";
    case 6: return "the producer waited for a tile record";
    case 7: return "the producer waited for records issued ahead";
    case 8: return "the dynamic shared memory was not 16-byte aligned";
    case 18: return "the producer waited for its warps to finish with a record";
    case 16: return "stepu waited for a tile's stress";
    case 17: return "stress waited for stepu to read the str tables";
    case 13: return "the producer waited for neighbouring tiles to finish a subcycle";
    case kResCode: return "a resident block waited for another block's velocities";
    case kMailProbeCode: return "the mailbox-wait probe (evp1d_debug_mail_wait_timeout)";
    case kProbeCode: return "the wait probe (evp1d_debug_wait_timeout)";
    case kDepProbeCode: return "the dependency-wait probe (evp1d_debug_dep_wait_timeout)";
    default: return "unknown";
  }
}

cudaError_t tma_binary_version(int *version) {
  cudaFuncAttributes at;
  const cudaError_t e = cudaFuncGetAttributes(&at, k_tma<false, true, false>);
  if (e == cudaSuccess) *version = at.binaryVersion;
  return e;
}

void launch_wait_probe(int *err, unsigned long long limit_ns, cudaStream_t st) {
  k_wait_probe<<<1, 32, 0, st>>>(err, limit_ns);
}

void launch_dep_probe(int *err, const unsigned *counter, unsigned long long limit_ns,
                      cudaStream_t st) {
  k_dep_probe<<<1, 32, 0, st>>>(err, counter, limit_ns);
}

using TmaKernel = void (*)(TmaArgs, Params);
const TmaKernel kTmaAll[] = {
    k_tma<false, false, false>, k_tma<true, false, false>, k_tma<false, true, false>,
    k_tma<true, true, false>,   k_tma<false, false, true>, k_tma<false, true, true>};

cudaError_t tma_prepare(int *short_of) {
  *short_of = 0;
  for (TmaKernel k : kTmaAll) {
    cudaFuncAttributes at;
    cudaError_t e = cudaFuncGetAttributes(&at, k);
    if (e != cudaSuccess) return e;
    if (at.numRegs < kLaunchRegs) {
      *short_of = kLaunchRegs;
      return cudaErrorInvalidKernelImage;
    }
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes());
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

bool tma_can_persist(int device, int nruns) {
  int coop = 0, sms = 0, per_sm = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tma<false, true, true>, kThreads,
                                                    smem_bytes()) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return coop != 0 && nruns <= sms * per_sm;
}

cudaError_t launch_tma(const TmaArgs &given, const Params &p, cudaStream_t st) {
  if (given.ntiles <= 0 || given.nruns <= 0 || given.nsub <= 0) return cudaSuccess;
  TmaArgs a = given;
  // the short stepu part replaces revp*uinit by a signed zero: revp == 0 only
  a.compact = given.compact && given.cflags && p.revp == 0.0;
  const bool std = std_params(p);
  if (a.nsub > 1 && a.epoch) {
    // CTAs wait on one another: all of them resident at once
    TmaKernel k = std ? k_tma<false, true, true> : k_tma<false, false, true>;
    TmaArgs aa = a;
    Params pp = p;
    void *args[] = {&aa, &pp};
    return cudaLaunchCooperativeKernel((const void *)k, dim3(a.nruns), dim3(kThreads), args,
                                       smem_bytes(), st);
  }
  if (a.nsub != 1) return cudaErrorInvalidValue;  // several subcycles need the counters
  TmaKernel k = a.last ? (std ? k_tma<true, true, false> : k_tma<true, false, false>)
                       : (std ? k_tma<false, true, false> : k_tma<false, false, false>);
  if (a.pdl) {
    // a programmatic dependent of the previous launch on the stream, which
    // must be the previous subcycle's k_tma (the caller's guarantee)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.nruns);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes();
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, p);
  }
  k<<<a.nruns, kThreads, smem_bytes(), st>>>(a, p);
  return cudaGetLastError();
}

}  // namespace evp
