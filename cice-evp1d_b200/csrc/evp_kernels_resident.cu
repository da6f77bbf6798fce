// evp_kernels_resident.cu -- a call's subcycles in one launch, for problems
// small enough to stay on chip (evp_resident.h).
//
// One CTA per block of the resident plan, one thread per compute point (owned
// points, then the forward halo).  A thread keeps its point's 12 stresses in
// registers (kSmemStress: in shared memory) and its constants in shared memory
// from the first subcycle to the last; only velocities move between blocks.
// Per subcycle:
//   stress  reads the corner velocities from shared memory, or, where another
//           block owns the point, from that point's mailbox; writes six of
//           str1..str8 to the block's str table (str1 and str5 are read only
//           by their own point and stay in its registers);
//   barrier
//   stepu   (owned points) writes the new velocity to shared memory and, for
//           a point other blocks read, to its mailbox;
//   barrier
// A mailbox is 32 bytes in L2: the four 32-bit halves of u and v, each beside
// the 32-bit number of the subcycle they belong to.  A 64-bit access is
// atomic, so a word whose number matches carries its half: the reader polls
// the data themselves, and a subcycle's exchange costs one trip to L2 each
// way, with no fence, no flag and no barrier between blocks.  Numbers grow
// across launches, so that nothing stale ever matches.  Each point has two
// mailboxes, for even and odd subcycles.  One can be written again without
// looking: a block writes number n+2 only after it has read number n+1 from
// every block it reads from; those had then passed the barrier after their
// stress n, and they include every block that reads this one (the plan
// requires the symmetry).
// The CTAs wait on one another, so the launch is cooperative (all resident or
// none).  Every wait is bounded: on expiry the code goes to the error word,
// the CTA leaves together at the next barrier, and its neighbours' waits run
// out in turn.
//
// What bounds it: the FP64 pipe (about 535 operations a point, two issue
// cycles each, 64 lanes an SM) for full blocks, the dependent chain through
// stress, stepu and the exchange for small ones; no HBM traffic per subcycle.
// Measured, us per subcycle, against the one-launch-per-subcycle kernel (before
// the straight-line divisions of evp_fp64.cuh): 18k points 2.6 / 5.0, 51k 3.2 /
// 7.8, 64k 3.9 / 8.0, 74k 6.1 / 10.4; smaller problems: k_resident_quad.
#include <cstdint>

#include "evp_kernels.cuh"
#include "evp_resident.h"
#include "evp_resident_mail.cuh"

namespace evp {

namespace {

constexpr int kResGeo = 10;  // dxT dyT cxp cyp cxm cym DminTarea dxhy dyhx strength

template <int NT, bool kSmemStress>
struct ResSmem {
  double2 uv[NT];           // velocities of the owned points
  double2 str[3][NT + 1];   // (str2, str7), (str3, str6), (str4, str8); [NT] stays 0
  double geo[kResGeo][NT];
  double cst[kTmaStepuFields][NT];
  double s[kSmemStress ? 12 : 1][kSmemStress ? NT : 1];
};

// Keeps the compiler from moving shared-memory accesses across: the lean
// stress below is written so that few values are live at once.
__device__ __forceinline__ void hold() { asm volatile("" ::: "memory"); }

// stress_point (evp_math.cuh) on a point's 12 stresses in shared memory (`s`,
// `stride` doubles apart), for the width that leaves a thread 96 registers:
// the relaxations corner by corner, then the x and the y half of str_combine
// with the stresses read again.  Every operation is stress_point's own, in its
// order, so the bits are the same.
template <bool kStd>
__device__ __forceinline__ void stress_lean(double *s, int stride, double (&out)[8],
                                            const Corners &c, const double *geo, int gs,
                                            const Params &p) {
  {
    Geom g;
    g.dxT = geo[0 * gs];
    g.dyT = geo[1 * gs];
    g.cxp = geo[2 * gs];
    g.cyp = geo[3 * gs];
    g.cxm = geo[4 * gs];
    g.cym = geo[5 * gs];
    const StrainSq q = strain_squares(c, g, p.e_factor);
    hold();
    const double strength = geo[9 * gs], least = geo[6 * gs];
    if (stress_in_range(strength, least, q.sq) &&
        (kStd || p.capping == kC1 || p.capping == 0.0)) {
      double Delta[4], visc[4];
      viscosities(strength, least, kStd || p.capping == kC1, q.sq, Delta, visc);
      hold();
#pragma unroll
      for (int k = 0; k < 4; k++) {
        double sp = s[k * stride], sm = s[(4 + k) * stride], st = s[(8 + k) * stride];
        corner_relax<kStd>(sp, sm, st, q.div[k], q.ten[k], q.shr[k], Delta[k], visc[k], p);
        s[k * stride] = sp;
        s[(4 + k) * stride] = sm;
        s[(8 + k) * stride] = st;
        hold();
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        double sp = s[k * stride], sm = s[(4 + k) * stride], st = s[(8 + k) * stride];
        corner_update(sp, sm, st, q.div[k], q.ten[k], q.shr[k], sqrt(q.sq[k]), strength, least, p);
        s[k * stride] = sp;
        s[(4 + k) * stride] = sm;
        s[(8 + k) * stride] = st;
        hold();
      }
    }
  }
#pragma unroll
  for (int half = 0; half < 2; half++) {
    double A[4], D[4];
    {
      const double a0 = s[0], a1 = s[stride], a2 = s[2 * stride], a3 = s[3 * stride];
      const double b0 = s[4 * stride], b1 = s[5 * stride], b2 = s[6 * stride],
                   b3 = s[7 * stride];
      const double d = kP25 * geo[(half == 0 ? 1 : 0) * gs];  // dyT for x, dxT for y
      const double pa = half == 0 ? a0 + a1 : a0 + a3, pb = half == 0 ? a2 + a3 : a1 + a2;
      const double ma = half == 0 ? b0 + b1 : b0 + b3, mb = half == 0 ? b2 + b3 : b1 + b2;
      const double strp = d * (kP333 * pa + kP166 * pb), strm = d * (kP333 * ma + kP166 * mb);
      const double strq = d * (kP333 * pb + kP166 * pa), strn = d * (kP333 * mb + kP166 * ma);
      if (half == 0) {
        A[0] = -strp - strm;
        A[1] = strp + strm;
        A[2] = -strq - strn;
        A[3] = strq + strn;
      } else {
        A[0] = -strp + strm;
        A[1] = strp - strm;
        A[2] = -strq + strn;
        A[3] = strq - strn;
      }
      const double p1 = (a0 + a2) * kP055, p2 = (a1 + a3) * kP055;
      const double m1 = (b0 + b2) * kP055, m2 = (b1 + b3) * kP055;
      const double pne = kP111 * a0 + p2 + kP027 * a2, pnw = kP111 * a1 + p1 + kP027 * a3;
      const double psw = kP111 * a2 + p2 + kP027 * a0, pse = kP111 * a3 + p1 + kP027 * a1;
      const double mne = kP111 * b0 + m2 + kP027 * b2, mnw = kP111 * b1 + m1 + kP027 * b3;
      const double msw = kP111 * b2 + m2 + kP027 * b0, mse = kP111 * b3 + m1 + kP027 * b1;
      if (half == 0) {  // str1..4: ne, nw, se, sw
        D[0] = -pne + mne;
        D[1] = -pnw + mnw;
        D[2] = -pse + mse;
        D[3] = -psw + msw;
      } else {  // str5..8: ne, se, nw, sw
        D[0] = pne + mne;
        D[1] = pse + mse;
        D[2] = pnw + mnw;
        D[3] = psw + msw;
      }
    }
    hold();
    const double c0 = s[8 * stride], c1 = s[9 * stride], c2 = s[10 * stride], c3 = s[11 * stride];
    const double t1 = (c0 + c2) * kP111, t2 = (c1 + c3) * kP111;
    const double tne = kP222 * c0 + t2 + kP055 * c2, tnw = kP222 * c1 + t1 + kP055 * c3;
    const double tsw = kP222 * c2 + t2 + kP055 * c0, tse = kP222 * c3 + t1 + kP055 * c1;
    const double dxhy = geo[7 * gs], dyhx = geo[8 * gs];
    const double h = kP5 * geo[(half == 0 ? 0 : 1) * gs];  // dxT for x, dyT for y
    const double ta = half == 0 ? c0 + c3 : c0 + c1;       // e, n
    const double tb = half == 0 ? c1 + c2 : c2 + c3;       // w, s
    const double ew = h * (kP333 * ta + kP166 * tb), we = h * (kP333 * tb + kP166 * ta);
    if (half == 0) {
      out[0] = A[0] - ew + dxhy * D[0] + dyhx * tne;
      out[1] = A[1] - we + dxhy * D[1] + dyhx * tnw;
      out[2] = A[2] + ew + dxhy * D[2] + dyhx * tse;
      out[3] = A[3] + we + dxhy * D[3] + dyhx * tsw;
    } else {
      out[4] = A[0] - ew - dyhx * D[0] + dxhy * tne;
      out[5] = A[1] - we - dyhx * D[1] + dxhy * tse;
      out[6] = A[2] + ew - dyhx * D[2] + dxhy * tnw;
      out[7] = A[3] + we - dyhx * D[3] + dxhy * tsw;
    }
    hold();
  }
}

template <int NT, bool kStd, bool kSmemStress>
__global__ void __launch_bounds__(NT, 1) k_resident(ResidentArgs a, Params p) {
  extern __shared__ __align__(16) unsigned char res_raw[];
  using S_t = ResSmem<NT, kSmemStress>;
  S_t &S = *reinterpret_cast<S_t *>(res_raw);
  const int c = threadIdx.x;
  const size_t at = (size_t)blockIdx.x * blockDim.x + c;
  const int slot = a.slot[at];
  const bool own = c < a.cnt[blockIdx.x];
  const uint32_t nbr = a.str_idx[at];
  const uint8_t fl = slot >= 0 ? a.flags[slot] : (uint8_t)(kSkipT | kSkipU);
  const bool actT = !(fl & kSkipT), actU = own && !(fl & kSkipU);
  const bool exported = own && (nbr & kResExport);

  // ---- the point's constants and state ------------------------------------
  int ref[4] = {0, 0, 0, 0};
  double sreg[12];
  if (slot >= 0) {
    const int4 q = reinterpret_cast<const int4 *>(a.corner)[at];
    ref[0] = q.x;
    ref[1] = q.y;
    ref[2] = q.z;
    ref[3] = q.w;
    const Geom g = make_geom(a.sg[0][slot], a.sg[1][slot], a.sg[2][slot], a.sg[3][slot],
                             a.sg[4][slot], a.sg[5][slot], p.deltaminEVP);
    S.geo[0][c] = g.dxT;
    S.geo[1][c] = g.dyT;
    S.geo[2][c] = g.cxp;
    S.geo[3][c] = g.cyp;
    S.geo[4][c] = g.cxm;
    S.geo[5][c] = g.cym;
    S.geo[6][c] = g.DminTarea;
    S.geo[7][c] = g.dxhy;
    S.geo[8][c] = g.dyhx;
    S.geo[9][c] = a.sg[6][slot];
#pragma unroll
    for (int k = 0; k < 12; k++) sreg[k] = a.s_in[k][slot];
  } else {
#pragma unroll
    for (int k = 0; k < 12; k++) sreg[k] = 0.0;
  }
  if (own) {
#pragma unroll
    for (int k = 0; k < kTmaStepuFields; k++) S.cst[k][c] = a.uf[k][slot];
    S.uv[c] = make_double2(a.u_in[slot], a.v_in[slot]);
  }
  if constexpr (kSmemStress) {
#pragma unroll
    for (int k = 0; k < 12; k++) S.s[k][c] = sreg[k];
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    S.str[k][c] = make_double2(0.0, 0.0);  // skipped T points keep str = 0
    if (c == 0) S.str[k][NT] = make_double2(0.0, 0.0);
  }
  __syncthreads();

  unsigned polled = 0;  // corners whose velocity another block owns
#pragma unroll
  for (int k = 0; k < 4; k++) polled |= (ref[k] < 0 && ~ref[k] < a.nslots) ? 1u << k : 0u;
  bool fail = false;
  double2 own_str = make_double2(0.0, 0.0);  // str1, str5
  for (int sub = 0; sub < a.nsub; sub++) {
    const bool wlast = a.last && sub == a.nsub - 1;
    // ---- stress ------------------------------------------------------------
    Mail m[4];  // velocities other blocks own
    if (sub > 0)
      fail |= !mail_wait(m, a.mail + (size_t)(sub & 1) * (size_t)a.nslots, ref,
                         actT ? polled : 0u, a.seq + (unsigned)sub);
    if (actT) {
      double2 w[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (ref[k] >= 0)
          w[k] = S.uv[ref[k]];
        else if (sub > 0 && (polled >> k & 1))
          w[k] = mail_value(m[k]);
        else
          w[k] = make_double2(a.u_in[~ref[k]], a.v_in[~ref[k]]);
      }
      Corners cr;
      cr.ucc = w[0].x;
      cr.vcc = w[0].y;
      cr.uee = w[1].x;
      cr.vee = w[1].y;
      cr.une = w[2].x;
      cr.vne = w[2].y;
      cr.use = w[3].x;
      cr.vse = w[3].y;
      double out[8];
      if constexpr (kSmemStress) {
        stress_lean<kStd>(&S.s[0][c], NT, out, cr, &S.geo[0][c], NT, p);
      } else {
        Geom g;
        g.dxT = S.geo[0][c];
        g.dyT = S.geo[1][c];
        g.cxp = S.geo[2][c];
        g.cyp = S.geo[3][c];
        g.cxm = S.geo[4][c];
        g.cym = S.geo[5][c];
        g.DminTarea = S.geo[6][c];
        g.dxhy = S.geo[7][c];
        g.dyhx = S.geo[8][c];
        stress_point<kStd>(cr, g, S.geo[9][c], sreg, out, p);
      }
      S.str[0][c] = make_double2(out[1], out[6]);
      S.str[1][c] = make_double2(out[2], out[5]);
      S.str[2][c] = make_double2(out[3], out[7]);
      own_str = make_double2(out[0], out[4]);
      if (wlast && own) {
#pragma unroll
        for (int k = 0; k < 8; k++) a.str_out[k][slot] = out[k];
      }
    }
    if (fail) atomicMax(a.err, kResCode);
    if (__syncthreads_or(fail)) return;
    // ---- stepu -------------------------------------------------------------
    if (own) {
      double2 z = S.uv[c];
      if (actU) {
        StepuIn in;
        in.uold = z.x;
        in.vold = z.y;
        in.kvrel = S.cst[0][c];
        in.uocn = S.cst[1][c];
        in.vocn = S.cst[2][c];
        in.waterx = S.cst[3][c];
        in.watery = S.cst[4][c];
        in.forcex = S.cst[5][c];
        in.forcey = S.cst[6][c];
        in.umassdti = S.cst[7][c];
        in.fm = S.cst[8][c];
        in.uarear = S.cst[9][c];
        in.Tbu = S.cst[10][c];
        in.uinit = S.cst[11][c];
        in.vinit = S.cst[12][c];
        const double2 nw = S.str[0][nbr & 1023], sse = S.str[1][(nbr >> 20) & 1023];
        const double2 sw = S.str[2][(nbr >> 10) & 1023];
        in.s1 = own_str.x;
        in.s5 = own_str.y;
        in.s2nw = nw.x;
        in.s7nw = nw.y;
        in.s3sse = sse.x;
        in.s6sse = sse.y;
        in.s4sw = sw.x;
        in.s8sw = sw.y;
        const StepuOut o = stepu_point(in, p);
        z = make_double2(o.u, o.v);
        S.uv[c] = z;
        if (wlast) {
          a.strintx[slot] = o.strintx;
          a.strinty[slot] = o.strinty;
          a.Cb[slot] = o.Cb;
        }
      }
      if (sub + 1 < a.nsub) {
        if (exported)
          mail_put(a.mail + (size_t)((sub + 1) & 1) * (size_t)a.nslots + slot, z.x, z.y,
                   a.seq + (unsigned)sub + 1u);
        if (actU && a.uv_step) {
          a.u_out[(size_t)(sub + 1) * a.uv_step + slot] = z.x;
          a.v_out[(size_t)(sub + 1) * a.uv_step + slot] = z.y;
        }
      } else if (actU) {
        a.u_out[(size_t)a.nsub * a.uv_step + slot] = z.x;
        a.v_out[(size_t)a.nsub * a.uv_step + slot] = z.y;
      }
    }
    __syncthreads();
  }
  // A block comes here only after its neighbours have read its starting state
  // (they sent it a later subcycle's velocities), or writes the other set.
  if (own && actT) {
#pragma unroll
    for (int k = 0; k < 12; k++) {
      if constexpr (kSmemStress)
        a.s_out[k][slot] = S.s[k][c];
      else
        a.s_out[k][slot] = sreg[k];
    }
  }
}

// ---- four lanes per point ---------------------------------------------------
// Lane k of a point's quad has corner k (0 ne, 1 nw, 2 sw, 3 se): its velocity
// (cc, ee, ne, se: one mailbox at most to poll), its strain rates, its
// viscosity and its three stresses.  The sums of str_combine
// (src/bench_v2b.F90:217-310) are symmetric in the corners: with s the own
// corner's stress and s1, s2, s3 those of lanes k^1, k^2, k^3,
//   sides        N = s + s1, N' = s2 + s3 (north/south), E = s + s3,
//                E' = s1 + s2 (east/west)
//   csig         P111*s + P055*(s1 + s3) + P027*s2
//   strp, str12  c * (P333*N + P166*N'), or with E, E'
// and lane k writes the two str of its corner, str1/5, 2/7, 4/8, 3/6, which
// differ in signs only.  Addition commutes and negation is exact, so these are
// the reference's values bit for bit.  stepu runs one thread per point, on the
// block's first warps.  A lane has 130 of stress's 440 FP64 operations, so a
// warp's chain is a third as long; all in all 17 % more operations, on SMs that
// one thread per point leaves four fifths idle.  us per subcycle against one
// thread per point: 2.0k points 1.65 / 2.55, 6.2k 1.70 / 2.53, 13.6k 1.78 / 2.64
// (above 128 points a block the lanes fill the SM, and one thread per point is
// as fast).
struct QuadSmem {
  double2 uv[kQuadMaxWidth];         // velocities of the owned points
  double2 str[4][kQuadMaxWidth + 1];  // by corner: (str1, str5), (2, 7), (4, 8), (3, 6)
  double cst[kTmaStepuFields][kQuadMaxWidth];
};

__device__ __forceinline__ double quad_xor(double x, int mask) {
  return __shfl_xor_sync(0xffffffffu, x, mask);
}

__device__ __forceinline__ double quad_sign(double x, bool negative) {
  return negative ? -x : x;
}

template <int NT, bool kStd>
__global__ void __launch_bounds__(NT, 1) k_resident_quad(ResidentArgs a, Params p) {
  extern __shared__ __align__(16) unsigned char res_raw[];
  QuadSmem &S = *reinterpret_cast<QuadSmem *>(res_raw);
  const int tid = threadIdx.x;
  const int M = blockDim.x >> 2;
  const int c = tid >> 2, k = tid & 3;  // the stress point and corner
  const int cnt = a.cnt[blockIdx.x];
  const size_t at = (size_t)blockIdx.x * M + c;
  const int slot = a.slot[at];
  const bool actT = slot >= 0 && !(a.flags[slot] & kSkipT);
  // the stepu point of this thread
  const bool own = tid < cnt;
  const size_t uat = (size_t)blockIdx.x * M + (own ? tid : 0);
  const int uslot = a.slot[uat];
  const uint32_t nbr = a.str_idx[uat];
  const bool actU = own && !(a.flags[uslot] & kSkipU);
  const bool exported = own && (nbr & kResExport);

  // ---- constants and state --------------------------------------------------
  int ref = 0;  // where the corner's velocity is (ResidentPlan::corner)
  Geom g = {};
  double strength = 0.0, sp = 0.0, sm = 0.0, st = 0.0;
  if (slot >= 0) {
    ref = a.corner[4 * at + k];
    g = make_geom(a.sg[0][slot], a.sg[1][slot], a.sg[2][slot], a.sg[3][slot], a.sg[4][slot],
                  a.sg[5][slot], p.deltaminEVP);
    strength = a.sg[6][slot];
    sp = a.s_in[k][slot];
    sm = a.s_in[4 + k][slot];
    st = a.s_in[8 + k][slot];
  }
  const bool polled = slot >= 0 && ref < 0 && ~ref < a.nslots;
  const bool ew = (k == 0) | (k == 3), ns = k < 2;
  if (own) {
#pragma unroll
    for (int f = 0; f < kTmaStepuFields; f++) S.cst[f][tid] = a.uf[f][uslot];
    S.uv[tid] = make_double2(a.u_in[uslot], a.v_in[uslot]);
  }
  if (c < M) S.str[k][c] = make_double2(0.0, 0.0);  // skipped T points keep str = 0
  if (tid < 4) S.str[tid][kQuadMaxWidth] = make_double2(0.0, 0.0);
  __syncthreads();

  bool fail = false;
  for (int sub = 0; sub < a.nsub; sub++) {
    const bool wlast = a.last && sub == a.nsub - 1;
    // ---- stress: whole warps (the shuffles), results of active points only ---
    double2 w = make_double2(0.0, 0.0);
    const bool wait = actT && polled && sub > 0;
    if (actT && !wait) w = ref >= 0 ? S.uv[ref] : make_double2(a.u_in[~ref], a.v_in[~ref]);
    // The warp polls together and stays converged (lanes that left a loop of
    // their own one by one went through the rest of the stress one after the
    // other: 4.7 us a subcycle instead of 1.65).
    if (__any_sync(0xffffffffu, wait)) {
      const unsigned seq = a.seq + (unsigned)sub;
      const double4 *box =
          a.mail + (size_t)(sub & 1) * (size_t)a.nslots + (wait ? ~ref : 0);
      bool left = wait;
      unsigned long long t0 = 0;
      for (unsigned tries = 1;; tries++) {
        if (left) {
          const Mail m = mail_get(box);
          if (mail_is(m, seq)) {
            w = mail_value(m);
            left = false;
          }
        }
        if (!__any_sync(0xffffffffu, left)) break;
        if ((tries & 63u) == 0) {
          const unsigned long long t = res_ns();
          if (t0 == 0) t0 = t;
          if (__any_sync(0xffffffffu, t - t0 > kResWaitNs)) {
            fail = left;
            break;
          }
        }
      }
    }
    const double u2 = quad_xor(w.x, 1), v2 = quad_xor(w.y, 1);
    const double u4 = quad_xor(w.x, 3), v4 = quad_xor(w.y, 3);
    double div, ten, shr, sq;
    corner_strain_sq(k, w.x, w.y, u2, v2, u4, v4, g, p.e_factor, div, ten, shr, sq);
    double Delta = 0.0;
    const bool fast = fp64_dividend(strength) & fp64_mid(g.DminTarea) & fp64_radicand(sq) &
                      (kStd | (p.capping == kC1) | (p.capping == 0.0));
    Delta = fp64_sqrt(sq);
    const bool capped = kStd || p.capping == kC1;
    const double den = capped ? fmax_ref(Delta, g.DminTarea) : Delta + g.DminTarea;
    const double visc = fp64_quot(strength, den, fp64_recip(den));
    if (actT) {
      if (fast)
        corner_relax<kStd>(sp, sm, st, div, ten, shr, Delta, visc, p);
      else
        corner_update(sp, sm, st, div, ten, shr, sqrt(sq), strength, g.DminTarea, p);
    }
    __syncwarp();
    const double p1 = quad_xor(sp, 1), p2 = quad_xor(sp, 2), p3 = quad_xor(sp, 3);
    const double m1 = quad_xor(sm, 1), m2 = quad_xor(sm, 2), m3 = quad_xor(sm, 3);
    const double t1 = quad_xor(st, 1), t2 = quad_xor(st, 2), t3 = quad_xor(st, 3);
    if (actT) {
      const double pN = sp + p1, pS = p2 + p3, pE = sp + p3, pW = p1 + p2;
      const double mN = sm + m1, mS = m2 + m3, mE = sm + m3, mW = m1 + m2;
      const double tN = st + t1, tS = t2 + t3, tE = st + t3, tW = t1 + t2;
      const double cp = kP111 * sp + (p1 + p3) * kP055 + kP027 * p2;
      const double cm = kP111 * sm + (m1 + m3) * kP055 + kP027 * m2;
      const double ct = kP222 * st + (t1 + t3) * kP111 + kP055 * t2;
      const double dx = g.dxT, dy = g.dyT;
      const double tx = kP5 * dx * (kP333 * tE + kP166 * tW);
      const double ty = kP5 * dy * (kP333 * tN + kP166 * tS);
      const double px = kP25 * dy * (kP333 * pN + kP166 * pS);
      const double mx = kP25 * dy * (kP333 * mN + kP166 * mS);
      const double py = kP25 * dx * (kP333 * pE + kP166 * pW);
      const double my = kP25 * dx * (kP333 * mE + kP166 * mW);
      // ne, se: -strp - strm; nw, sw: +strp + strm; north: -str12, south: +
      const double ox = quad_sign(px, ew) + quad_sign(mx, ew) + quad_sign(tx, ns) +
                        g.dxhy * (-cp + cm) + g.dyhx * ct;
      // north: -strp + strm; south: +strp - strm; east: -str12, west: +
      const double oy = quad_sign(py, ns) + quad_sign(my, !ns) + quad_sign(ty, ew) -
                        g.dyhx * (cp + cm) + g.dxhy * ct;
      S.str[k][c] = make_double2(ox, oy);
      if (wlast && c < cnt) {
        // str1/5, str2/7, str4/8, str3/6
        const int ix = ns ? k : 5 - k, iy = k == 0 ? 4 : k == 1 ? 6 : k == 2 ? 7 : 5;
        a.str_out[ix][slot] = ox;
        a.str_out[iy][slot] = oy;
      }
    }
    if (fail) atomicMax(a.err, kResCode);
    if (__syncthreads_or(fail)) return;
    // ---- stepu ---------------------------------------------------------------
    if (own) {
      double2 z = S.uv[tid];
      if (actU) {
        StepuIn in;
        in.uold = z.x;
        in.vold = z.y;
        in.kvrel = S.cst[0][tid];
        in.uocn = S.cst[1][tid];
        in.vocn = S.cst[2][tid];
        in.waterx = S.cst[3][tid];
        in.watery = S.cst[4][tid];
        in.forcex = S.cst[5][tid];
        in.forcey = S.cst[6][tid];
        in.umassdti = S.cst[7][tid];
        in.fm = S.cst[8][tid];
        in.uarear = S.cst[9][tid];
        in.Tbu = S.cst[10][tid];
        in.uinit = S.cst[11][tid];
        in.vinit = S.cst[12][tid];
        const double2 s0 = S.str[0][tid], nw = S.str[1][nbr & 1023];
        const double2 sw = S.str[2][(nbr >> 10) & 1023], sse = S.str[3][(nbr >> 20) & 1023];
        in.s1 = s0.x;
        in.s5 = s0.y;
        in.s2nw = nw.x;
        in.s7nw = nw.y;
        in.s3sse = sse.x;
        in.s6sse = sse.y;
        in.s4sw = sw.x;
        in.s8sw = sw.y;
        const StepuOut o = stepu_point(in, p);
        z = make_double2(o.u, o.v);
        S.uv[tid] = z;
        if (wlast) {
          a.strintx[uslot] = o.strintx;
          a.strinty[uslot] = o.strinty;
          a.Cb[uslot] = o.Cb;
        }
      }
      if (sub + 1 < a.nsub) {
        if (exported)
          mail_put(a.mail + (size_t)((sub + 1) & 1) * (size_t)a.nslots + uslot, z.x, z.y,
                   a.seq + (unsigned)sub + 1u);
        if (actU && a.uv_step) {
          a.u_out[(size_t)(sub + 1) * a.uv_step + uslot] = z.x;
          a.v_out[(size_t)(sub + 1) * a.uv_step + uslot] = z.y;
        }
      } else if (actU) {
        a.u_out[(size_t)a.nsub * a.uv_step + uslot] = z.x;
        a.v_out[(size_t)a.nsub * a.uv_step + uslot] = z.y;
      }
    }
    __syncthreads();
  }
  if (c < cnt && actT) {  // (see k_resident)
    a.s_out[k][slot] = sp;
    a.s_out[4 + k][slot] = sm;
    a.s_out[8 + k][slot] = st;
  }
}

using ResKernel = void (*)(ResidentArgs, Params);
struct ResVariant {
  int width;
  ResKernel k[2];  // [kStd]
  size_t smem;
};
template <int NT, bool kSmemStress>
constexpr ResVariant variant() {
  return {NT, {k_resident<NT, false, kSmemStress>, k_resident<NT, true, kSmemStress>},
          sizeof(ResSmem<NT, kSmemStress>)};
}
// 640 threads leave 96 registers each: the stresses go to shared memory there.
// At 512 they stay in registers (4.2 us per subcycle against 5.6 from shared
// memory, 63.8k points: the extra 48 shared-memory accesses a point cost more
// than 36 bytes of spills).
const ResVariant kVariants[] = {variant<128, false>(), variant<256, false>(),
                                variant<384, false>(), variant<512, false>(),
                                variant<640, true>()};
static_assert(sizeof(ResSmem<640, true>) <= 227 * 1024, "shared memory per block");

// The class of a quad plan is kQuadMaxWidth, of four threads a point.
const ResVariant kQuad = {4 * kQuadMaxWidth,
                          {k_resident_quad<4 * kQuadMaxWidth, false>,
                           k_resident_quad<4 * kQuadMaxWidth, true>},
                          sizeof(QuadSmem)};

const ResVariant *find_variant(bool quad, int cls) {
  if (quad) return cls == kQuadMaxWidth ? &kQuad : nullptr;
  for (const ResVariant &v : kVariants)
    if (v.width == cls) return &v;
  return nullptr;
}

}  // namespace

int resident_prepare(int device, bool quad, int cls, int nblocks) {
  const ResVariant *v = find_variant(quad, cls);
  if (!v) return 0;
  int coop = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 2 && e == cudaSuccess; k++)
    e = cudaFuncSetAttribute(v->k[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v->smem);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v->k[1], v->width, v->smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return coop && nblocks <= sms * per_sm ? 1 : 0;
}

cudaError_t launch_resident(const ResidentArgs &given, const Params &p, bool quad, int cls,
                            int threads, int nblocks, cudaStream_t st) {
  const ResVariant *v = find_variant(quad, cls);
  if (!v || nblocks <= 0 || given.nsub <= 0) return cudaErrorInvalidValue;
  ResidentArgs a = given;
  Params pp = p;
  void *args[] = {&a, &pp};
  return cudaLaunchCooperativeKernel((const void *)v->k[std_params(p) ? 1 : 0], dim3(nblocks),
                                     dim3(quad ? 4 * threads : threads), args, v->smem, st);
}

}  // namespace evp
