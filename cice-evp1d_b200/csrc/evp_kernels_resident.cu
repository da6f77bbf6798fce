// evp_kernels_resident.cu -- a call's subcycles in one launch, for problems
// small enough to stay on chip (evp_resident.h).
//
// One CTA per block of the resident plan, one thread per compute point (owned
// points, then the forward halo).  A thread keeps its point's 12 stresses in
// registers and its constants in shared memory from the first subcycle to the
// last; only velocities move between blocks.
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
// stress n, and they include every block that waits for this one (the plan
// requires inverse neighbour relations, which make waiting mutual whatever
// the mask: inverse_relations in evp_resident.cpp).
// The CTAs wait on one another, so the launch is cooperative (all resident or
// none).  Every wait is bounded: on expiry the code goes to the error word,
// the CTA leaves together at the next barrier, and its neighbours' waits run
// out in turn.
//
// What bounds it: the FP64 pipe (about 535 operations a point, two issue
// cycles each, 64 lanes an SM) for full blocks, the dependent chain through
// stress, stepu and the exchange for small ones; no HBM traffic per subcycle.
// Measured, us per subcycle, against the one-launch-per-subcycle kernel (before
// the straight-line divisions of evp_fp64.cuh): 18k points 2.6 / 5.0, 51k 3.3 /
// 7.8, 64k 3.9 / 8.0; smaller problems: k_resident_quad.
// Above 512 positions a block (70k points on 148 SMs) a thread for each would
// leave a thread 96 registers, which cannot hold the stresses: 640 threads with
// them in shared memory took 6.05 us at 74k points.  Instead 512 threads keep
// the registers, and the positions beyond take four lanes each (below), which
// need few: 5.1 us there (9.9 with a launch per subcycle), 5.7 / 9.9 at 79k,
// 6.7 / 10.0 at 89k.  Three choices matter: those positions are interior points
// and go first, so that their chain runs while other warps wait for their
// mailboxes (last, as halo points: 6.5 at 74k); blocks own at most 512 points
// where that fits, so that stepu is one pass; and where it is two, the exported
// points are in the first.
#include <algorithm>
#include <cstdint>

#include "evp_internal.h"
#include "evp_resident_mail.cuh"

namespace evp {

namespace {

constexpr int kResGeo = 10;  // dxT dyT cxp cyp cxm cym DminTarea dxhy dyhx strength

// EX > 0: blocks of up to NT + EX positions.  The first M - NT of them ("extra"
// positions: interior points, whose stress waits for no other block) take four
// lanes each, before the threads' own points.
template <int NT, int EX>
struct ResSmem {
  double2 uv[NT + EX];  // velocities of the owned points
  // (str2, str7), (str3, str6), (str4, str8), EX: (str1, str5); the last stays 0
  double2 str[EX ? 4 : 3][NT + EX + 1];
  double geo[kResGeo][NT + EX];
  double cst[kTmaStepuFields][NT + EX];
  uint32_t nbr[EX ? NT + EX : 1];  // str positions, kResExport, kResSkipU
  // extra positions: stresses and velocity references by lane, flags
  double xs[3][EX ? 4 * EX : 1];
  int xref[EX ? 4 * EX : 1];
  uint8_t xfl[EX ? EX : 1];
};
constexpr uint32_t kResSkipU = 1u << 31;

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
__device__ __forceinline__ double quad_xor(double x, int mask) {
  return __shfl_xor_sync(0xffffffffu, x, mask);
}

__device__ __forceinline__ double quad_sign(double x, bool negative) {
  return negative ? -x : x;
}

// The velocity a lane's corner reads, for the whole warp (`act`: the lane has a
// point).  It polls together and stays converged (lanes that left a loop of
// their own one by one went through the rest of the stress one after the other:
// 4.7 us a subcycle instead of 1.65).
__device__ __forceinline__ double2 quad_velocity(const double2 *uv, const ResidentArgs &a, int sub,
                                                 int ref, bool act, bool &fail) {
  double2 w = make_double2(0.0, 0.0);
  const bool wait = act && sub > 0 && ref < 0 && ~ref < a.nslots;
  if (act && !wait) w = ref >= 0 ? uv[ref] : make_double2(a.u_in[~ref], a.v_in[~ref]);
  const double4 *box = a.mail + (size_t)(sub & 1) * (size_t)a.nslots + (wait ? ~ref : 0);
  fail |= mail_wait_one(w, box, wait, a.seq + (unsigned)sub);
  return w;
}

// The stress of corner k of a point on its quad (whole warps): the corner's
// stresses in place, its two str in `o`.
template <bool kStd>
__device__ __forceinline__ void quad_stress(int k, bool act, double2 w, const Geom &g,
                                            double strength, double &sp, double &sm, double &st,
                                            double2 &o, const Params &p) {
  const bool ew = (k == 0) | (k == 3), ns = k < 2;
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
  if (act) {
    if (fast)
      corner_relax<kStd>(sp, sm, st, div, ten, shr, Delta, visc, p);
    else
      corner_update(sp, sm, st, div, ten, shr, sqrt(sq), strength, g.DminTarea, p);
  }
  __syncwarp();
  const double p1 = quad_xor(sp, 1), p2 = quad_xor(sp, 2), p3 = quad_xor(sp, 3);
  const double m1 = quad_xor(sm, 1), m2 = quad_xor(sm, 2), m3 = quad_xor(sm, 3);
  const double t1 = quad_xor(st, 1), t2 = quad_xor(st, 2), t3 = quad_xor(st, 3);
  if (act) {
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
    o = make_double2(ox, oy);
  }
}

__device__ __forceinline__ Geom load_geom(const double *geo, int gs) {
  Geom g;
  g.dxT = geo[0 * gs];
  g.dyT = geo[1 * gs];
  g.cxp = geo[2 * gs];
  g.cyp = geo[3 * gs];
  g.cxm = geo[4 * gs];
  g.cym = geo[5 * gs];
  g.DminTarea = geo[6 * gs];
  g.dxhy = geo[7 * gs];
  g.dyhx = geo[8 * gs];
  return g;
}

// A position's constants in shared memory.
template <class Smem>
__device__ __forceinline__ void load_position(Smem &S, const ResidentArgs &a, const Params &p,
                                              int c, int slot, bool own) {
  if (slot >= 0) {
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
  }
  if (own) {
#pragma unroll
    for (int k = 0; k < kTmaStepuFields; k++) S.cst[k][c] = a.uf[k][slot];
    S.uv[c] = make_double2(a.u_in[slot], a.v_in[slot]);
  }
#pragma unroll
  for (int k = 0; k < (int)(sizeof S.str / sizeof S.str[0]); k++)
    S.str[k][c] = make_double2(0.0, 0.0);  // skipped T points keep str = 0
}

// stepu of owned position c, and where its velocity goes.
template <class Smem>
__device__ __forceinline__ void step_position(Smem &S, const ResidentArgs &a, const Params &p,
                                              int sub, bool wlast, int c, int slot, uint32_t nbr,
                                              double2 own_str) {
  const bool actU = !(nbr & kResSkipU);
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
    if (nbr & kResExport)
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

// The two str of corner k (0 ne, 1 nw, 2 sw, 3 se) of a point: str1/5, 2/7,
// 4/8, 3/6.
__device__ __forceinline__ void store_str(const ResidentArgs &a, int k, int slot, double2 o) {
  const int ix = k < 2 ? k : 5 - k, iy = k == 0 ? 4 : k == 1 ? 6 : k == 2 ? 7 : 5;
  a.str_out[ix][slot] = o.x;
  a.str_out[iy][slot] = o.y;
}

template <int NT, bool kStd, int EX>
__global__ void __launch_bounds__(NT, 1) k_resident(ResidentArgs a, Params p) {
  extern __shared__ __align__(16) unsigned char res_raw[];
  using S_t = ResSmem<NT, EX>;
  S_t &S = *reinterpret_cast<S_t *>(res_raw);
  const int tid = threadIdx.x;
  const int M = EX ? a.width : (int)blockDim.x;  // positions per block
  const int nx = EX ? M - NT : 0;                // extra ones
  const int cnt = a.cnt[blockIdx.x];
  const size_t base = (size_t)blockIdx.x * M;
  // the position whose stress the thread does; its stepu is that of position
  // u0 + tid: the last NT owned ones (among them the exported ones, which the
  // neighbours wait for), then, if there are more, the first u0
  const int c = nx + tid;
  const int u0 = EX ? max(0, cnt - NT) : 0;
  const int slot = a.slot[base + c];
  const bool own = c < cnt;
  const uint8_t fl = slot >= 0 ? a.flags[slot] : (uint8_t)(kSkipT | kSkipU);
  const bool actT = !(fl & kSkipT);
  uint32_t nbr = a.str_idx[base + c] | (fl & kSkipU ? kResSkipU : 0u);

  // ---- constants and state --------------------------------------------------
  int ref[4] = {0, 0, 0, 0};
  double sreg[12];
  if (slot >= 0) {
    const int4 q = reinterpret_cast<const int4 *>(a.corner)[base + c];
    ref[0] = q.x;
    ref[1] = q.y;
    ref[2] = q.z;
    ref[3] = q.w;
  }
#pragma unroll
  for (int k = 0; k < 12; k++) sreg[k] = slot >= 0 ? a.s_in[k][slot] : 0.0;
  load_position(S, a, p, c, slot, own);
  if (tid < (EX ? 4 : 3)) S.str[tid][NT + EX] = make_double2(0.0, 0.0);
  if constexpr (EX > 0) {
    S.nbr[c] = nbr;
    for (int e = tid; e < nx; e += NT) {
      const int xslot = a.slot[base + e];
      load_position(S, a, p, e, xslot, e < cnt);
      S.xfl[e] = xslot >= 0 ? a.flags[xslot] : (uint8_t)(kSkipT | kSkipU);
      S.nbr[e] = a.str_idx[base + e] | (S.xfl[e] & kSkipU ? kResSkipU : 0u);
      for (int k = 0; k < 4; k++) {
        S.xref[4 * e + k] = xslot >= 0 ? a.corner[4 * (base + e) + k] : 0;
        for (int f = 0; f < 3; f++)
          S.xs[f][4 * e + k] = xslot >= 0 ? a.s_in[4 * f + k][xslot] : 0.0;
      }
    }
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
    if constexpr (EX > 0) {
      for (int r = tid & ~31; r < 4 * nx; r += NT) {  // whole warps
        const int l = r + (tid & 31), e = l >> 2, k = l & 3;
        const bool act = !(S.xfl[e] & kSkipT);
        const double2 w = quad_velocity(S.uv, a, sub, S.xref[l], act, fail);
        const Geom g = load_geom(&S.geo[0][e], NT + EX);
        double sp = S.xs[0][l], sm = S.xs[1][l], st = S.xs[2][l];
        double2 o;
        quad_stress<kStd>(k, act, w, g, S.geo[9][e], sp, sm, st, o, p);
        if (act) {
          S.xs[0][l] = sp;
          S.xs[1][l] = sm;
          S.xs[2][l] = st;
          S.str[k == 0 ? 3 : k == 1 ? 0 : 4 - k][e] = o;
          if (wlast && e < cnt) store_str(a, k, a.slot[base + e], o);
        }
      }
    }
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
      const Geom g = load_geom(&S.geo[0][c], NT + EX);
      stress_point<kStd>(cr, g, S.geo[9][c], sreg, out, p);
      S.str[0][c] = make_double2(out[1], out[6]);
      S.str[1][c] = make_double2(out[2], out[5]);
      S.str[2][c] = make_double2(out[3], out[7]);
      own_str = make_double2(out[0], out[4]);
      if constexpr (EX > 0) S.str[3][c] = own_str;
      if (wlast && own) {
#pragma unroll
        for (int k = 0; k < 8; k++) a.str_out[k][slot] = out[k];
      }
    }
    if (fail) atomicMax(a.err, kResCode);
    if (__syncthreads_or(fail)) return;
    // ---- stepu -------------------------------------------------------------
    if constexpr (EX > 0) {
      for (int q = u0 + tid; q < cnt; q = q >= u0 && tid < u0 ? tid : cnt)
        step_position(S, a, p, sub, wlast, q, a.slot[base + q], S.nbr[q], S.str[3][q]);
    } else {
      if (own) step_position(S, a, p, sub, wlast, c, slot, nbr, own_str);
    }
    __syncthreads();
  }
  // A block comes here only after its neighbours have read its starting state
  // (they sent it a later subcycle's velocities), or writes the other set.
  if (own && actT) {
#pragma unroll
    for (int k = 0; k < 12; k++) a.s_out[k][slot] = sreg[k];
  }
  if constexpr (EX > 0) {
    for (int l = tid; l < 4 * min(nx, cnt); l += NT) {
      if (S.xfl[l >> 2] & kSkipT) continue;
      const int xslot = a.slot[base + (l >> 2)];
      for (int f = 0; f < 3; f++) a.s_out[4 * f + (l & 3)][xslot] = S.xs[f][l];
    }
  }
}

// ---- every point on four lanes ------------------------------------------------
struct QuadSmem {
  double2 uv[kQuadMaxWidth];         // velocities of the owned points
  double2 str[4][kQuadMaxWidth + 1];  // by corner: (str1, str5), (2, 7), (4, 8), (3, 6)
  double cst[kTmaStepuFields][kQuadMaxWidth];
};

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
    const double2 w = quad_velocity(S.uv, a, sub, ref, actT, fail);
    double2 o;
    quad_stress<kStd>(k, actT, w, g, strength, sp, sm, st, o, p);
    if (actT) {
      S.str[k][c] = o;
      if (wlast && c < cnt) store_str(a, k, slot, o);
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
  int cls, threads;  // positions, most threads per block
  ResKernel k[2];    // [kStd]
  size_t smem;
};
template <int NT, int EX>
constexpr ResVariant variant() {
  return {NT + EX, NT, {k_resident<NT, false, EX>, k_resident<NT, true, EX>},
          sizeof(ResSmem<NT, EX>)};
}
const ResVariant kVariants[] = {variant<128, 0>(), variant<256, 0>(), variant<384, 0>(),
                                variant<kResMaxThreads, 0>(),
                                variant<kResMaxThreads, kResMaxWidth - kResMaxThreads>()};
static_assert(sizeof(ResSmem<kResMaxThreads, kResMaxWidth - kResMaxThreads>) <= 227 * 1024, "shared memory per block");

// One warp waits, as the resident kernels do, for messages that nobody sends:
// lane l's velocities are those of slots 0 .. nslots - 1 in turn.  Both forms of
// the wait must run out.
__global__ void k_mail_probe(int *err, const double4 *mail, int nslots, unsigned seq,
                             unsigned long long limit_ns) {
  const int l = threadIdx.x;
  int ref[4];
  for (int k = 0; k < 4; k++) ref[k] = ~((4 * l + k) % nslots);
  Mail m[4];
  const bool came = mail_wait(m, mail, ref, l < 8 ? 15u : 0u, seq, limit_ns);
  double2 w = make_double2(0.0, 0.0);
  const bool out = mail_wait_one(w, mail + ~ref[0], l < 8, seq, limit_ns);
  if (!came && out) atomicMax(err, kMailProbeCode);
}

// The class of a quad plan is kQuadMaxWidth, of four threads a point.
const ResVariant kQuad = {kQuadMaxWidth, 4 * kQuadMaxWidth,
                          {k_resident_quad<4 * kQuadMaxWidth, false>,
                           k_resident_quad<4 * kQuadMaxWidth, true>},
                          sizeof(QuadSmem)};

const ResVariant *find_variant(bool quad, int cls) {
  if (quad) return cls == kQuadMaxWidth ? &kQuad : nullptr;
  for (const ResVariant &v : kVariants)
    if (v.cls == cls) return &v;
  return nullptr;
}

}  // namespace

void launch_mail_probe(int *err, const double4 *mail, int nslots, unsigned seq,
                       unsigned long long limit_ns, cudaStream_t st) {
  k_mail_probe<<<1, 32, 0, st>>>(err, mail, nslots, seq, limit_ns);
}

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
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v->k[1], v->threads, v->smem);
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
  a.width = threads;
  Params pp = p;
  void *args[] = {&a, &pp};
  return launch_cooperative((const void *)v->k[std_params(p) ? 1 : 0], dim3(nblocks),
                            dim3(quad ? 4 * threads : std::min(threads, v->threads)), args,
                            v->smem, st);
}

}  // namespace evp
