// evp_adjoint_resident.cu -- the reverse sweep's subcycles in one launch, on
// the resident plan of the forward (evp_resident.h, evp_kernels_resident.cu).
//
// On a grid the reverse of a subcycle has the forward's own shape.  A T point
// reads lam of str1..str8 from its own U point and those at ee, ne and se (the
// points that read its str as nw, sw and sse): the places where its forward
// read velocities.  A U point reads the corner shares of lam of its velocity
// from its own T point and those at nw, sw and sse: the places where its
// forward read str.  So the blocks, the forward halo (T points reversed in
// every block that reads their shares, from the same inputs and with the same
// results) and the mailboxes carry over, with (Lx, Ly) = uarear * lam of
// (strintx, strinty) in the place of (u, v) and the corner shares in the
// place of str1..str8.  Per subcycle:
//   stepu reversed (owned points): completes lam of the new velocity from the
//           shares, writes Lx, Ly to shared memory and, for a point other
//           blocks read, to its mailbox;
//   barrier
//   stress reversed (owned and halo points): the 12 stress adjoints stay in
//           registers; the forward's velocities come from the tape;
//   barrier
// A block's halo points start from its neighbour's stress adjoints, which the
// neighbour overwrites at its end: after this block's first message, and this
// block sends none before the barrier that its halo threads reach with their
// loads complete.
//
// What bounds it: the dependent chain through both reversals and one exchange
// a subcycle, 3.3 us where the two kernels of a subcycle took 8 (18.7k points).
// Blocks of 512 hold 128 registers a thread, too few for the 12 stress adjoints
// beside a corner's reversal: 580 bytes of a thread are spilled, to L1 (blocks
// of 384: 44 bytes); 7.3 us a subcycle at 54k points, against 10.3 in the two
// kernels.
#include <cstdint>

#include "evp_adjoint_math.cuh"
#include "evp_internal.h"
#include "evp_resident_mail.cuh"

namespace evp {

namespace {

template <int NT>
struct AdjSmem {
  double2 lam[NT];         // Lx, Ly of the owned points
  double2 share[3][NT + 1];  // lam of (u, v) at ee, ne, se of a T point; [NT] stays 0
  double2 uv[NT];          // the owned points' velocities before the subcycle
  double geo[10][NT];      // dxT dyT cxp cyp cxm cym DminTarea dxhy dyhx strength
  double cst[10][NT];      // kvrel aiu*rhow uocn vocn waterx watery umassdti fm Tbu uarear
  double acc[6][NT];       // Pu Pv, gradients of Cw, forcex, forcey, strength
};

template <int NT>
__global__ void __launch_bounds__(NT, 1) k_resident_adj(ResidentAdjArgs a, Params p) {
  extern __shared__ __align__(16) unsigned char adj_raw[];
  AdjSmem<NT> &S = *reinterpret_cast<AdjSmem<NT> *>(adj_raw);
  const int c = threadIdx.x;
  // whole warps: a plan of four lanes a point may have a width that is none
  const size_t at = (size_t)blockIdx.x * a.width + c;
  const int slot = c < a.width ? a.slot[at] : -1;
  const bool own = c < a.cnt[blockIdx.x];
  const uint32_t nbr = own ? a.str_idx[at] : 0u;
  const uint8_t fl = slot >= 0 ? a.flags[slot] : (uint8_t)(kSkipT | kSkipU);
  const bool actT = !(fl & kSkipT), actU = own && !(fl & kSkipU);
  const bool exported = own && (nbr & kResExport);
  const int inw = nbr & 1023, isw = (nbr >> 10) & 1023, isse = (nbr >> 20) & 1023;

  int ref[4] = {0, 0, 0, 0};
  double ls[12];
  if (slot >= 0) {
    const int4 q = reinterpret_cast<const int4 *>(a.corner)[at];
    ref[0] = q.x;
    ref[1] = q.y;
    ref[2] = q.z;
    ref[3] = q.w;
    const Geom g = make_geom_fw(a.sg[0][slot], a.sg[1][slot], a.sg[2][slot], a.sg[3][slot],
                                a.sg[4][slot], a.sg[5][slot], p.deltaminEVP);
    const double gg[10] = {g.dxT, g.dyT, g.cxp, g.cyp, g.cxm, g.cym,
                           g.DminTarea, g.dxhy, g.dyhx, a.sg[6][slot]};
#pragma unroll
    for (int k = 0; k < 10; k++) S.geo[k][c] = gg[k];
#pragma unroll
    for (int k = 0; k < 12; k++) ls[k] = a.LS[k][slot];
  } else {
#pragma unroll
    for (int k = 0; k < 12; k++) ls[k] = 0.0;
  }
  unsigned polled = 0;  // corners whose point another block owns
#pragma unroll
  for (int k = 0; k < 4; k++) polled |= (ref[k] < 0 && ~ref[k] < a.nslots) ? 1u << k : 0u;
  // the corner shares of the owned points' velocity lam: from the arrays at
  // first, then from the block's table
  double2 own_share = make_double2(0.0, 0.0), s_nw = own_share, s_sw = own_share,
          s_sse = own_share;
  double2 unew = own_share, uold = own_share;
  if (own) {
    const double cc[10] = {a.kvrel[slot],  a.aiu[slot] * p.rhow, a.uocn[slot],
                           a.vocn[slot],   a.waterx[slot],       a.watery[slot],
                           a.umassdti[slot], a.fm[slot],         a.Tbu[slot],
                           a.uarear[slot]};
#pragma unroll
    for (int k = 0; k < 10; k++) S.cst[k][c] = cc[k];
    S.acc[0][c] = a.Pu[slot];
    S.acc[1][c] = a.Pv[slot];
    S.acc[2][c] = a.gC[slot];
    S.acc[3][c] = a.gx[slot];
    S.acc[4][c] = a.gy[slot];
    S.acc[5][c] = a.gs[slot];
    own_share = make_double2(a.C8[0][slot], a.C8[1][slot]);
    s_nw = make_double2(a.C8[2][slot], a.C8[3][slot]);
    s_sw = make_double2(a.C8[4][slot], a.C8[5][slot]);
    s_sse = make_double2(a.C8[6][slot], a.C8[7][slot]);
    const size_t e = (size_t)a.nsub * a.step + slot;
    unew = make_double2(a.tu[e], a.tv[e]);
    uold = make_double2(a.tu[e - a.step], a.tv[e - a.step]);
    S.uv[c] = uold;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    S.share[k][c] = make_double2(0.0, 0.0);  // skipped T points have no shares
    if (c == 0) S.share[k][NT] = make_double2(0.0, 0.0);
  }
  // the barrier's operand depends on every loaded stress adjoint: none is still
  // on its way when a message goes out
  int seen = 0;
#pragma unroll
  for (int k = 0; k < 12; k++) seen |= __double2hiint(ls[k]);
  __syncthreads_or(seen);

  bool fail = false;
  for (int it = 0; it < a.nsub; it++) {
    const int n = a.nsub - 1 - it;
    const double *tu = a.tu + (size_t)n * a.step, *tv = a.tv + (size_t)n * a.step;
    double4 *box = a.mail + (size_t)(it & 1) * (size_t)a.nslots;
    double2 next = make_double2(0.0, 0.0);  // the velocities one subcycle earlier
    if (own && n > 0) next = make_double2(tu[(ptrdiff_t)slot - (ptrdiff_t)a.step],
                                          tv[(ptrdiff_t)slot - (ptrdiff_t)a.step]);
    // ---- stepu reversed ------------------------------------------------------
    if (own) {
      // velocity_lam's sum, in its order
      const double lu = S.acc[0][c] + own_share.x + s_nw.x + s_sw.x + s_sse.x;
      const double lv = S.acc[1][c] + own_share.y + s_nw.y + s_sw.y + s_sse.y;
      double2 l = make_double2(0.0, 0.0);
      if (actU) {
        StepuAdjIn in;
        in.uold = uold.x;
        in.vold = uold.y;
        in.unew = unew.x;
        in.vnew = unew.y;
        in.lun = lu;
        in.lvn = lv;
        in.kvrel = S.cst[0][c];
        in.aiXrhow = S.cst[1][c];
        in.uocn = S.cst[2][c];
        in.vocn = S.cst[3][c];
        in.waterx = S.cst[4][c];
        in.watery = S.cst[5][c];
        in.umassdti = S.cst[6][c];
        in.fm = S.cst[7][c];
        in.Tbu = S.cst[8][c];
        bool ok = true;
        StepuAdjOut o = stepu_adjoint_t<true>(in, p, &ok);
        if (!ok) o = stepu_adjoint(in, p);
        S.acc[0][c] = o.luold;
        S.acc[1][c] = o.lvold;
        S.acc[2][c] += o.gCw;
        S.acc[3][c] += o.lcc1;
        S.acc[4][c] += o.lcc2;
        const double ar = S.cst[9][c];
        l = make_double2(ar * o.lcc1, ar * o.lcc2);
      } else {  // a skipped point passes lam on
        S.acc[0][c] = lu;
        S.acc[1][c] = lv;
      }
      S.lam[c] = l;
      if (exported) mail_put(box + slot, l.x, l.y, a.seq + (unsigned)it);
    }
    __syncthreads();
    // ---- stress reversed -----------------------------------------------------
    Mail m[4];
    fail |= !mail_wait(m, box, ref, actT ? polled : 0u, a.seq + (unsigned)it);
    if (actT) {
      double2 w[4];  // velocities of cc, ee, ne, se
#pragma unroll
      for (int k = 0; k < 4; k++)
        w[k] = ref[k] >= 0 ? S.uv[ref[k]] : make_double2(tu[~ref[k]], tv[~ref[k]]);
      double2 l[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (ref[k] >= 0)
          l[k] = S.lam[ref[k]];
        else if (polled >> k & 1)
          l[k] = mail_value(m[k]);
        else
          l[k] = make_double2(0.0, 0.0);  // a halo slot has no U point
      }
      // str1, str5 by the point itself; str2, str7 by the one at ee; str4,
      // str8 at ne; str3, str6 at se
      const double lo[8] = {l[0].x, l[1].x, l[3].x, l[2].x, l[0].y, l[3].y, l[1].y, l[2].y};
      Corners cr;
      cr.ucc = w[0].x;
      cr.vcc = w[0].y;
      cr.uee = w[1].x;
      cr.vee = w[1].y;
      cr.une = w[2].x;
      cr.vne = w[2].y;
      cr.use = w[3].x;
      cr.vse = w[3].y;
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
      double lc[8], lstr;
      // (the straight-line form needs more registers than wider blocks have)
      stress_adjoint_t<(NT <= 256)>(cr, g, S.geo[9][c], p, lo, ls, lc, lstr);
      own_share = make_double2(lc[0], lc[1]);
#pragma unroll
      for (int k = 0; k < 3; k++) S.share[k][c] = make_double2(lc[2 + 2 * k], lc[3 + 2 * k]);
      if (own) S.acc[5][c] += lstr;
    }
    if (fail) atomicMax(a.err, kResCode);
    if (__syncthreads_or(fail)) return;
    if (own) {
      s_nw = S.share[0][inw];
      s_sw = S.share[1][isw];
      s_sse = S.share[2][isse];
      S.uv[c] = next;  // read again only after the next barrier
      unew = uold;
      uold = next;
    }
  }
  if (own) {
    if (!actT) own_share = make_double2(0.0, 0.0);
    a.Pu[slot] = S.acc[0][c];
    a.Pv[slot] = S.acc[1][c];
    a.gC[slot] = S.acc[2][c];
    a.gx[slot] = S.acc[3][c];
    a.gy[slot] = S.acc[4][c];
    a.gs[slot] = S.acc[5][c];
    a.C8[0][slot] = own_share.x;
    a.C8[1][slot] = own_share.y;
    a.C8[2][slot] = s_nw.x;
    a.C8[3][slot] = s_nw.y;
    a.C8[4][slot] = s_sw.x;
    a.C8[5][slot] = s_sw.y;
    a.C8[6][slot] = s_sse.x;
    a.C8[7][slot] = s_sse.y;
#pragma unroll
    for (int k = 0; k < 12; k++) a.LS[k][slot] = ls[k];
  }
}

using AdjKernel = void (*)(ResidentAdjArgs, Params);
struct AdjVariant {
  int width;
  AdjKernel k;
  size_t smem;
};
const AdjVariant kAdjVariants[] = {{128, k_resident_adj<128>, sizeof(AdjSmem<128>)},
                                   {256, k_resident_adj<256>, sizeof(AdjSmem<256>)},
                                   {384, k_resident_adj<384>, sizeof(AdjSmem<384>)},
                                   {512, k_resident_adj<512>, sizeof(AdjSmem<512>)}};
static_assert(sizeof(AdjSmem<kResAdjointMax>) <= 227 * 1024, "shared memory per block");

const AdjVariant *find_variant(int cls) {
  for (const AdjVariant &v : kAdjVariants)
    if (v.width == cls) return &v;
  return nullptr;
}

}  // namespace

int resident_adjoint_prepare(int device, int cls, int nblocks) {
  const AdjVariant *v = find_variant(cls);
  if (!v) return 0;
  int sms = 0, per_sm = 0;
  cudaError_t e =
      cudaFuncSetAttribute(v->k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v->smem);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v->k, v->width, v->smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nblocks <= sms * per_sm ? 1 : 0;
}

cudaError_t launch_resident_adjoint(const ResidentAdjArgs &given, const Params &p, int cls,
                                    int threads, int nblocks, cudaStream_t st) {
  const AdjVariant *v = find_variant(cls);
  if (!v || nblocks <= 0 || given.nsub < 1) return cudaErrorInvalidValue;
  ResidentAdjArgs a = given;
  a.width = threads;
  Params pp = p;
  void *args[] = {&a, &pp};
  return launch_cooperative((const void *)v->k, dim3(nblocks), dim3((threads + 31) / 32 * 32), args,
                            v->smem, st);
}

}  // namespace evp
