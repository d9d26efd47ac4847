// k_scal.cu -- scalar advection of one RK stage for every advected field in
// one launch: advs (adv.F:14-903) as solve2 calls it for theta
// (solve2.F:1394), each moisture array (1490/1510) and each passive tracer
// (1941), followed by the RK update of each (solve2.F:1419-1425, 1513-1520,
// 1951-1957).  All fields of a stage are advected by the same averaged
// velocities rru/rrv/rrw, so one block advances every field over its tile:
//
//  * a block owns TX x TY columns and kc levels; it walks the items
//    (field n, level k) field by field, level by level upward;
//  * the level of a field is staged in shared memory with its 3-point halo by
//    one-dimensional bulk copies (cp.async.bulk), one per row, into a ring of
//    RD planes; warp 0 issues the copies of item t+RD as soon as item t's
//    plane has been read, and an mbarrier per ring slot tells the block when
//    they have landed, so each plane is in flight while RD-1 others compute;
//  * the caller's rows are not 16-byte aligned (a row holds NI = ni+6
//    floats), so each row copy takes the aligned superset of its 38 values;
//    the plane's row pitch SP is chosen congruent to NI modulo 4, so that
//    every row lands with element x at plane[c + r*SP + x] for a c that is
//    the same for all rows of the plane;
//  * each x- and y-face flux is evaluated once (face5, the WENO5 or
//    5th-order value), the vertical face of the level above comes from a
//    per-thread register window of the column and is carried to the next level;
//  * one barrier per item: the face fluxes and face velocities are double
//    buffered by item parity.
//
// Bound by instruction issue (67 % of the cycles): three faces are some 400 of an
// item's 650 to 760 instructions, at 24 warps a SM (80 registers).  So the faces that the fast
// WENO5 leaves open are evaluated beside it from shared memory without a call,
// the item's global reads are issued after its faces and not before (their
// registers are then free while a face is evaluated), and a flux lies beside
// its velocity in one 8-byte word.  256x256x80, seven fields: 1.33 ms a stage
// where the faces at a tracer's edge and in uniform layers took the reference's
// divisions one by one, now 1.14 ms; 512x512x128, three fields: 4.1 to 2.95 ms.
// (Two blocks a SM without the limit of 80 registers: 10 % slower.)
//
// Every face value and the update use the operations of k_advs_tile in the
// same order, so the result is bit-identical to advancing the fields one
// launch at a time.  Waits on the mbarriers are bounded: a block that gives
// up sets *err and leaves without writing (the host reports the error).
#include <cstdint>
#include "cm1g_common.cuh"
#include "k_face.cuh"

namespace cm1g {

constexpr int SC_MAX = 16;      // fields per launch
constexpr int SC_KMAX = 32;     // levels per block at most (a word of signs holds a bit for each)

struct ScalPass {
  ScalField f[SC_MAX];
  int n, kc;                    // fields; levels per block
  const float *rru, *rrv, *rrw; // small-step-averaged velocities (sound.F:806-835)
  const float *thterm;          // moist theta: thten -= div(u_avg) * thterm (solve2.F:1320-1329); null: none
  float dt;
  int *err;                     // set to 1 when a block gives up waiting for its staged data
  // positive-definite pass (one field): advx, advy, advz and the provisional
  // masses dumx, dumy, dumz; a word for each level chunk, row and 32 columns,
  // bit m set where a provisional mass at level m of the chunk is negative
  float *adv[3], *dum[3];
  unsigned *neg;
  // the caller's own mass fluxes (adv.F's arguments) in place of velocities to
  // weight: its divx, and where the positive-definite pass keeps its tendency
  const float *divx;
  float *tsave;
};

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_arrive(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false if the phase did not complete within the limit
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 22); it++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

}  // namespace

// Row pitch of a staged plane: at least TX + 16 floats (the aligned superset
// of a row's TX + 6 values is at most TX + 12) and congruent to NI modulo 4.
template <int TX>
__host__ __device__ __forceinline__ int scal_pitch(int NI) {
  const int p0 = TX + 16;
  return p0 + (((NI - p0) % 4) + 4) % 4;
}

// Profiles of one level k of a block, read as two 16-byte words.
struct __align__(16) ScLev {
  float r0, rf, rf1, mh;     // rho0(k), rf0(k), rf0(k+1), mh(k)
  float rr, th, th3, pad;    // rr0(k), th0(k)-300, th0(k+3)-300
};

// One cell's advection from its faces, (flux, averaged velocity) each, with the
// open-boundary fix-ups of adv.F where the tile touches an open edge; fz* and w*
// are the vertical fluxes and averaged velocities; in la the density is 1 where
// the velocities are the caller's mass fluxes.
struct ScAdv {
  float x, y, z, sum;          // advx, advy, advz and (advx + advy + advz + s div)/rho0
  bool w, e, s, n;             // inflow through an open edge
};
__device__ __forceinline__ ScAdv scal_advection(const DGrid &g, float2 xw, float2 xe, float2 ys, float2 yn, float fzlo,
                                                float fzhi, float wlo, float whi, float4 la, float rr0, int i, int j, int k,
                                                bool edge, float uh_i, float vh_j, float sc, const float *divx) {
  const float r0k = la.x, mhk = la.w;
  float fx0 = xw.x, fxp = xe.x, fy0 = ys.x, fyp = yn.x;
  const float fu0 = xw.y * r0k, fu1 = xe.y * r0k, fv0 = ys.y * r0k, fv1 = yn.y * r0k;
  const float rdx = g.rdx, rdy = g.rdy, rdz = g.rdz;
  ScAdv a;
  a.w = a.e = a.s = a.n = false;
  if (!edge) {
    a.x = -(fxp - fx0) * rdx * uh_i;
    a.y = -(fyp - fy0) * rdy * vh_j;
  } else {
    a.w = g.wbc == 2 && g.ibw && i == 1 && fu0 >= 0.0f; a.e = g.ebc == 2 && g.ibe && i == g.ni && fu1 <= 0.0f;
    a.s = g.sbc == 2 && g.ibs && j == 1 && fv0 >= 0.0f; a.n = g.nbc == 2 && g.ibn && j == g.nj && fv1 <= 0.0f;
    // adv.F:212-268
    if (a.w) fx0 = fxp;
    if (a.e) fxp = fx0;
    if (a.s) fy0 = fyp;
    if (a.n) fyp = fy0;
    a.x = -(fxp - fx0) * rdx * uh_i;
    a.y = -(fyp - fy0) * rdy * vh_j;
    // adv.F:286-335
    if (a.w) a.x = a.x - sc * (fu1 - fu0) * rdx * uh_i;
    if (a.e) a.x = a.x - sc * (fu1 - fu0) * rdx * uh_i;
    if (a.s) a.y = a.y - sc * (fv1 - fv0) * rdy * vh_j;
    if (a.n) a.y = a.y - sc * (fv1 - fv0) * rdy * vh_j;
  }
  if (k == 1) a.z = -fzhi * rdz * mhk;
  else if (k == g.nk) a.z = +fzlo * rdz * mhk;
  else a.z = -(fzhi - fzlo) * rdz * mhk;
  float div;
  if (divx) {
    div = *divx;
  } else {
    div = ((fu1 - fu0) * rdx * uh_i + (fv1 - fv0) * rdy * vh_j) + (whi * la.z - wlo * la.y) * rdz * mhk;
    if (fabsf(div) < g.smeps) div = 0.0f;
  }
  a.sum = (((a.x + a.y) + a.z) + sc * div) * rr0;
  return a;
}

__device__ __forceinline__ ScLev scal_level(const DGrid &g, int k) {
  ScLev l;
  l.r0 = LDG(&g.rho0[k]); l.rf = LDG(&g.rf0[k]); l.rf1 = LDG(&g.rf0[k + 1]); l.mh = LDG(&g.mh[k]);
  l.rr = LDG(&g.rr0[k]); l.th = LDG(&g.th0[k]) - 300.0f;
  l.th3 = k + 3 <= g.nk + 1 ? LDG(&g.th0[k + 3]) - 300.0f : 0.0f;
  l.pad = 0.0f;
  return l;
}

// PDEF: the first pass of the positive-definite scheme (pdef.F:35-102, 289-340,
// 478-496) of one field: advx..dumz and neg beside the value that holds where no
// neighbouring provisional mass is negative (k_pdef_fix does the other cells).
// RAW: the caller's mass fluxes and divx; the value is the tendency.
template <int TX, int TY, int WENO, int PDEF, int RAW>
__global__ void __launch_bounds__(TX * (TY + 1), 3) k_scal_tile(const __grid_constant__ DGrid g,
                                                                 const __grid_constant__ ScalPass P) {
  constexpr int SW = TX + 6, SH = TY + 6;                  // staged columns and rows
  constexpr int RD = 4;                                     // ring of staged planes
  constexpr int PL = ((8 + (SH - 1) * (TX + 19) + TX + 12) + 3) / 4 * 4;   // floats per plane
  constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
  static_assert(SH <= 32, "one lane per staged row");
  __shared__ __align__(128) float ring[RD][PL];
  __shared__ float2 fx[2][NFX], fy[2][NFY];                // flux and averaged velocity of each face
  __shared__ ScLev lev[SC_KMAX];
  __shared__ __align__(8) uint64_t bars[RD];

  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty, lane = tid & 31;
  // the first warp of the extra row issues the staging copies
  const bool stager = (tid >= TX * TY && tid < TX * TY + 32);
  const int i0 = 1 + (int)blockIdx.x * TX, j0 = 1 + (int)blockIdx.y * TY;
  const int i = i0 + tx, j = j0 + ty;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI, NJ = g.NJ;
  const bool active = (ty < TY && i <= ni && j <= nj);
  const int planeS = NI * NJ, planeU = (NI + 1) * NJ, planeV = NI * (NJ + 1);
  const int SP = scal_pitch<TX>(NI);
  const float uh_i = active ? LDG(&g.uh[i - g.ib]) : 0.0f, vh_j = active ? LDG(&g.vh[j - g.jb]) : 0.0f;
  const int orow0 = (i0 - 3 - g.ib) + NI * (j0 - 3 - g.jb);    // first staged element of a plane
  const int kc0 = 1 + (int)blockIdx.z * P.kc, kc1 = min(nk, kc0 + P.kc - 1);
  const int nlev = kc1 - kc0 + 1, nitem = P.n * nlev;

  // faces of this thread: a cell row's thread owns the x face on the west of
  // its cell and the y face on its south; the extra row's threads own the y
  // faces north of the tile and (the first TY of them) the x faces east of it,
  // so that every cell thread evaluates three faces and no thread more.
  // oc: the thread's column in an s or v plane; xo: its x face in a u plane;
  // xs, ys: the stencils' first values in a staged plane
  const bool yface_on = (i <= ni && j <= nj + 1);
  const int oc = yface_on ? (i - g.ib) + NI * (j - g.jb) : 0;
  const int ys = ty * SP + tx + 3;
  bool xface_on = false;
  int xo = 0, xs = 0, xd = 0;
  {
    const int xrow = ty < TY ? ty : tx, xcol = ty < TY ? tx : TX;
    const int ii = i0 + xcol, jj = j0 + xrow;
    if (xrow < TY && ii <= ni + 1 && jj <= nj) {
      xface_on = true;
      xo = (ii - g.ib) + (NI + 1) * (jj - g.jb);
      xs = (xrow + 3) * SP + xcol;
      xd = xrow * (TX + 1) + xcol;
    }
  }

  // profiles of the block's levels (0 above nk+1, not used there)
  if (tid < nlev) {
    lev[tid] = scal_level(g, kc0 + tid);
  }

  // the open-boundary fix-ups of adv.F touch only the cells next to an open edge
  const bool edge = (g.wbc == 2 && g.ibw && i0 == 1) || (g.ebc == 2 && g.ibe && i0 + TX - 1 >= ni) ||
                    (g.sbc == 2 && g.ibs && j0 == 1) || (g.nbc == 2 && g.ibn && j0 + TY - 1 >= nj);

  // ---- staging: items in order (field, level) -> ring slot item % RD
  const uint32_t bar0 = smem_u32(&bars[0]);
  if (tid == 0) {
    for (int b = 0; b < RD; b++) mbar_init(bar0 + 8 * b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // the row copies of the item (field nf, level kf) into slot `slot` (rows
  // beyond the last halo row are never read)
  auto issue = [&](int nf, int kf, int slot) {
    const float *p0 = P.f[nf].s + (kf * planeS + orow0);
    const int l0 = (int)(((uintptr_t)p0 >> 2) & 3);
    uint32_t bytes = 0, dst = 0;
    const float *src = nullptr;
    if (lane < SH && j0 - 3 + lane <= nj + g.ngxy) {
      const uintptr_t a0 = (uintptr_t)(p0 + lane * NI);
      const uintptr_t as = a0 & ~(uintptr_t)15, ae = (a0 + 4 * SW + 15) & ~(uintptr_t)15;
      const int lr = (int)((a0 >> 2) & 3);
      bytes = (uint32_t)(ae - as);
      src = (const float *)as;
      dst = smem_u32(&ring[slot][l0 + 4 + lane * SP - lr]);
    }
    const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
    if (lane == 0) mbar_expect_arrive(bar0 + 8 * slot, total);
    __syncwarp();
    if (bytes) bulk_g2s(dst, src, bytes, bar0 + 8 * slot);
  };
  int in_ = 0, ik_ = kc0, it_ = 0;   // next item to issue
  auto issue_next = [&]() {
    issue(in_, ik_, it_ % RD);
    it_++;
    if (++ik_ > kc1) { ik_ = kc0; in_++; }
  };
  if (stager)
    while (it_ < RD && it_ < nitem) issue_next();

  // ---- per-item global reads: issued once the previous item's faces are done,
  // so that they are in flight during its update and take no register while a
  // face is evaluated (the faces need nearly all 80 of them)
  float ru = 0.0f, rv = 0.0f, whi = 0.0f, e0 = 0.0f, e1 = 0.0f, e2 = 0.0f, stop = 0.0f;
  auto fetch = [&](int nf, int kf) {
    const ScalField &F = P.f[nf];
    if (xface_on) ru = LDG(&P.rru[kf * planeU + xo]);
    if (yface_on) rv = LDG(&P.rrv[kf * planeV + oc]);
    if (active) {
      const int o = kf * planeS + oc;
      whi = (!RAW && kf == nk) ? 0.0f : LDG(&P.rrw[o + planeS]);
      e0 = F.ten1[o];
      if (PDEF || !RAW) e1 = LDG(&F.sbase[o]);
      if (RAW) e2 = LDG(&P.divx[o]);
      else if (!PDEF && F.sadd && P.thterm) e2 = LDG(&P.thterm[o]);
      // s(kf+3), the last value under the upper face of level kf
      stop = (kf + 3 <= nk + 1) ? LDG(&F.s[o + 3 * planeS]) : 0.0f;
    }
  };

  int tfail = -1, t = 0;
  unsigned neg = 0;
  fetch(0, kc0);
  for (int n = 0; n < P.n && tfail < 0; n++) {
    const ScalField &F = P.f[n];
    const int sadd = F.sadd, pdw = F.pdefweno;
    const double weps = F.weps;
    // the column window, wv[d] = s(k-2+d) for the upper face of level k, and
    // the face below the first level; the window's last value is fetched
    float wv[6] = {0, 0, 0, 0, 0, 0}, fzlo = 0.0f, wlo = 0.0f;
    if (active) {
      float w0 = 0.0f;
#pragma unroll
      for (int d = -1; d < 5; d++) {
        const int kk = kc0 - 2 + d;
        float v = 0.0f;
        if (kk >= 0 && kk <= nk + 1) {
          v = LDG(&F.s[kk * planeS + oc]);
          if (sadd) v = (LDG(&g.th0[kk]) - 300.0f) + v;
        }
        if (d < 0) w0 = v;
        else wv[d] = v;
      }
      if (RAW || kc0 >= 2) wlo = LDG(&P.rrw[kc0 * planeS + oc]);
      if (kc0 >= 2) {
        const float r = RAW ? wlo : wlo * lev[0].rf;
        const float w[6] = {w0, wv[0], wv[1], wv[2], wv[3], wv[4]};
        fzlo = face5(r, w0, wv[0], wv[1], wv[2], wv[3], wv[4], WENO, pdw, weps);
        if (WENO && fzlo != fzlo) fzlo = face5_exact(r, w0, wv[0], wv[1], wv[2], wv[3], wv[4], weps);
        if (kc0 <= 3 || kc0 >= nk - 1) fzlo = zface_edge(fzlo, w, r, kc0, nk, g.c1, g.c2, WENO, pdw, weps);
      }
    }
    int cal = (int)(((uintptr_t)(F.s + (kc0 * planeS + orow0)) >> 2) & 3);   // alignment of the staged plane
    for (int k = kc0; k <= kc1; k++, t++) {
      const float4 la = *(const float4 *)&lev[k - kc0].r0, lb = *(const float4 *)&lev[k - kc0].rr;
      const float r0k = RAW ? 1.0f : la.x, th0m = lb.y;
      const int b = t & 1, slot = t % RD;
      // ---- the staged plane of this item
      const bool ok = mbar_wait(bar0 + 8 * slot, (uint32_t)((t / RD) & 1));
      const float *pl = &ring[slot][cal + 4];
      cal = (cal + planeS) & 3;
      // ---- face values: each x/y face once, the upper z face once per column
      auto staged = [&](float *s, int o, int st) {
#pragma unroll
        for (int d = 0; d < 6; d++) { s[d] = pl[o + d * st]; if (sadd) s[d] = th0m + s[d]; }
      };
      if (xface_on) {
        float s[6];
        staged(s, xs, 1);
        float f = face5(ru * r0k, s[0], s[1], s[2], s[3], s[4], s[5], WENO, PDEF, weps);
        if (WENO && f != f) { staged(s, xs, 1); f = face5_exact(ru * r0k, s[0], s[1], s[2], s[3], s[4], s[5], weps); }
        fx[b][xd] = make_float2(f, ru);
      }
      if (yface_on) {
        float s[6];
        staged(s, ys, SP);
        float f = face5(rv * r0k, s[0], s[1], s[2], s[3], s[4], s[5], WENO, PDEF, weps);
        if (WENO && f != f) { staged(s, ys, SP); f = face5_exact(rv * r0k, s[0], s[1], s[2], s[3], s[4], s[5], weps); }
        fy[b][tid] = make_float2(f, rv);
      }
      float fzhi = 0.0f;
      if (active) {
        wv[5] = (sadd && k + 3 <= nk + 1) ? lb.z + stop : stop;
        const int kk = k + 1;
        const float r = RAW ? whi : whi * la.z;
        if (kk <= nk) {
          fzhi = face5(r, wv[0], wv[1], wv[2], wv[3], wv[4], wv[5], WENO, pdw, weps);
          if (WENO && fzhi != fzhi) fzhi = face5_exact(r, wv[0], wv[1], wv[2], wv[3], wv[4], wv[5], weps);
          if (kk <= 3 || kk >= nk - 1) fzhi = zface_edge(fzhi, wv, r, kk, nk, g.c1, g.c2, WENO, pdw, weps);
        }
      }
      float sc = 0.0f;
      if (active) {
        sc = pl[ys + 3 * SP];
        if (sadd) sc = th0m + sc;
      }
      if (__syncthreads_or(!ok)) { tfail = t; break; }
      // the plane of this item has been read: its slot takes the item RD later
      if (stager && it_ < nitem) issue_next();
      const float whik = whi, ten1 = e0, base = e1, e2k = e2;
      bool negative = false;
      if (k < kc1) fetch(n, k + 1);
      else if (n + 1 < P.n) fetch(n + 1, kc0);
      if (active) {
        const float2 xw = fx[b][xd], xe = fx[b][xd + 1], ysw = fy[b][tid], yn = fy[b][tid + TX];
        const ScAdv a = scal_advection(g, xw, xe, ysw, yn, fzlo, fzhi, wlo, whik,
                                       RAW ? make_float4(1.0f, 1.0f, 1.0f, la.w) : la, lb.x, i, j, k, edge, uh_i, vh_j, sc,
                                       RAW ? &e2k : nullptr);
        const int o = k * planeS + oc;
        float ten = ten1;
        if (!RAW && !PDEF && sadd && P.thterm) {   // getdiv of the averaged velocities (misclibs.F:127-136)
          float rd = ((xe.y - xw.y) * g.rdx * uh_i + (yn.y - ysw.y) * g.rdy * vh_j) + (whik - wlo) * g.rdz * la.w;
          if (fabsf(rd) < g.smeps) rd = 0.0f;
          ten = ten - rd * e2k;
        }
        ten = ten + a.sum;
        float v = RAW ? ten : base + P.dt * ten;
        if (!RAW && F.flush && fabsf(v) < g.smeps) v = 0.0f;
        if (PDEF) {   // provisional masses
          const float dt = P.dt, m0 = la.x * base;
          const float fu0 = xw.y * r0k, fu1 = xe.y * r0k, fv0 = ysw.y * r0k, fv1 = yn.y * r0k;
          float dx = m0 + dt * (a.x + sc * (fu1 - fu0) * g.rdx * uh_i), dy = m0 + dt * (a.y + sc * (fv1 - fv0) * g.rdy * vh_j);
          if (a.w || a.e) dx = m0;
          if (a.s || a.n) dy = m0;
          const float fwhi = RAW ? whik : whik * la.z, fwlo = RAW ? wlo : wlo * la.y;
          const float dz = m0 + dt * (a.z + sc * (fwhi - fwlo) * g.rdz * la.w);
          P.adv[0][o] = a.x; P.adv[1][o] = a.y; P.adv[2][o] = a.z;
          P.dum[0][o] = dx; P.dum[1][o] = dy; P.dum[2][o] = dz;
          if (RAW) P.tsave[o] = ten1;
          negative = dx < 0.0f || dy < 0.0f || dz < 0.0f;
        }
        F.snew[o] = v;
        // slide the column window and carry the upper face to the next level
#pragma unroll
        for (int d = 0; d < 5; d++) wv[d] = wv[d + 1];
        fzlo = fzhi;
        wlo = whik;
      }
      if (PDEF && __any_sync(0xffffffffu, negative)) neg |= 1u << (k - kc0);
    }
  }
  if (PDEF && ty < TY && j <= nj && i - lane <= ni && lane == 0) {
    const int nch = (ni + 31) / 32;
    P.neg[((int)blockIdx.z * nj + j - 1) * nch + (i - 1) / 32] = neg;
  }
  if (tfail >= 0) {
    // leave no bulk copy in flight into this block's shared memory: wait (each
    // wait bounded) for the items issued but not consumed
    if (tid == 0) atomicExch(P.err, 1);
    for (int u = tfail; u < nitem && u < tfail + RD; u++) (void)mbar_wait(bar0 + 8 * (u % RD), (uint32_t)((u / RD) & 1));
  }
}

// Second pass of the positive-definite scheme: pdefz, pdefx2, pdefy2
// (pdef.F:117-264, 358-454, 459-581) and the update of adv.F:650-659 and
// solve2.F:1513-1520, for the cells whose value they change.  A warp owns 32
// columns of a row over a chunk of the first pass's levels; it reads the chunk's word of
// negative provisional masses and its neighbours' (a cell changes only if its
// own, or one beside it in x, y or z, is negative) and visits the levels named
// there, all loads of a level in flight at once.  A field without such masses
// costs the launch (256x256x80: 10 us against 135 us when every cell read the six
// arrays back), a tracer of a few blobs after two stages 100 us; the host entry at
// 251x187x79 with every level named 74 us, where a thread a cell took 97.  Beyond
// the domain the masses are those of the points that the lateral bc copies there
// (pdef.F:102, 338).
template <int RAW>
__global__ void __launch_bounds__(256) k_pdef_fix(const __grid_constant__ DGrid g, const __grid_constant__ ScalPass P) {
  const int lane = (int)(threadIdx.x & 31);
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI, KC = P.kc, nch = (ni + 31) / 32, nkb = (nk + KC - 1) / KC;
  const int ch = (int)blockIdx.x, j = 1 + (int)(blockIdx.y * 8 + (threadIdx.x >> 5)), kb = (int)blockIdx.z;   // 8 rows a block
  if (j > nj) return;
  const int i0 = 1 + 32 * ch, i = i0 + lane, kc0 = 1 + kb * KC;
  auto bcx = [&](int ii) { return bc_source(ii, ni, g.wbc, g.ebc); };
  auto bcy = [&](int jj) { return bc_source(jj, nj, g.sbc, g.nbc); };
  unsigned w = 0;
  {   // lane 0 own, 1-2 x neighbours, 3-4 y neighbours, 5-6 the chunks below and above
    int c = ch, r = j, b = kb;
    if (lane == 1) c = (bcx(i0 - 1) - 1) / 32;
    if (lane == 2) c = (bcx(min(i0 + 31, ni) + 1) - 1) / 32;
    if (lane == 3) r = bcy(j - 1);
    if (lane == 4) r = bcy(j + 1);
    if (lane == 5) b = kb - 1;
    if (lane == 6) b = kb + 1;
    if (lane < 7 && b >= 0 && b < nkb) w = P.neg[(b * nj + r - 1) * nch + c];
    if (lane == 0) w |= (w << 1) | (w >> 1);
    if (lane == 5) w >>= KC - 1;
    if (lane == 6) w = (w & 1) << (KC - 1);
  }
  unsigned todo = __reduce_or_sync(0xffffffffu, w);
  const int left = nk - kc0 + 1;
  if (left < 32) todo &= (1u << left) - 1;
  if (KC < 32) todo &= (1u << KC) - 1;
  if (i > ni) return;
  const ScalField &F = P.f[0];
  const int plane = NI * g.NJ, oc = (i - g.ib) + NI * (j - g.jb);
  const int xr = NI * (j - g.jb) - g.ib, yc = i - g.ib;
  const int xm2 = xr + bcx(i - 2), xm1 = xr + bcx(i - 1), xp1 = xr + bcx(i + 1), xp2 = xr + bcx(i + 2);
  const int ym2 = yc + NI * (bcy(j - 2) - g.jb), ym1 = yc + NI * (bcy(j - 1) - g.jb);
  const int yp1 = yc + NI * (bcy(j + 1) - g.jb), yp2 = yc + NI * (bcy(j + 2) - g.jb);
  const float smeps = g.smeps, rdt = 1.0f / P.dt;
  for (; todo; todo &= todo - 1) {
    const int k = kc0 + __ffs(todo) - 1, ok = k * plane, o = ok + oc;
    const float *X = P.dum[0] + ok, *Y = P.dum[1] + ok, *Z = P.dum[2] + o;
    const float x0 = LDG(&X[oc]), y0 = LDG(&Y[oc]), z0 = LDG(&Z[0]);
    const float xa = LDG(&X[xm2]), xb = LDG(&X[xm1]), xc = LDG(&X[xp1]), xd = LDG(&X[xp2]);
    const float ya = LDG(&Y[ym2]), yb = LDG(&Y[ym1]), yc_ = LDG(&Y[yp1]), yd = LDG(&Y[yp2]);
    const float za = k > 2 ? LDG(&Z[-2 * plane]) : 0.0f, zb = k > 1 ? LDG(&Z[-plane]) : 0.0f;
    const float zc = k < nk ? LDG(&Z[plane]) : 0.0f, zd = k < nk - 1 ? LDG(&Z[2 * plane]) : 0.0f;
    float s = LDG(&F.s[o]);
    const float s0 = LDG(&F.sbase[o]);
    const float *u = P.rru + k * ((NI + 1) * g.NJ) + (i - g.ib) + (NI + 1) * (j - g.jb);
    const float *v = P.rrv + k * (NI * (g.NJ + 1)) + oc;
    const float u0 = LDG(&u[0]), u1 = LDG(&u[1]), v0 = LDG(&v[0]), v1 = LDG(&v[NI]);
    const float w0 = (RAW || k > 1) ? LDG(&P.rrw[o]) : 0.0f, w1 = (RAW || k < nk) ? LDG(&P.rrw[o + plane]) : 0.0f;
    float ax = LDG(&P.adv[0][o]), ay = LDG(&P.adv[1][o]), az = LDG(&P.adv[2][o]);
    const float t1 = RAW ? P.tsave[o] : F.ten1[o];
    float mx, my, mz;
    bool fx, fy, fz;
    pdef_gather(xa, xb, x0, xc, xd, smeps, &mx, &fx);
    pdef_gather(ya, yb, y0, yc_, yd, smeps, &my, &fy);
    pdef_gather(za, zb, z0, zc, zd, smeps, &mz, &fz);
    if (!(fx || fy || fz)) continue;   // the first pass's value stands
    const float r0 = LDG(&g.rho0[k]), r0k = RAW ? 1.0f : r0, mhk = LDG(&g.mh[k]);
    const float uh_i = LDG(&g.uh[i - g.ib]), vh_j = LDG(&g.vh[j - g.jb]);
    if (F.sadd) s = (LDG(&g.th0[k]) - 300.0f) + s;
    const float fu0 = u0 * r0k, fu1 = u1 * r0k, fv0 = v0 * r0k, fv1 = v1 * r0k;
    const float fwlo = RAW ? w0 : k == 1 ? 0.0f : w0 * LDG(&g.rf0[k]);
    const float fwhi = RAW ? w1 : k == nk ? 0.0f : w1 * LDG(&g.rf0[k + 1]);
    if (fx) ax = (x0 + mx - r0 * s0) * rdt - s * (fu1 - fu0) * g.rdx * uh_i;
    if (fy) ay = (y0 + my - r0 * s0) * rdt - s * (fv1 - fv0) * g.rdy * vh_j;
    if (fz) az = (z0 + mz - r0 * s0) * rdt - s * (fwhi - fwlo) * g.rdz * mhk;
    float div;
    if (RAW) {
      div = LDG(&P.divx[o]);
    } else {
      div = ((fu1 - fu0) * g.rdx * uh_i + (fv1 - fv0) * g.rdy * vh_j) + (fwhi - fwlo) * g.rdz * mhk;
      if (fabsf(div) < smeps) div = 0.0f;
    }
    const float ten = t1 + (((ax + ay) + az) + s * div) * LDG(&g.rr0[k]);
    float x = RAW ? ten : s0 + P.dt * ten;
    if (!RAW && F.flush && fabsf(x) < smeps) x = 0.0f;
    F.snew[o] = x;
  }
}

// kc: levels per block; 0: those whose blocks finish first.  A block costs about
// SC_OVER levels besides its own (its first plane's latency, the window and the
// face below its first level).  Scalar passes of a step with 16, 8 and 32 levels
// and with this rule: 64x64x40 82, 51, 137, 39 us; 203x150x61, four fields 713, 628,
// 838, 665 us; 256x256x80 2.60, 2.53, 2.51, 2.47 ms; 512x512x128 6.78, 7.20, 6.74, 6.78 ms.
// The host entry's single field takes at most 16: its second pass walks a chunk
// level by level (251x187x79, the one grid measured: 95 us with 20 levels, 76 with
// 12).  A step's passes keep the rule's choice: one launch's rule serves both, and
// their words name few levels where tracers are sparse.  Without a second pass (a
// word holds 4 levels at least) it takes as few as one: 16x16x20 40 to 35 us.
constexpr int SC_OVER = 2;
template <int TX, int TY, int PDEF, int RAW>
static void scal_shape(const DGrid &g, ScalPass P, int kc, int weno, cudaStream_t st, int64_t *nl) {
  dim3 blk(TX, TY + 1), grid((g.ni + TX - 1) / TX, (g.nj + TY - 1) / TY, 1);
  if (!kc) kc = tile_levels((long)grid.x * grid.y, g.nk, 3 * 148, SC_OVER, RAW && !PDEF ? 1 : 4, RAW ? 16 : SC_KMAX);
  P.kc = kc;
  grid.z = (g.nk + kc - 1) / kc;
  {
    ProfScope _ps(PDEF ? "k_scal_pdef" : "k_scal_tile", st);
    if (weno) k_scal_tile<TX, TY, 1, PDEF, RAW><<<grid, blk, 0, st>>>(g, P);
    else k_scal_tile<TX, TY, 0, PDEF, RAW><<<grid, blk, 0, st>>>(g, P);
  }
  if (PDEF) {
    ProfScope _ps("k_pdef_fix", st);
    k_pdef_fix<RAW><<<dim3((g.ni + 31) / 32, (g.nj + 7) / 8, grid.z), 256, 0, st>>>(g, P);
  }
  if (nl) *nl += PDEF ? 2 : 1;
}

// the tile of a shape, with the levels of its table but for the default's
template <int PDEF>
static void scal_launch(const DGrid &g, const ScalPass &P, int weno, cudaStream_t st, int64_t *nl) {
  static_assert(kNumTileShapes == 5 && kScalShapes[0][0] == 32 && kScalShapes[0][1] == 7 && kScalShapes[1][1] == 7 &&
                    kScalShapes[2][1] == 3 && kScalShapes[3][0] == 64 && kScalShapes[4][1] == 7,
                "the tiles of the shapes");
  const int kc = g.tile_adv > 0 ? kScalShapes[g.tile_adv][2] : 0;
  switch (g.tile_adv) {
    case 2: scal_shape<32, 3, PDEF, 0>(g, P, kc, weno, st, nl); break;
    case 3: scal_shape<64, 3, PDEF, 0>(g, P, kc, weno, st, nl); break;
    default: scal_shape<32, 7, PDEF, 0>(g, P, kc, weno, st, nl);
  }
}

// One launch for `n` fields (at most SC_MAX) advanced by the same averaged
// velocities; thterm applies to the field with sadd set.
void launch_scal_pass(const DGrid &g, const ScalField *f, int n, const float *rru, const float *rrv,
                      const float *rrw, const float *thterm, int weno, float dt, int *err, cudaStream_t st,
                      int64_t *nl) {
  for (int a = 0; a < n; a += SC_MAX) {
    ScalPass P{};
    P.n = (n - a < SC_MAX) ? n - a : SC_MAX;
    for (int m = 0; m < P.n; m++) P.f[m] = f[a + m];
    P.rru = rru; P.rrv = rrv; P.rrw = rrw; P.thterm = thterm; P.dt = dt; P.err = err;
    scal_launch<0>(g, P, weno, st, nl);
  }
}

static void pdef_scratch(const DGrid &g, ScalPass &P, float *scratch, unsigned *neg) {
  const long n = nS(g);
  for (int d = 0; d < 3; d++) { P.adv[d] = scratch + d * n; P.dum[d] = scratch + (3 + d) * n; }
  P.neg = neg;
}

// The positive-definite pass of one field (f.pdefweno as its vertical form);
// scratch holds 6 s-arrays, neg scal_neg_words(g) words.
void launch_scal_pdef(const DGrid &g, const ScalField &f, const float *rru, const float *rrv, const float *rrw, int weno,
                      float dt, float *scratch, unsigned *neg, int *err, cudaStream_t st, int64_t *nl) {
  ScalPass P{};
  P.n = 1; P.f[0] = f; P.rru = rru; P.rrv = rrv; P.rrw = rrw; P.dt = dt; P.err = err;
  pdef_scratch(g, P, scratch, neg);
  scal_launch<1>(g, P, weno, st, nl);
}

size_t scal_neg_words(const DGrid &g) { return (size_t)((g.nk + 3) / 4) * g.nj * ((g.ni + 31) / 32); }

// adv.F's advs: sten += the advection of s by the caller's mass fluxes, with its
// divx; pdef with the RK base s0 (tsave: an s-array that keeps sten).
void launch_advs(const DGrid &g, const float *rru, const float *rrv, const float *rrw, const float *divx, const float *s,
                 const float *s0, float *sten, int weno, int pdef, int pdefweno, double weps, float dt, float *scratch,
                 unsigned *neg, float *tsave, int *err, cudaStream_t st, int64_t *nl) {
  ScalPass P{};
  P.n = 1; P.rru = rru; P.rrv = rrv; P.rrw = rrw; P.divx = divx; P.dt = dt; P.err = err; P.tsave = tsave;
  P.f[0].s = s; P.f[0].sbase = s0; P.f[0].ten1 = sten; P.f[0].snew = sten; P.f[0].weps = weps; P.f[0].pdefweno = pdefweno;
  if (pdef) {
    pdef_scratch(g, P, scratch, neg);
    scal_shape<32, 7, 1, 1>(g, P, 0, weno, st, nl);
  } else {
    scal_shape<32, 7, 0, 1>(g, P, 0, weno, st, nl);
  }
}

}  // namespace cm1g
