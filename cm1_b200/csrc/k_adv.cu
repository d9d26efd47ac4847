// k_adv.cu -- flux-form advection tendencies (adv.F, adv_routines.F).
//
// The production passes are k-marching tiles (k_mom for u, v, w, or
// k_mom_tile with the 6th-order diffusion; k_advs_tile for the scalars): each
// face flux is evaluated once, from a level staged in shared memory with its
// 3-point halo, instead of being stored in dumx/dumy/dumz; the rho0-weighted
// fluxes rru/rrv/rrw and their divergence are formed on the fly, so a momentum
// pass reads u, v, w (and theta/qv for buoyancy) and writes only the tendency.
// The scalars of a plain step and the per-routine entry cm1g_advs take
// k_scal_tile; k_advs_tile here serves the learned closure, the flux capture and
// the 6th-order diffusion, one field a launch.  Every expression keeps the
// reference's operand order.
#include "cm1g_common.cuh"
#include "k_face.cuh"

namespace cm1g {

// ---------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------
struct Vel {  // momentum-pass view of u,v,w and the mass-flux weights
  const float *__restrict__ u, *__restrict__ v, *__restrict__ w;
};

__device__ __forceinline__ float RRU(const DGrid &g, const Vel &q, int i, int j, int k) {
  return LDG(&g.rho0[k]) * LDG(&q.u[iU(g, i, j, k)]);             // solve2.F:499
}
__device__ __forceinline__ float RRV(const DGrid &g, const Vel &q, int i, int j, int k) {
  return LDG(&g.rho0[k]) * LDG(&q.v[iV(g, i, j, k)]);             // solve2.F:504
}
__device__ __forceinline__ float RRW(const DGrid &g, const Vel &q, int i, int j, int k) {
  if (k <= 1 || k >= g.nk + 1) return 0.0f;                       // solve2.F:509-511
  return LDG(&g.rf0[k]) * LDG(&q.w[iW(g, i, j, k)]);              // solve2.F:516
}
// divx of the momentum pass (solve2.F:590-596)
__device__ __forceinline__ float DIVX(const DGrid &g, const Vel &q, int i, int j, int k) {
  float d = ((RRU(g, q, i + 1, j, k) - RRU(g, q, i, j, k)) * g.rdx * LDG(&g.uh[i - g.ib]) +
             (RRV(g, q, i, j + 1, k) - RRV(g, q, i, j, k)) * g.rdy * LDG(&g.vh[j - g.jb])) +
            (RRW(g, q, i, j, k + 1) - RRW(g, q, i, j, k)) * g.rdz * LDG(&g.mh[k]);
  if (fabsf(d) < g.smeps) d = 0.0f;
  return d;
}

// buoyancy of a w level from th3d(i,j,kk) and qv(i,j,kk) (solve2.F:313-446, dum8 of the moist and dry forms)
__device__ __forceinline__ float buoy_v(const DGrid &g, float th3, float qvv, bool moist, int kk) {
  if (moist) {
    float q = fmaxf(qvv, 0.0f);
    float qli = fmaxf(0.0f, 0.0f + 0.0f);
    return g.c.g * ((th3 * LDG(&g.rth0[kk]) + g.c.repsm1 * (q - LDG(&g.qv0[kk]))) - ((qli - LDG(&g.qc0[kk])) - LDG(&g.qi0[kk])));
  }
  return g.c.g * th3 * LDG(&g.rth0[kk]);
}


// ---------------------------------------------------------------------
// Tiled momentum advection with the 6th-order diffusion (one component a
// launch; without it all three advance in k_mom below).
//
// divx of the momentum pass (solve2.F:590-596) is formed once per stage at
// the s-points i = 0..ni+1, j = 0..nj+1 by k_mom_divx.  k_mom_tile then
// works like the scalar tile: a block owns TX x TY points of one velocity
// component (STAG 2 u, 3 v, 4 w) and marches upward; at each level the
// component is staged with a 3-point lateral halo in shared memory, every
// x- and y-face flux (hadv_flx5 stag=2/3/4) is evaluated once, and the
// vertical face flux (vadv_flx5 with the lower-order pieces at the column
// ends) comes from a per-thread register window and is carried to the next
// level.  The face velocities are formed exactly as the reference forms
// them (ubar/vbar/wbar of adv_routines.F:1388-1460, 3299-3384) and the
// open-boundary fixes of adv.F are applied to the cells they concern.
// ---------------------------------------------------------------------
__global__ void k_mom_divx(DGrid g, Vel q, float *__restrict__ divx) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = (int)blockIdx.y, k = 1 + (int)blockIdx.z;
  if (i > g.ni + 1) return;
  divx[iS(g, i, j, k)] = DIVX(g, q, i, j, k);
}

// vertical face flux of a u/v column at w-level kk; wv[d+3] = a(kk+d), d = -3..2
__device__ __forceinline__ float zflux_uv(const DGrid &g, const float *wv, float wbar, int kk) {
  const int nk = g.nk;
  auto A = [&](int d) { return wv[d + 3]; };
  if (kk >= 4 && kk <= nk - 2) {
    const bool up = (wbar >= 0.0f);
    return wbar * flx5(up ? A(-3) : A(2), up ? A(-2) : A(1), up ? A(-1) : A(0), up ? A(0) : A(-1), up ? A(1) : A(-2));
  }
  const float c2k = LDG(&g.c2[kk]);
  if (kk == 2) {
    if (wbar >= 0.0f) { float cc2 = 0.5f * (c2k + c2k), cc1 = 1.0f - cc2; return wbar * (cc1 * A(-1) + cc2 * A(0)); }
    return wbar * flx3(A(1), A(0), A(-1));
  }
  if (kk == nk) {
    if (wbar >= 0.0f) return wbar * flx3(A(-2), A(-1), A(0));
    float cc2 = 0.5f * (c2k + c2k), cc1 = 1.0f - cc2; return wbar * (cc1 * A(-1) + cc2 * A(0));
  }
  if (kk == 3) {
    if (wbar >= 0.0f) return wbar * flx3(A(-2), A(-1), A(0));
    return wbar * flx5(A(2), A(1), A(0), A(-1), A(-2));
  }
  if (wbar >= 0.0f) return wbar * flx5(A(-3), A(-2), A(-1), A(0), A(1));
  return wbar * flx3(A(1), A(0), A(-1));
}

// vertical face flux of a w column at s-level kk; wv[d+2] = w(kk+d), d = -2..3
__device__ __forceinline__ float zflux_w(const DGrid &g, const float *wv, float wbar, int kk) {
  const int nk = g.nk;
  auto A = [&](int d) { return wv[d + 2]; };
  if (kk >= 3 && kk <= nk - 2) {
    const bool up = (wbar >= 0.0f);
    return wbar * flx5(up ? A(-2) : A(3), up ? A(-1) : A(2), up ? A(0) : A(1), up ? A(1) : A(0), up ? A(2) : A(-1));
  }
  if (kk == 1) {
    if (wbar >= 0.0f) return wbar * 0.5f * (A(0) + A(1));
    return wbar * flx3(A(2), A(1), A(0));
  }
  if (kk == nk) {
    if (wbar >= 0.0f) return wbar * flx3(A(-1), A(0), A(1));
    return wbar * 0.5f * (A(0) + A(1));
  }
  if (kk == 2) {
    if (wbar >= 0.0f) return wbar * flx3(A(-1), A(0), A(1));
    return wbar * flx5(A(3), A(2), A(1), A(0), A(-1));
  }
  if (wbar >= 0.0f) return wbar * flx5(A(-2), A(-1), A(0), A(1), A(2));
  return wbar * flx3(A(2), A(1), A(0));
}

__device__ __forceinline__ float hflux_mom(float r, const float *p, int stride) {
  const float a0 = p[0], a1 = p[stride], a2 = p[2 * stride], a3 = p[3 * stride], a4 = p[4 * stride], a5 = p[5 * stride];
  const bool up = (r >= 0.0f);
  return r * flx5(up ? a0 : a5, up ? a1 : a4, up ? a2 : a3, up ? a3 : a2, up ? a4 : a1);
}

template <int TX, int TY, int KC, int STAG>
__global__ void __launch_bounds__(TX * TY, 3) k_mom_tile(DGrid g, Vel q, const float *__restrict__ divx,
                                                      const float *ten1, float *ten,
                                                      const float *__restrict__ th3d, const float *__restrict__ qv,
                                                      const float *__restrict__ b8, Diff6 df) {
  constexpr int NT = TX * TY;
  constexpr int SW = TX + 6, SH = TY + 6, SP = SW + 1;
  constexpr int NST = (SW * SH + NT - 1) / NT;
  constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
  __shared__ float ss[SH * SP];
  __shared__ float fx[NFX], fxv[NFX], fy[NFY], fyv[NFY];
  __shared__ float dfx[NFX], dfy[NFY];     // 6th-order diffusion fluxes
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
  const int i0 = 1 + (int)blockIdx.x * TX, j0 = 1 + (int)blockIdx.y * TY;
  const int i = i0 + tx, j = j0 + ty;
  const int ni = g.ni, nj = g.nj, nk = g.nk;
  const int pitch = (STAG == 2) ? g.NI + 1 : g.NI;      // x extent of the component's array
  const int rows = (STAG == 3) ? g.NJ + 1 : g.NJ;
  const int plane = pitch * rows;   // < 2^31 points (cm1g_init)
  const float *__restrict__ A = (STAG == 2) ? q.u : (STAG == 3) ? q.v : q.w;
  const int ilo = (STAG == 2) ? (g.ibw ? 2 : 1) : 1, ihi = (STAG == 2) ? (g.ibe ? ni : ni + 1) : ni;
  const int jlo = (STAG == 3) ? (g.ibs ? 2 : 1) : 1, jhi = (STAG == 3) ? (g.ibn ? nj : nj + 1) : nj;
  const bool active = (i >= ilo && i <= ihi && j >= jlo && j <= jhi);
  const int iea = ni + g.ngxy + (STAG == 2 ? 1 : 0), jea = nj + g.ngxy + (STAG == 3 ? 1 : 0);
  const bool doitw = (g.wbc == 2 && g.ibw), doite = (g.ebc == 2 && g.ibe);
  const bool doits = (g.sbc == 2 && g.ibs), doitn = (g.nbc == 2 && g.ibn);
  const int oc = active ? (i - g.ib) + pitch * (j - g.jb) : 0;

  int soff[NST], sidx[NST];
#pragma unroll
  for (int s = 0; s < NST; s++) {
    const int t = tid + s * NT;
    soff[s] = -1; sidx[s] = -1;
    if (t < SW * SH) {
      const int yy = t / SW, xx = t - yy * SW;
      const int ii = i0 - 3 + xx, jj = j0 - 3 + yy;
      sidx[s] = yy * SP + xx;
      if (ii <= iea && jj <= jea) soff[s] = (ii - g.ib) + pitch * (jj - g.jb);
    }
  }
  // faces owned by this thread: index-space position (-1 in fxi: none)
  using FS = FaceSlots<NT, NFX, NFY>;
  int fxi[2], fxj[2], fyi[2], fyj[2];
#pragma unroll
  for (int s = 0; s < 2; s++) {
    fxi[s] = -1; fxj[s] = 0; fyi[s] = -1; fyj[s] = 0;
    const int f = FS::x(tid, s), fy_ = FS::y(tid, s);
    if (f < NFX) {
      const int row = f / (TX + 1), col = f - row * (TX + 1);
      const int ii = (STAG == 2) ? i0 - 1 + col : i0 + col, jj = j0 + row;   // s-point (u) or u-point (v, w)
      if (ii >= 0 && ii <= ni + 1 && jj <= nj + 1) { fxi[s] = ii; fxj[s] = jj; }
    }
    if (fy_ < NFY) {
      const int row = fy_ / TX, col = fy_ - row * TX;
      const int ii = i0 + col, jj = (STAG == 3) ? j0 - 1 + row : j0 + row;    // s-point (v) or v-point (u, w)
      if (jj >= 0 && jj <= nj + 1 && ii <= ni + 1) { fyi[s] = ii; fyj[s] = jj; }
    }
  }

  // vertical window: wv[d] = a(kb0 + d), kb0 = upper face - 3 (u, v) or - 2 (w)
  const int kfirst = (STAG == 4) ? 2 : 1;
  const int kc0 = kfirst + (int)blockIdx.z * KC, kc1 = min(nk, kc0 + KC - 1);
  const int koff = (STAG == 4) ? -2 : -3;
  const int kmaxA = (STAG == 4) ? nk + 2 : nk + 1;
  auto AV = [&](int kk) -> float { return (kk >= 0 && kk <= kmaxA) ? LDG(&A[kk * plane + oc]) : 0.0f; };
  auto RRWc = [&](int ii, int jj, int kk) -> float {
    if (kk <= 1 || kk >= nk + 1) return 0.0f;
    return LDG(&g.rf0[kk]) * LDG(&q.w[iW(g, ii, jj, kk)]);
  };
  auto WBAR = [&](int kk) -> float {
    if (STAG == 2) return 0.5f * (RRWc(i, j, kk) + RRWc(i - 1, j, kk));
    if (STAG == 3) return 0.5f * (RRWc(i, j, kk) + RRWc(i, j - 1, kk));
    return 0.5f * (RRWc(i, j, kk) + RRWc(i, j, kk + 1));
  };
  auto ZF = [&](const float *win, int kk) -> float {
    return (STAG == 4) ? zflux_w(g, win, WBAR(kk), kk) : zflux_uv(g, win, WBAR(kk), kk);
  };
  // faces of level k: upper ku, lower ku-1; u/v faces exist for kk = 2..nk, w faces for kk = 1..nk
  const int kfmin = (STAG == 4) ? 1 : 2;
  float wv[6];
  float fzlo = 0.0f;
  {
    const int ku = (STAG == 4) ? kc0 : kc0 + 1;
#pragma unroll
    for (int d = 0; d < 6; d++) wv[d] = active ? AV(ku + koff + d) : 0.0f;
    if (active && ku - 1 >= kfmin) {
      float w0[6];
#pragma unroll
      for (int d = 0; d < 6; d++) w0[d] = AV(ku - 1 + koff + d);
      fzlo = ZF(w0, ku - 1);
    }
  }

  // Every global read of a level is issued one level ahead (into the p*
  // registers), so it is in flight while the previous level computes; the
  // component arrays and the other inputs are not written by this kernel
  // (ten may alias ten1 only point by point).
  float pst[NST], pxa[2], pxb[2], pya[2], pyb[2], pw0 = 0.0f, pw1 = 0.0f, pt1 = 0.0f, pd0 = 0.0f, pd1 = 0.0f;
  float pb0 = 0.0f, pb1 = 0.0f, pb2 = 0.0f, pb3 = 0.0f, pwtop = 0.0f;
  auto fetch = [&](int kf) {
    const float *Ak = A + kf * plane;
#pragma unroll
    for (int s = 0; s < NST; s++) pst[s] = (soff[s] >= 0) ? LDG(&Ak[soff[s]]) : 0.0f;
#pragma unroll
    for (int s = 0; s < 2; s++) {
      pxa[s] = pxb[s] = pya[s] = pyb[s] = 0.0f;
      if (fxi[s] >= 0) {
        const int ii = fxi[s], jj = fxj[s];
        if (STAG == 3) { pxa[s] = LDG(&q.u[iU(g, ii, jj, kf)]); pxb[s] = LDG(&q.u[iU(g, ii, jj - 1, kf)]); }
        if (STAG == 4) { pxa[s] = LDG(&q.u[iU(g, ii, jj, kf)]); pxb[s] = LDG(&q.u[iU(g, ii, jj, kf - 1)]); }
      }
      if (fyi[s] >= 0) {
        const int ii = fyi[s], jj = fyj[s];
        if (STAG == 2) { pya[s] = LDG(&q.v[iV(g, ii, jj, kf)]); pyb[s] = LDG(&q.v[iV(g, ii - 1, jj, kf)]); }
        if (STAG == 4) { pya[s] = LDG(&q.v[iV(g, ii, jj, kf)]); pyb[s] = LDG(&q.v[iV(g, ii, jj, kf - 1)]); }
      }
    }
    if (active) {
      const int ku = (STAG == 4) ? kf : kf + 1;       // upper face of level kf
      if (ku <= nk) {
        const int ia = (STAG == 2) ? i - 1 : i, ja = (STAG == 3) ? j - 1 : j, ka = (STAG == 4) ? ku + 1 : ku;
        pw0 = (ku <= 1 || ku >= nk + 1) ? 0.0f : LDG(&q.w[iW(g, i, j, ku)]);
        pw1 = (ka <= 1 || ka >= nk + 1) ? 0.0f : LDG(&q.w[iW(g, ia, ja, ka)]);
      }
      const int oS = (int)iS(g, i, j, kf);
      pt1 = ten1[kf * plane + oc];
      pd0 = LDG(&divx[oS]);
      pd1 = LDG(&divx[oS - ((STAG == 2) ? 1 : (STAG == 3) ? g.NI : g.NI * g.NJ)]);
      if (STAG == 4 && b8) {          // buoyancy of the stage set-up (liquid water present)
        pb0 = LDG(&b8[oS - g.NI * g.NJ]); pb1 = LDG(&b8[oS]);
      } else if (STAG == 4 && th3d) {
        pb0 = LDG(&th3d[oS - g.NI * g.NJ]); pb1 = LDG(&th3d[oS]);
        if (qv) { pb2 = LDG(&qv[oS - g.NI * g.NJ]); pb3 = LDG(&qv[oS]); }
      }
      pwtop = AV(ku + koff + 5);
    }
  };
  // wbar of face kk from its two averaged w values (RRW of solve2.F:509-516)
  auto WBARp = [&](int kk, float w0, float w1) -> float {
    const int ka = (STAG == 4) ? kk + 1 : kk;
    const float r0 = (kk <= 1 || kk >= nk + 1) ? 0.0f : LDG(&g.rf0[kk]) * w0;
    const float r1 = (ka <= 1 || ka >= nk + 1) ? 0.0f : LDG(&g.rf0[ka]) * w1;
    return 0.5f * (r0 + r1);
  };
  fetch(kc0);

  for (int k = kc0; k <= kc1; k++) {
    const float r0k = LDG(&g.rho0[k]);
#pragma unroll
    for (int s = 0; s < NST; s++)
      if (sidx[s] >= 0) ss[sidx[s]] = pst[s];
    // face velocities that come from the other components
    float ubar[2] = {0.0f, 0.0f}, vbar[2] = {0.0f, 0.0f};
    float c1k = 0.0f, c2k = 0.0f, cc1 = 0.0f, cc2 = 0.0f;
    if (STAG == 4) {
      c1k = LDG(&g.c1[k]); c2k = LDG(&g.c2[k]);
      cc2 = 0.5f * (c2k + c2k); cc1 = 1.0f - cc2;
    }
#pragma unroll
    for (int s = 0; s < 2; s++) {
      if (STAG == 3) ubar[s] = 0.5f * (r0k * pxa[s] + r0k * pxb[s]);
      if (STAG == 4) ubar[s] = cc2 * (r0k * pxa[s]) + cc1 * (LDG(&g.rho0[k - 1]) * pxb[s]);
      if (STAG == 2) vbar[s] = 0.5f * (r0k * pya[s] + r0k * pyb[s]);
      if (STAG == 4) vbar[s] = cc2 * (r0k * pya[s]) + cc1 * (LDG(&g.rho0[k - 1]) * pyb[s]);
    }
    const float w0 = pw0, w1 = pw1, t1 = pt1, dv0 = pd0, dv1 = pd1, b0 = pb0, b1 = pb1, b2 = pb2, b3 = pb3;
    if (k < kc1) fetch(k + 1);
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int f = FS::x(tid, s);
      if (fxi[s] >= 0) {
        const int row = f / (TX + 1), col = f - row * (TX + 1);
        const float *p = &ss[(row + 3) * SP + col];
        float r = ubar[s];
        if (STAG == 2) r = 0.5f * (r0k * p[2] + r0k * p[3]);
        fx[f] = hflux_mom(r, p, 1);
        fxv[f] = r;
        {
          // the face between p[2] and p[3]: s-point fxi (u: adv.F:1190-1193),
          // u-point fxi (v: adv.F:2128-2132; w: adv.F:3124-3130)
          const int ii = fxi[s], jj = fxj[s];
          const float d = diff6_stencil(p[0], p[1], p[2], p[3], p[4], p[5]);
          float fd;
          if (STAG == 2) {
            fd = d * LDG(&df.rho[iS(g, ii, jj, k)]);
          } else if (STAG == 3) {
            fd = d * 0.25f * ((LDG(&df.rho[iS(g, ii - 1, jj - 1, k)]) + LDG(&df.rho[iS(g, ii, jj, k)])) +
                              (LDG(&df.rho[iS(g, ii - 1, jj, k)]) + LDG(&df.rho[iS(g, ii, jj - 1, k)])));
          } else {
            fd = d * 0.5f * (cc2 * (LDG(&df.rho[iS(g, ii - 1, jj, k)]) + LDG(&df.rho[iS(g, ii, jj, k)])) +
                             cc1 * (LDG(&df.rho[iS(g, ii - 1, jj, k - 1)]) + LDG(&df.rho[iS(g, ii, jj, k - 1)])));
          }
          dfx[f] = diff6_limit(fd, p[3], p[2], df.mdiff);
        }
      }
      if (fyi[s] >= 0) {
        const int fy_ = FS::y(tid, s);
        const int row = fy_ / TX, col = fy_ - row * TX;
        const float *p = &ss[row * SP + col + 3];
        float r = vbar[s];
        if (STAG == 3) r = 0.5f * (r0k * p[2 * SP] + r0k * p[3 * SP]);
        fy[fy_] = hflux_mom(r, p, SP);
        fyv[fy_] = r;
        {
          // the face between p[2 SP] and p[3 SP]: v-point fyj (u: adv.F:1210-1215;
          // w: adv.F:3146-3152), s-point fyj (v: adv.F:2151-2153)
          const int ii = fyi[s], jj = fyj[s];
          const float d = diff6_stencil(p[0], p[SP], p[2 * SP], p[3 * SP], p[4 * SP], p[5 * SP]);
          float fd;
          if (STAG == 2) {
            fd = d * 0.25f * ((LDG(&df.rho[iS(g, ii - 1, jj - 1, k)]) + LDG(&df.rho[iS(g, ii, jj, k)])) +
                              (LDG(&df.rho[iS(g, ii - 1, jj, k)]) + LDG(&df.rho[iS(g, ii, jj - 1, k)])));
          } else if (STAG == 3) {
            fd = d * LDG(&df.rho[iS(g, ii, jj, k)]);
          } else {
            fd = d * 0.5f * (cc2 * (LDG(&df.rho[iS(g, ii, jj - 1, k)]) + LDG(&df.rho[iS(g, ii, jj, k)])) +
                             cc1 * (LDG(&df.rho[iS(g, ii, jj - 1, k - 1)]) + LDG(&df.rho[iS(g, ii, jj, k - 1)])));
          }
          dfy[fy_] = diff6_limit(fd, p[3 * SP], p[2 * SP], df.mdiff);
        }
      }
    }
    const int ku = (STAG == 4) ? k : k + 1;
    float fzhi = 0.0f, ac = 0.0f;
    if (active) {
      ac = ss[(ty + 3) * SP + tx + 3];
      if (ku <= nk) {
        const float wb = WBARp(ku, w0, w1);
        fzhi = (STAG == 4) ? zflux_w(g, wv, wb, ku) : zflux_uv(g, wv, wb, ku);
      }
    }
    __syncthreads();
    if (active) {
      const int xi = ty * (TX + 1) + tx, yi = ty * TX + tx;
      float fx0 = fx[xi], fxp = fx[xi + 1], fy0 = fy[yi], fyp = fy[yi + TX];
      float advx, advy, advz;
      const int oS = (int)iS(g, i, j, k);
      if (STAG == 2) {
        auto RRV2 = [&](int ii, int jj) { return LDG(&g.rho0[k]) * LDG(&q.v[iV(g, ii, jj, k)]); };
        advx = -(fxp - fx0) * g.rdx * LDG(&g.uf[i - g.ib]);
        const bool fs = doits && j == 1 && (RRV2(i, 1) + RRV2(i - 1, 1)) >= 0.0f;
        const bool fn = doitn && j == nj && (RRV2(i, nj + 1) + RRV2(i - 1, nj + 1)) <= 0.0f;
        if (fs) fy0 = fyp;
        if (fn) fyp = fy0;
        advy = -(fyp - fy0) * g.rdy * LDG(&g.vh[j - g.jb]);
        if (fs)
          advy = advy - LDG(&q.u[iU(g, i, 1, k)]) * 0.5f *
                            ((RRV2(i - 1, 2) - RRV2(i - 1, 1)) + (RRV2(i, 2) - RRV2(i, 1))) * g.rdy * LDG(&g.vh[1 - g.jb]);
        if (fn)
          advy = advy - LDG(&q.u[iU(g, i, nj, k)]) * 0.5f *
                            ((RRV2(i - 1, nj + 1) - RRV2(i - 1, nj)) + (RRV2(i, nj + 1) - RRV2(i, nj))) * g.rdy *
                            LDG(&g.vh[nj - g.jb]);
      } else if (STAG == 3) {
        auto RRU2 = [&](int ii, int jj) { return LDG(&g.rho0[k]) * LDG(&q.u[iU(g, ii, jj, k)]); };
        const bool fw = doitw && i == 1 && (RRU2(1, j) + RRU2(1, j - 1)) >= 0.0f;
        const bool fe = doite && i == ni && (RRU2(ni + 1, j) + RRU2(ni + 1, j - 1)) <= 0.0f;
        if (fw) fx0 = fxp;
        if (fe) fxp = fx0;
        advx = -(fxp - fx0) * g.rdx * LDG(&g.uh[i - g.ib]);
        advy = -(fyp - fy0) * g.rdy * LDG(&g.vf[j - g.jb]);
        if (fw)
          advx = advx - LDG(&q.v[iV(g, 1, j, k)]) * 0.5f *
                            ((RRU2(2, j - 1) - RRU2(1, j - 1)) + (RRU2(2, j) - RRU2(1, j))) * g.rdx * LDG(&g.uh[1 - g.ib]);
        if (fe)
          advx = advx - LDG(&q.v[iV(g, ni, j, k)]) * 0.5f *
                            ((RRU2(ni + 1, j - 1) - RRU2(ni, j - 1)) + (RRU2(ni + 1, j) - RRU2(ni, j))) * g.rdx *
                            LDG(&g.uh[ni - g.ib]);
      } else {
        const float ub0 = fxv[xi], ubp = fxv[xi + 1], vb0 = fyv[yi], vbp = fyv[yi + TX];
        const bool fw = doitw && i == 1 && ub0 >= 0.0f, fe = doite && i == ni && ubp <= 0.0f;
        const bool fs = doits && j == 1 && vb0 >= 0.0f, fn = doitn && j == nj && vbp <= 0.0f;
        if (fw) fx0 = fxp;
        if (fe) fxp = fx0;
        if (fs) fy0 = fyp;
        if (fn) fyp = fy0;
        advx = -(fxp - fx0) * g.rdx * LDG(&g.uh[i - g.ib]);
        advy = -(fyp - fy0) * g.rdy * LDG(&g.vh[j - g.jb]);
        auto RRUk = [&](int ii, int kk) { return LDG(&g.rho0[kk]) * LDG(&q.u[iU(g, ii, j, kk)]); };
        auto RRVk = [&](int jj, int kk) { return LDG(&g.rho0[kk]) * LDG(&q.v[iV(g, i, jj, kk)]); };
        const float ww = ac;
        if (fw)
          advx = advx - ww * (c1k * (RRUk(2, k - 1) - RRUk(1, k - 1)) + c2k * (RRUk(2, k) - RRUk(1, k))) * g.rdx *
                            LDG(&g.uh[1 - g.ib]);
        if (fe)
          advx = advx - ww * (c1k * (RRUk(ni + 1, k - 1) - RRUk(ni, k - 1)) + c2k * (RRUk(ni + 1, k) - RRUk(ni, k))) *
                            g.rdx * LDG(&g.uh[ni - g.ib]);
        if (fs)
          advy = advy - ww * (c1k * (RRVk(2, k - 1) - RRVk(1, k - 1)) + c2k * (RRVk(2, k) - RRVk(1, k))) * g.rdy *
                            LDG(&g.vh[1 - g.jb]);
        if (fn)
          advy = advy - ww * (c1k * (RRVk(nj + 1, k - 1) - RRVk(nj, k - 1)) + c2k * (RRVk(nj + 1, k) - RRVk(nj, k))) *
                            g.rdy * LDG(&g.vh[nj - g.jb]);
      }
      {   // adv.F:1199-1201, 1220-1222; 2139-2141, 2160-2162; 3135-3137, 3160-3162
        const float ddx = df.coef * (dfx[xi + 1] - dfx[xi]), ddy = df.coef * (dfy[yi + TX] - dfy[yi]);
        if (STAG == 2) {
          const float rs = LDG(&df.rho[iS(g, i - 1, j, k)]) + LDG(&df.rho[iS(g, i, j, k)]);
          advx = advx + ddx * (r0k + r0k) / rs;
          advy = advy + ddy * (r0k + r0k) / rs;
        } else if (STAG == 3) {
          const float rs = LDG(&df.rho[iS(g, i, j - 1, k)]) + LDG(&df.rho[iS(g, i, j, k)]);
          advx = advx + ddx * (r0k + r0k) / rs;
          advy = advy + ddy * (r0k + r0k) / rs;
        } else {
          const float rf = LDG(&g.rf0[k]);
          const float rs = 0.5f * (LDG(&df.rho[iS(g, i, j, k - 1)]) + LDG(&df.rho[iS(g, i, j, k)]));
          advx = advx + ddx * rf / rs;
          advy = advy + ddy * rf / rs;
        }
      }
      if (STAG == 4) {
        advz = -(fzhi - fzlo) * g.rdz * LDG(&g.mf[k]);
      } else {
        const float mhk = LDG(&g.mh[k]);
        if (k == 1) advz = -fzhi * g.rdz * mhk;
        else if (k == nk) advz = +fzlo * g.rdz * mhk;
        else advz = -(fzhi - fzlo) * g.rdz * mhk;
      }
      const int o = k * plane + oc;
      if (STAG == 2) {
        ten[o] = t1 + (((advx + advy) + advz) + ac * 0.5f * (dv0 + dv1)) * LDG(&g.rr0[k]);
      } else if (STAG == 3) {
        ten[o] = t1 + (((advx + advy) + advz) + ac * 0.5f * (dv0 + dv1)) * LDG(&g.rr0[k]);
      } else {
        float t = t1 + (((advx + advy) + advz) + ac * (c2k * dv0 + c1k * dv1)) * LDG(&g.rrf0[k]);
        if (b8) t = t + (c1k * b0 + c2k * b1);
        else if (th3d) t = t + (c1k * buoy_v(g, b0, b2, qv != nullptr, k - 1) + c2k * buoy_v(g, b1, b3, qv != nullptr, k));
        ten[o] = t;
      }
#pragma unroll
      for (int d = 0; d < 5; d++) wv[d] = wv[d + 1];
      wv[5] = pwtop;            // top of the window of level k+1 (fetched above)
      fzlo = fzhi;
    }
  }
}

// ---------------------------------------------------------------------
// Momentum advection of all three components in one pass (advu, advv, advw).
//
// A block owns 31 x (TY-1) points and KC levels and marches upward.  u, v and
// w of a level are staged once, with their 3-point halo, by asynchronous
// copies into a ring of six levels (k-1, k, k+1 in use, three in flight) and
// serve as the advected field of their own component and as the face
// velocities and divergence of all three.  Thread (lane, row) evaluates, for
// every component, the x face west of its point, the y face south of it and
// the z face above it (hadv_flx5/vadv_flx5, stag=2/3/4): the east face comes
// from the next lane by a shuffle, the north face from the next row through
// shared memory, the lower face from the level below in registers; the last
// lane and row only supply faces.  The face velocities are formed exactly as
// the reference forms them (ubar/vbar/wbar of adv_routines.F:1388-1460,
// 3299-3384), divx as solve2.F:590-596 does, and the open-boundary fixes of
// adv.F are applied in the blocks that touch an open edge.
//
// Bound by instruction issue and latency: 890 warp instructions per 32 points
// at 60 % issue with 17 warps an SM; DRAM moves 159 MB (9 % of the peak), less than
// the arrays because L2 keeps part of the tendencies.  256x256x80: 0.230 ms against 0.370
// for a divergence pass and one marching tile per component, which staged u, v
// and w separately and read them again as face velocities; 64x64x40: 27 us
// against 62.  Three blocks an SM at 72 registers spill and measured 4 to 14 %
// slower than two at 96; 16 rows of threads 5 to 15 % slower than 9.
// ---------------------------------------------------------------------
// vertical profiles of one level
struct MomLev { float rho0, c1, c2, rf0, mh, rr0, rrf0, mf; };
constexpr int MOM_TY = 9;          // rows of threads
constexpr int MOM_KC = 64;         // levels of a block at most

struct MomIO {
  const float *uten1, *vten1, *wten1;
  float *uten, *vten, *wten;
  const float *th3d, *qv, *b8;     // buoyancy of w: theta and qv, or the array of the stage set-up, or none
};

__device__ __forceinline__ void cp_async4(void *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int WHICH>
__global__ void __launch_bounds__(32 * MOM_TY, 2) k_mom(DGrid g, Vel q, MomIO io, int kc) {
  constexpr int TY = MOM_TY;
  constexpr int NT = 32 * TY;
  constexpr int SW = 38, SH = TY + 6, SP = 40;             // staged columns, rows and pitch
  constexpr int NST = (SW * SH + NT - 1) / NT;
  constexpr int PLANE = SH * SP;
  constexpr bool DU = (WHICH & 1) != 0, DV = (WHICH & 2) != 0, DW = (WHICH & 4) != 0;
  constexpr int RD = 6;
  __shared__ float ring[RD][3][PLANE];
  __shared__ float fyu[TY][32], fyv[TY][32], fyw[TY][32];
  extern __shared__ float4 mom_lev[];    // levels kc0-1 .. kc1+1
  const int lane = threadIdx.x, row = threadIdx.y, tid = lane + 32 * row;
  const int i0 = 1 + (int)blockIdx.x * 31, j0 = 1 + (int)blockIdx.y * (TY - 1);
  const int i = i0 + lane, j = j0 + row;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI;
  const int plS = NI * g.NJ, plU = (NI + 1) * g.NJ, plV = NI * (g.NJ + 1);   // < 2^31 points (cm1g_init)
  const bool in = i <= ni + 2 && j <= nj + 2;              // the last u and v points need the face beyond them
  const bool own = i <= ni + 1 && j <= nj + 1 && lane < 31 && row < TY - 1;
  const bool own_u = DU && own && i >= (g.ibw ? 2 : 1) && i <= (g.ibe ? ni : ni + 1) && j <= nj;
  const bool own_v = DV && own && j >= (g.ibs ? 2 : 1) && j <= (g.ibn ? nj : nj + 1) && i <= ni;
  const bool own_w = DW && own && i <= ni && j <= nj;
  const bool doitw = g.wbc == 2 && g.ibw, doite = g.ebc == 2 && g.ibe;
  const bool doits = g.sbc == 2 && g.ibs, doitn = g.nbc == 2 && g.ibn;
  const bool edge = (doitw && i0 == 1) || (doite && i0 + 31 >= ni) || (doits && j0 == 1) || (doitn && j0 + TY - 1 >= nj);
  const int oc = in ? (i - g.ib) + NI * (j - g.jb) : 0, ocu = in ? (i - g.ib) + (NI + 1) * (j - g.jb) : 0;
  const int kc0 = 1 + (int)blockIdx.z * kc, kc1 = min(nk, kc0 + kc - 1);
  const float rdx = g.rdx, rdy = g.rdy, rdz = g.rdz, smeps = g.smeps;
  float uh = 0, uhw = 0, vh = 0, vhs = 0, uf = 0, vf = 0;
  if (in) {
    uh = LDG(&g.uh[i - g.ib]); uhw = LDG(&g.uh[i - 1 - g.ib]); uf = LDG(&g.uf[i - g.ib]);
    vh = LDG(&g.vh[j - g.jb]); vhs = LDG(&g.vh[j - 1 - g.jb]); vf = LDG(&g.vf[j - g.jb]);
  }

  MomLev *LV = reinterpret_cast<MomLev *>(mom_lev) - (kc0 - 1);
  for (int k = kc0 - 1 + tid; k <= kc1 + 1; k += NT) {
    LV[k] = MomLev{LDG(&g.rho0[k]), LDG(&g.c1[k]), LDG(&g.c2[k]), LDG(&g.rf0[k]), LDG(&g.mh[k]), LDG(&g.rr0[k]),
                   LDG(&g.rrf0[k]), LDG(&g.mf[k])};
  }

  // ---- staging
  int so[NST], sd[NST];            // in-plane source offset of an s-shaped plane (-1: none), slot
  unsigned sm = 0;                 // bit s: row exists in u and w; bit 8+s: in v; the u offset is so + (jj - jb)
  int sr[NST];
#pragma unroll
  for (int s = 0; s < NST; s++) {
    const int t = tid + s * NT;
    so[s] = 0; sd[s] = 0; sr[s] = 0;
    if (t < SW * SH) {
      const int yy = t / SW, xx = t - yy * SW;
      const int ii = i0 - 3 + xx, jj = j0 - 3 + yy;
      sd[s] = yy * SP + xx;
      so[s] = (ii - g.ib) + NI * (jj - g.jb);
      sr[s] = jj - g.jb;
      if (ii <= ni + g.ngxy + 1 && jj <= nj + g.ngxy) sm |= 1u << s;                   // u
      if (ii <= ni + g.ngxy && jj <= nj + g.ngxy + 1) sm |= 0x100u << s;               // v
      if (ii <= ni + g.ngxy && jj <= nj + g.ngxy) sm |= 0x10000u << s;                 // w
    }
  }
  int slot = 0, lev = kc0 - 1;     // next slot and level to stage
  auto issue = [&]() {
    float *d = &ring[slot][0][0];
    const int k = lev++;
    slot = slot + 1 == RD ? 0 : slot + 1;
#pragma unroll
    for (int s = 0; s < NST && k <= kc1 + 1; s++) {
      if (sm & (1u << s)) cp_async4(d + sd[s], q.u + (k * plU + so[s] + sr[s]));
      if (sm & (0x100u << s)) cp_async4(d + PLANE + sd[s], q.v + (k * plV + so[s]));
      if (sm & (0x10000u << s)) cp_async4(d + 2 * PLANE + sd[s], q.w + (k * plS + so[s]));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int d = 0; d < RD - 1; d++) issue();

  // ---- column windows: a(k-2 .. k+3) of each component
  auto AU = [&](int kk) -> float { return (kk >= 0 && kk <= nk + 1) ? LDG(&q.u[kk * plU + ocu]) : 0.0f; };
  auto AV = [&](int kk) -> float { return (kk >= 0 && kk <= nk + 1) ? LDG(&q.v[kk * plV + oc]) : 0.0f; };
  auto AW = [&](int kk) -> float { return (kk >= 0 && kk <= nk + 2) ? LDG(&q.w[kk * plS + oc]) : 0.0f; };
  // rf0-weighted w of a neighbour column (offset d) at w-level kk (solve2.F:509-516)
  auto RWg = [&](int kk, float rf, float w) -> float { return (kk <= 1 || kk >= nk + 1) ? 0.0f : rf * w; };
  auto RW = [&](int kk, float w) -> float { return RWg(kk, LDG(&g.rf0[kk]), w); };
  float uw[6], vw[6], ww[6];
  float fzu = 0.0f, fzv = 0.0f, fzw = 0.0f, divm = 0.0f;
#pragma unroll
  for (int d = 0; d < 6; d++) { uw[d] = vw[d] = ww[d] = 0.0f; }
  if (own) {
#pragma unroll
    for (int d = 0; d < 6; d++) {
      if (DU) uw[d] = AU(kc0 - 2 + d);
      if (DV) vw[d] = AV(kc0 - 2 + d);
      if (DW) ww[d] = AW(kc0 - 2 + d);
    }
    if (kc0 >= 2) {                 // the faces below level kc0
      const float rc = RW(kc0, LDG(&q.w[kc0 * plS + oc]));
      float z[6];
      if (DU) {
        z[0] = AU(kc0 - 3);
#pragma unroll
        for (int d = 0; d < 5; d++) z[d + 1] = uw[d];
        fzu = zflux_uv(g, z, 0.5f * (rc + RW(kc0, LDG(&q.w[kc0 * plS + oc - 1]))), kc0);
      }
      if (DV) {
        z[0] = AV(kc0 - 3);
#pragma unroll
        for (int d = 0; d < 5; d++) z[d + 1] = vw[d];
        fzv = zflux_uv(g, z, 0.5f * (rc + RW(kc0, LDG(&q.w[kc0 * plS + oc - NI]))), kc0);
      }
      if (DW) {
        z[0] = AW(kc0 - 3);
#pragma unroll
        for (int d = 0; d < 5; d++) z[d + 1] = ww[d];
        fzw = zflux_w(g, z, 0.5f * (RW(kc0 - 1, LDG(&q.w[(kc0 - 1) * plS + oc])) + rc), kc0 - 1);
      }
    }
  }
  // buoyancy of a level: from its theta and qv, or as the stage set-up left it
  auto buoy = [&](float t, float q, int k) -> float {
    return io.b8 ? t : io.th3d ? buoy_v(g, t, q, io.qv != nullptr, k) : 0.0f;
  };
  float bu0 = 0.0f;                // of level k-1
  if (own_w && kc0 >= 2) {
    const int o = (kc0 - 1) * plS + oc;
    float t = 0.0f, qq = 0.0f;
    if (io.b8) t = LDG(&io.b8[o]);
    else if (io.th3d) { t = LDG(&io.th3d[o]); if (io.qv) qq = LDG(&io.qv[o]); }
    bu0 = buoy(t, qq, kc0 - 1);
  }
  const int pc = (row + 3) * SP + lane + 3;                // the point in a staged plane
  // rho0-weighted velocities of a staged level (solve2.F:499-516) and divx (solve2.F:590-596)
  auto DIV = [&](const float *P, const float *Pup, int k, const MomLev &lv, float rfu, int d, float uhd, float vhd) -> float {
    const float r0 = lv.rho0;
    const float *u = P + pc + d, *v = P + PLANE + pc + d;
    float x = ((r0 * u[1] - r0 * u[0]) * rdx * uhd + (r0 * v[SP] - r0 * v[0]) * rdy * vhd) +
              (RWg(k + 1, rfu, Pup[2 * PLANE + pc + d]) - RWg(k, lv.rf0, P[2 * PLANE + pc + d])) * rdz * lv.mh;
    if (fabsf(x) < smeps) x = 0.0f;
    return x;
  };

  int sl = 0;                      // slot of level k-1
  for (int k = kc0; k <= kc1; k++) {
    // this level's own inputs and the next tops of the column windows
    float t1u = 0, t1v = 0, t1w = 0, nu = 0, nv = 0, nw = 0, tb1 = 0, tq1 = 0;
    const int ou = k * plU + ocu, ov = k * plV + oc, ow = k * plS + oc;
    if (own_u) t1u = io.uten1[ou];
    if (own_v) t1v = io.vten1[ov];
    if (own_w) {
      t1w = k >= 2 ? io.wten1[ow] : 0.0f;
      if (io.b8) tb1 = LDG(&io.b8[ow]);
      else if (io.th3d) { tb1 = LDG(&io.th3d[ow]); if (io.qv) tq1 = LDG(&io.qv[ow]); }
    }
    if (own) {
      if (DU) nu = AU(k + 4);
      if (DV) nv = AV(k + 4);
      if (DW) nw = AW(k + 4);
    }
    if (own && k + 3 <= kc1) {      // levels ahead towards L2
      if (own_u) prefetch_l2(&io.uten1[ou + 3 * plU]);
      if (own_v) prefetch_l2(&io.vten1[ov + 3 * plV]);
      if (own_w) {
        prefetch_l2(&io.wten1[ow + 3 * plS]);
        if (io.b8) prefetch_l2(&io.b8[ow + 3 * plS]);
        else if (io.th3d) { prefetch_l2(&io.th3d[ow + 3 * plS]); if (io.qv) prefetch_l2(&io.qv[ow + 3 * plS]); }
      }
    }
    // groups are committed one a level, up to k+3 here: level k+1 has landed
    asm volatile("cp.async.wait_group %0;" ::"n"(RD - 4) : "memory");
    __syncthreads();
    issue();                       // level k+4 into the slot of level k-2
    const int s0 = sl + 1 >= RD ? sl + 1 - RD : sl + 1, s1 = s0 + 1 == RD ? 0 : s0 + 1;
    const float *Pm = &ring[sl][0][0], *P = &ring[s0][0][0], *Pp = &ring[s1][0][0];
    sl = s0;
    const MomLev lv = LV[k];
    const float r0k = lv.rho0, r0m = LV[k - 1].rho0, rfu = LV[k + 1].rf0, c1k = lv.c1, c2k = lv.c2;
    const float cc2 = 0.5f * (c2k + c2k), cc1 = 1.0f - cc2;
    float fxu = 0, fxv = 0, fxw = 0, fyu0 = 0, fyv0 = 0, fyw0 = 0, rxw = 0, ryw = 0;
    const float *pu = P + pc, *pv = P + PLANE + pc, *pw = P + 2 * PLANE + pc;
    if (in) {
      if (DU) {
        fxu = hflux_mom(0.5f * (r0k * pu[-1] + r0k * pu[0]), pu - 3, 1);
        fyu0 = hflux_mom(0.5f * (r0k * pv[0] + r0k * pv[-1]), pu - 3 * SP, SP);
      }
      if (DV) {
        fxv = hflux_mom(0.5f * (r0k * pu[0] + r0k * pu[-SP]), pv - 3, 1);
        fyv0 = hflux_mom(0.5f * (r0k * pv[-SP] + r0k * pv[0]), pv - 3 * SP, SP);
      }
      if (DW && k >= 2) {
        rxw = cc2 * (r0k * pu[0]) + cc1 * (r0m * Pm[pc]);
        ryw = cc2 * (r0k * pv[0]) + cc1 * (r0m * Pm[PLANE + pc]);
        fxw = hflux_mom(rxw, pw - 3, 1);
        fyw0 = hflux_mom(ryw, pw - 3 * SP, SP);
      }
    }
    if (DU) fyu[row][lane] = fyu0;
    if (DV) fyv[row][lane] = fyv0;
    if (DW) fyw[row][lane] = fyw0;
    float fxu1 = 0, fxv1 = 0, fxw1 = 0;
    if (DU) fxu1 = __shfl_down_sync(0xffffffffu, fxu, 1);
    if (DV) fxv1 = __shfl_down_sync(0xffffffffu, fxv, 1);
    if (DW) fxw1 = __shfl_down_sync(0xffffffffu, fxw, 1);
    float hzu = 0, hzv = 0, hzw = 0, div0 = 0, divx = 0, divy = 0;
    if (own) {
      // the faces above: w-level k+1 for u and v, s-level k for w
      const float *wu = Pp + 2 * PLANE + pc;
      const float rc = RWg(k + 1, rfu, wu[0]);
      if (k + 1 <= nk) {
        if (DU) hzu = zflux_uv(g, uw, 0.5f * (rc + RWg(k + 1, rfu, wu[-1])), k + 1);
        if (DV) hzv = zflux_uv(g, vw, 0.5f * (rc + RWg(k + 1, rfu, wu[-SP])), k + 1);
      }
      if (DW) hzw = zflux_w(g, ww, 0.5f * (RWg(k, lv.rf0, pw[0]) + rc), k);
      if (DW && k == kc0 && k >= 2) divm = DIV(Pm, P, k - 1, LV[k - 1], lv.rf0, 0, uh, vh);
      div0 = DIV(P, Pp, k, lv, rfu, 0, uh, vh);
      if (DU) divx = DIV(P, Pp, k, lv, rfu, -1, uhw, vh);
      if (DV) divy = DIV(P, Pp, k, lv, rfu, -SP, uh, vhs);
    }
    __syncthreads();
    if (own_u) {
      const float ac = pu[0];
      float fy0 = fyu0, fyp = fyu[row + 1][lane];
      float advx = -(fxu1 - fxu) * rdx * uf, advy;
      if (!edge) {
        advy = -(fyp - fy0) * rdy * vh;
      } else {
        const bool fs = doits && j == 1 && (r0k * pv[0] + r0k * pv[-1]) >= 0.0f;
        const bool fn = doitn && j == nj && (r0k * pv[SP] + r0k * pv[SP - 1]) <= 0.0f;
        if (fs) fy0 = fyp;
        if (fn) fyp = fy0;
        advy = -(fyp - fy0) * rdy * vh;
        const float dd = ((r0k * pv[SP - 1] - r0k * pv[-1]) + (r0k * pv[SP] - r0k * pv[0]));
        if (fs) advy = advy - ac * 0.5f * dd * rdy * vh;
        if (fn) advy = advy - ac * 0.5f * dd * rdy * vh;
      }
      const float mhk = lv.mh;
      float advz;
      if (k == 1) advz = -hzu * rdz * mhk;
      else if (k == nk) advz = +fzu * rdz * mhk;
      else advz = -(hzu - fzu) * rdz * mhk;
      io.uten[ou] = t1u + (((advx + advy) + advz) + ac * 0.5f * (div0 + divx)) * lv.rr0;
    }
    if (own_v) {
      const float ac = pv[0];
      float fx0 = fxv, fxp = fxv1;
      float advx;
      const float advy = -(fyv[row + 1][lane] - fyv0) * rdy * vf;
      if (!edge) {
        advx = -(fxp - fx0) * rdx * uh;
      } else {
        const bool fw = doitw && i == 1 && (r0k * pu[0] + r0k * pu[-SP]) >= 0.0f;
        const bool fe = doite && i == ni && (r0k * pu[1] + r0k * pu[1 - SP]) <= 0.0f;
        if (fw) fx0 = fxp;
        if (fe) fxp = fx0;
        advx = -(fxp - fx0) * rdx * uh;
        const float dd = ((r0k * pu[1 - SP] - r0k * pu[-SP]) + (r0k * pu[1] - r0k * pu[0]));
        if (fw) advx = advx - ac * 0.5f * dd * rdx * uh;
        if (fe) advx = advx - ac * 0.5f * dd * rdx * uh;
      }
      const float mhk = lv.mh;
      float advz;
      if (k == 1) advz = -hzv * rdz * mhk;
      else if (k == nk) advz = +fzv * rdz * mhk;
      else advz = -(hzv - fzv) * rdz * mhk;
      io.vten[ov] = t1v + (((advx + advy) + advz) + ac * 0.5f * (div0 + divy)) * lv.rr0;
    }
    const float bu1 = own_w ? buoy(tb1, tq1, k) : 0.0f;
    if (own_w && k >= 2) {
      const float ac = pw[0];
      float fx0 = fxw, fxp = fxw1, fy0 = fyw0, fyp = fyw[row + 1][lane];
      float advx, advy;
      if (!edge) {
        advx = -(fxp - fx0) * rdx * uh;
        advy = -(fyp - fy0) * rdy * vh;
      } else {
        const float *mu = Pm + pc, *mv = Pm + PLANE + pc;
        const float rxe = cc2 * (r0k * pu[1]) + cc1 * (r0m * mu[1]), ryn = cc2 * (r0k * pv[SP]) + cc1 * (r0m * mv[SP]);
        const bool fw = doitw && i == 1 && rxw >= 0.0f, fe = doite && i == ni && rxe <= 0.0f;
        const bool fs = doits && j == 1 && ryw >= 0.0f, fn = doitn && j == nj && ryn <= 0.0f;
        if (fw) fx0 = fxp;
        if (fe) fxp = fx0;
        if (fs) fy0 = fyp;
        if (fn) fyp = fy0;
        advx = -(fxp - fx0) * rdx * uh;
        advy = -(fyp - fy0) * rdy * vh;
        const float dx = c1k * (r0m * mu[1] - r0m * mu[0]) + c2k * (r0k * pu[1] - r0k * pu[0]);
        const float dy = c1k * (r0m * mv[SP] - r0m * mv[0]) + c2k * (r0k * pv[SP] - r0k * pv[0]);
        if (fw) advx = advx - ac * dx * rdx * uh;
        if (fe) advx = advx - ac * dx * rdx * uh;
        if (fs) advy = advy - ac * dy * rdy * vh;
        if (fn) advy = advy - ac * dy * rdy * vh;
      }
      const float advz = -(hzw - fzw) * rdz * lv.mf;
      float t = t1w + (((advx + advy) + advz) + ac * (c2k * div0 + c1k * divm)) * lv.rrf0;
      if (io.b8 || io.th3d) t = t + (c1k * bu0 + c2k * bu1);
      io.wten[ow] = t;
    }
#pragma unroll
    for (int d = 0; d < 5; d++) { uw[d] = uw[d + 1]; vw[d] = vw[d + 1]; ww[d] = ww[d + 1]; }
    uw[5] = nu; vw[5] = nv; ww[5] = nw;
    fzu = hzu; fzv = hzv; fzw = hzw;
    divm = div0; bu0 = bu1;
  }
}

template <int TX, int TY, int KC>
static void mom_tiles_shape(const DGrid &g, const Vel &q, const float *uten1, const float *vten1,
                            const float *wten1, float *uten, float *vten, float *wten, const float *th3d,
                            const float *qv, const float *b8, const float *divx, const Diff6 &df,
                            cudaStream_t st, int which) {
  dim3 blk(TX, TY);
  const int kch = (g.nk + KC - 1) / KC, kchw = (g.nk - 1 + KC - 1) / KC;
  if (which & 1) {
    dim3 grid((g.ni + 1 + TX - 1) / TX, (g.nj + TY - 1) / TY, kch);
    ProfScope _ps("k_advu", st);
    k_mom_tile<TX, TY, KC, 2><<<grid, blk, 0, st>>>(g, q, divx, uten1, uten, nullptr, nullptr, nullptr, df);
  }
  if (which & 2) {
    dim3 grid((g.ni + TX - 1) / TX, (g.nj + 1 + TY - 1) / TY, kch);
    ProfScope _ps("k_advv", st);
    k_mom_tile<TX, TY, KC, 3><<<grid, blk, 0, st>>>(g, q, divx, vten1, vten, nullptr, nullptr, nullptr, df);
  }
  if (which & 4) {
    dim3 grid((g.ni + TX - 1) / TX, (g.nj + TY - 1) / TY, kchw);
    ProfScope _ps("k_advw", st);
    k_mom_tile<TX, TY, KC, 4><<<grid, blk, 0, st>>>(g, q, divx, wten1, wten, th3d, qv, b8, df);
  }
}

void launch_adv_momentum(const DGrid &g, const float *u, const float *v, const float *w,
                         const float *uten1, const float *vten1, const float *wten1,
                         float *uten, float *vten, float *wten, const float *th3d, const float *qv,
                         float *divx, cudaStream_t st, int64_t *nl, const Diff6 *diff, const float *b8,
                         int which) {
  // which: bit 0 u (advu), bit 1 v (advv), bit 2 w (advw)
  Vel q{u, v, w};
  if (!diff) {
    const MomIO io{uten1, vten1, wten1, uten, vten, wten, th3d, qv, b8};
    ProfScope _ps("k_mom", st);
    // launch shape 0: the levels that end first; the other shapes: their table's levels
    const long tiles = (long)((g.ni + 31) / 31) * ((g.nj + MOM_TY - 1) / (MOM_TY - 1));
    int kc = g.tile_mom > 0 ? kTileShapes[g.tile_mom][2] : tile_levels(tiles, g.nk, 2 * 148, 3, 4, MOM_KC);
    if (kc > MOM_KC) kc = MOM_KC;
    const size_t sm = (size_t)(kc + 2) * sizeof(MomLev);
    dim3 blk(32, MOM_TY), grid((g.ni + 31) / 31, (g.nj + MOM_TY - 1) / (MOM_TY - 1), (g.nk + kc - 1) / kc);
    switch (which) {
      case 1: k_mom<1><<<grid, blk, sm, st>>>(g, q, io, kc); break;
      case 2: k_mom<2><<<grid, blk, sm, st>>>(g, q, io, kc); break;
      case 4: k_mom<4><<<grid, blk, sm, st>>>(g, q, io, kc); break;
      default: k_mom<7><<<grid, blk, sm, st>>>(g, q, io, kc); break;
    }
    if (nl) *nl += 1;
    return;
  }
  const Diff6 df = *diff;
  {
    dim3 grid((g.ni + 2 + 127) / 128, g.nj + 2, g.nk);
    ProfScope _ps("k_mom_divx", st);
    k_mom_divx<<<grid, 128, 0, st>>>(g, q, divx);
  }
#define CM1G_MOM_SHAPE(n)                                                                                     \
  case n:                                                                                                     \
    mom_tiles_shape<kTileShapes[n][0], kTileShapes[n][1], kTileShapes[n][2]>(g, q, uten1, vten1, wten1, uten, \
                                                                             vten, wten, th3d, qv, b8, divx, df, st, \
                                                                             which);                                \
    break;
  switch (g.tile_mom) {
    CM1G_MOM_SHAPE(1)
    CM1G_MOM_SHAPE(2)
    CM1G_MOM_SHAPE(3)
    CM1G_MOM_SHAPE(4)
    default: CM1G_MOM_SHAPE(0)
  }
#undef CM1G_MOM_SHAPE
  if (nl) *nl += 1 + ((which & 1) != 0) + ((which & 2) != 0) + ((which & 4) != 0);
}

// ---------------------------------------------------------------------
// advs: adv.F:14-903 for one scalar.
//
// The fluxes use the small-step-averaged velocities rru/rrv/rrw as sound
// leaves them; getdivx's rho0/rf0 weighting (misclibs.F:251-276) and divx
// (misclibs.F:330-340) are applied on the fly.  `sadd` (the theta offset
// th0-300, solve2.F:1365-1372) is added to s when given.
// ---------------------------------------------------------------------
struct SAdv {
  const float *__restrict__ rru, *__restrict__ rrv, *__restrict__ rrw;  // averaged velocities
  const float *__restrict__ s;      // advected field (full halo)
  const float *__restrict__ s0;     // RK base value (pdef only)
  const float *__restrict__ thterm; // moist theta: thten -= div(u_avg)*thterm (solve2.F:1320-1329)
  int sadd;                         // add th0(k)-th0r to s (theta)
  Diff6 df{};                       // 6th-order diffusion (df.rho null: none)
};

// Tiled form of pass 2: a block owns TX x TY columns and marches upward;
// each level's dumx (with its +-2 halo in x) and dumy (+-2 in y) are staged
// in shared memory (double-buffered, one barrier per level; beyond the domain's
// edges from the points that the lateral bc copies there, pdef.F:102, 338),
// dumz comes from a per-column register window, and every read of a level is issued
// one level ahead.
template <int TX, int TY, int KC>
__global__ void __launch_bounds__(TX * TY) k_advs_pdef2_tile(DGrid g, SAdv a, const float *__restrict__ advx,
                                                             const float *__restrict__ advy, const float *__restrict__ advz,
                                                             const float *__restrict__ dumx, const float *__restrict__ dumy,
                                                             const float *__restrict__ dumz, const float *__restrict__ sten_in,
                                                             float *__restrict__ snew, const float *__restrict__ sbase,
                                                             float dt, int flush) {
  constexpr int NT = TX * TY;
  constexpr int XW = TX + 4, YH = TY + 4;
  constexpr int NSX = (XW * TY + NT - 1) / NT, NSY = (TX * YH + NT - 1) / NT;
  __shared__ float sx[2][TY * XW], sy[2][YH * TX];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
  const int i0 = 1 + (int)blockIdx.x * TX, j0 = 1 + (int)blockIdx.y * TY;
  const int i = i0 + tx, j = j0 + ty;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI, NJ = g.NJ;
  const bool active = (i <= ni && j <= nj);
  const int planeS = NI * NJ, planeU = (NI + 1) * NJ, planeV = NI * (NJ + 1);   // < 2^31 points (cm1g_init)
  const float smeps = g.smeps, rdt = 1.0f / dt;
  const float uh_i = active ? LDG(&g.uh[i - g.ib]) : 0.0f, vh_j = active ? LDG(&g.vh[j - g.jb]) : 0.0f;
  const int oc = active ? (i - g.ib) + NI * (j - g.jb) : 0;
  const int ocu = active ? (i - g.ib) + (NI + 1) * (j - g.jb) : 0;
  int xo[NSX], xs[NSX], yo[NSY], ys[NSY];   // staging: source offset in the plane (-1: none), slot
#pragma unroll
  for (int q = 0; q < NSX; q++) {
    const int t = tid + q * NT;
    xo[q] = -1; xs[q] = 0;
    if (t < XW * TY) {
      const int yy = t / XW, xx = t - yy * XW, ii = i0 - 2 + xx, jj = j0 + yy;
      if (ii <= ni + 2 && jj <= nj) { xo[q] = (bc_source(ii, ni, g.wbc, g.ebc) - g.ib) + NI * (jj - g.jb); xs[q] = t; }
    }
  }
#pragma unroll
  for (int q = 0; q < NSY; q++) {
    const int t = tid + q * NT;
    yo[q] = -1; ys[q] = 0;
    if (t < TX * YH) {
      const int yy = t / TX, xx = t - yy * TX, ii = i0 + xx, jj = j0 - 2 + yy;
      if (ii <= ni && jj <= nj + 2) { yo[q] = (ii - g.ib) + NI * (bc_source(jj, nj, g.sbc, g.nbc) - g.jb); ys[q] = t; }
    }
  }
  const int kc0 = 1 + (int)blockIdx.z * KC, kc1 = min(nk, kc0 + KC - 1);
  auto DZ = [&](int kk) { return (kk < 1 || kk > nk) ? 0.0f : LDG(&dumz[kk * planeS + oc]); };
  auto WR = [&](int kk) { return (kk <= 1 || kk >= nk + 1) ? 0.0f : LDG(&a.rrw[kk * planeS + oc]); };
  float zw[5];                                  // dumz(k-2 .. k+2)
#pragma unroll
  for (int d = 0; d < 5; d++) zw[d] = active ? DZ(kc0 - 2 + d) : 0.0f;
  float wlo = active ? WR(kc0) : 0.0f;          // raw averaged w through the bottom face

  float psx[NSX], psy[NSY], pax = 0.f, pay = 0.f, paz = 0.f, ps = 0.f, ps0 = 0.f, pt = 0.f, pb = 0.f;
  float pu0 = 0.f, pu1 = 0.f, pv0 = 0.f, pv1 = 0.f, pwhi = 0.f, pztop = 0.f;
  auto fetch = [&](int kf) {
#pragma unroll
    for (int q = 0; q < NSX; q++) psx[q] = (xo[q] >= 0) ? LDG(&dumx[kf * planeS + xo[q]]) : 0.0f;
#pragma unroll
    for (int q = 0; q < NSY; q++) psy[q] = (yo[q] >= 0) ? LDG(&dumy[kf * planeS + yo[q]]) : 0.0f;
    if (active) {
      const int o = kf * planeS + oc, ou = kf * planeU + ocu, ov = kf * planeV + oc;
      pax = LDG(&advx[o]); pay = LDG(&advy[o]); paz = LDG(&advz[o]);
      ps = LDG(&a.s[o]);
      if (a.sadd) ps = (LDG(&g.th0[kf]) - 300.0f) + ps;
      ps0 = LDG(&a.s0[o]); pt = sten_in[o]; pb = LDG(&sbase[o]);
      pu0 = LDG(&a.rru[ou]); pu1 = LDG(&a.rru[ou + 1]);
      pv0 = LDG(&a.rrv[ov]); pv1 = LDG(&a.rrv[ov + NI]);
      pwhi = WR(kf + 1);
      pztop = DZ(kf + 2);                       // top of the dumz window of level kf
    }
  };
  fetch(kc0);
  for (int k = kc0; k <= kc1; k++) {
    const int b = k & 1;
#pragma unroll
    for (int q = 0; q < NSX; q++) if (xo[q] >= 0) sx[b][xs[q]] = psx[q];
#pragma unroll
    for (int q = 0; q < NSY; q++) if (yo[q] >= 0) sy[b][ys[q]] = psy[q];
    const float ax0 = pax, ay0 = pay, az0 = paz, s = ps, s0 = ps0, t1 = pt, base = pb;
    const float u0r = pu0, u1r = pu1, v0r = pv0, v1r = pv1, whi = pwhi;
    if (k < kc1) fetch(k + 1);
    __syncthreads();
    if (active) {
      const float r0k = LDG(&g.rho0[k]), mhk = LDG(&g.mh[k]);
      const float fu0 = u0r * r0k, fu1 = u1r * r0k, fv0 = v0r * r0k, fv1 = v1r * r0k;
      const float fwlo = wlo * LDG(&g.rf0[k]), fwhi = whi * LDG(&g.rf0[k + 1]);
      float m; bool f;
      // z (pdefz): dum(0)=dum(nk+1)=0
      float az = az0;
      pdef_gather(zw[0], zw[1], zw[2], zw[3], zw[4], smeps, &m, &f);
      if (f) az = (zw[2] + m - r0k * s0) * rdt - s * (fwhi - fwlo) * g.rdz * mhk;
      // x (pdefx2)
      const float *px = &sx[b][ty * XW + tx];
      float ax = ax0;
      pdef_gather(px[0], px[1], px[2], px[3], px[4], smeps, &m, &f);
      if (f) ax = (px[2] + m - r0k * s0) * rdt - s * (fu1 - fu0) * g.rdx * uh_i;
      // y (pdefy2)
      const float *py = &sy[b][ty * TX + tx];
      float ay = ay0;
      pdef_gather(py[0], py[TX], py[2 * TX], py[3 * TX], py[4 * TX], smeps, &m, &f);
      if (f) ay = (py[2 * TX] + m - r0k * s0) * rdt - s * (fv1 - fv0) * g.rdy * vh_j;
      float div = ((fu1 - fu0) * g.rdx * uh_i + (fv1 - fv0) * g.rdy * vh_j) + (fwhi - fwlo) * g.rdz * mhk;
      if (fabsf(div) < g.smeps) div = 0.0f;
      const float ten = t1 + (((ax + ay) + az) + s * div) * LDG(&g.rr0[k]);
      float v = base + dt * ten;
      if (flush && fabsf(v) < g.smeps) v = 0.0f;
      snew[k * planeS + oc] = v;
#pragma unroll
      for (int d = 0; d < 4; d++) zw[d] = zw[d + 1];
      zw[4] = pztop;            // dumz(k+3), fetched with level k+1 above
      wlo = whi;
    }
  }
}

// ---------------------------------------------------------------------
// Tiled scalar advection (the production path of advs).
//
// A block owns TX x TY columns and marches upward through the levels.  At
// each level the advected field is staged with its 3-point lateral halo in
// shared memory; every x- and y-face flux is evaluated once (the WENO5 or
// 5th-order value of hadv_weno5/hadv_flx5) and shared by the two cells it
// separates; the vertical face flux of the level above is evaluated from a
// per-thread register window of the column and carried to the next level as
// its lower face.  Each cell therefore costs three face evaluations instead
// of six.  MODE_UPDATE writes snew = s0 + dt*ten (solve2.F:1419-1425,
// 1513-1520, 1951-1957); MODE_PDEF1 writes advx/advy/advz and the
// provisional masses of pdefx1/pdefy1/pdefz for the second pdef pass.
// ---------------------------------------------------------------------
enum { MODE_UPDATE = 0, MODE_PDEF1 = 1 };

struct STileOut {
  const float *sten_in;       // fixed tendency (thten1, qten, ptten)
  const float *sbase;         // RK base value (tha, qa, pta)
  float *snew;                // MODE_UPDATE output
  float *advx, *advy, *advz, *dumx, *dumy, *dumz;   // MODE_PDEF1 outputs
  TileExtras ex;              // learned face values / flux capture (update mode)
};

// The block has TY rows of cell threads and one more row of TX threads:
// the (TX+1)*TY x-faces and TX*(TY+1) y-faces of a level are spread at most
// one of each per thread, so the cell threads evaluate three faces (x, y and
// the z face above their cell) and the extra row two; staging
// sources, face addresses and the column offset are 32-bit in-plane offsets
// computed once per block; the raw averaged velocities of the faces are kept
// in shared memory for the divergence terms of the cell owners.  All
// arrays must have fewer than 2^31 points per horizontal plane.
template <int TX, int TY, int KC, int MODE, int WENO, int DIFF>
__global__ void __launch_bounds__(TX * (TY + 1), 3) k_advs_tile(DGrid g, SAdv a, STileOut out, int pdef, int pdefweno,
                                                       double weps, float dt, int flush) {
  constexpr int NT = TX * (TY + 1);                        // TY cell rows + the row of the extra faces
  constexpr int SW = TX + 6, SH = TY + 6, SP = SW + 1;     // staged plane, pitch SP
  constexpr int NST = (SW * SH + NT - 1) / NT;              // staging slots per thread
  constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);   // faces of one level
  __shared__ float ss[SH * SP];
  __shared__ float fx[NFX], ux[NFX], fy[NFY], vy[NFY];
  __shared__ float dfx[NFX], dfy[NFY];     // 6th-order diffusion fluxes (adv.F:356-395)
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
  const int i0 = 1 + (int)blockIdx.x * TX, j0 = 1 + (int)blockIdx.y * TY;
  const int i = i0 + tx, j = j0 + ty;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI, NJ = g.NJ;
  const bool active = (ty < TY && i <= ni && j <= nj);
  const bool doitw = (g.wbc == 2 && g.ibw), doite = (g.ebc == 2 && g.ibe);
  const bool doits = (g.sbc == 2 && g.ibs), doitn = (g.nbc == 2 && g.ibn);
  const int ie = ni + g.ngxy, je = nj + g.ngxy;
  const int planeS = NI * NJ, planeU = (NI + 1) * NJ, planeV = NI * (NJ + 1);   // < 2^31 points (cm1g_init)
  const float uh_i = active ? LDG(&g.uh[i - g.ib]) : 0.0f, vh_j = active ? LDG(&g.vh[j - g.jb]) : 0.0f;
  const int oc = active ? (i - g.ib) + NI * (j - g.jb) : 0;   // the column's in-plane offset

  int soff[NST], sidx[NST];     // staging: source offset (-1: outside the arrays), slot in ss (-1: none)
#pragma unroll
  for (int q = 0; q < NST; q++) {
    const int t = tid + q * NT;
    soff[q] = -1; sidx[q] = -1;
    if (t < SW * SH) {
      const int yy = t / SW, xx = t - yy * SW;
      const int ii = i0 - 3 + xx, jj = j0 - 3 + yy;
      sidx[q] = yy * SP + xx;
      if (ii <= ie && jj <= je) soff[q] = (ii - g.ib) + NI * (jj - g.jb);
    }
  }
  int fxo[2], fxs[2], fyo[2], fys[2];   // face offsets (-1: no face) and stencil starts in ss
  int fxl[2], fyl[2];                   // in-level index of the face in the learned-value arrays
  int fxr[2];                           // s-plane offset of the cell (i, j) right of an x-face
  using FS = FaceSlots<NT, NFX, NFY>;
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int f = FS::x(tid, q), fy_ = FS::y(tid, q);
    fxo[q] = -1; fxs[q] = 0; fyo[q] = -1; fys[q] = 0; fxl[q] = 0; fyl[q] = 0; fxr[q] = 0;
    if (f < NFX) {
      const int row = f / (TX + 1), col = f - row * (TX + 1);
      const int ii = i0 + col, jj = j0 + row;
      if (ii <= ni + 1 && jj <= nj) {
        fxo[q] = (ii - g.ib) + (NI + 1) * (jj - g.jb); fxs[q] = (row + 3) * SP + col;
        fxl[q] = (jj - 1) * (ni + 1) + (ii - 1);
        fxr[q] = (ii - g.ib) + NI * (jj - g.jb);
      }
    }
    if (fy_ < NFY) {
      const int row = fy_ / TX, col = fy_ - row * TX;
      const int ii = i0 + col, jj = j0 + row;
      if (ii <= ni && jj <= nj + 1) {
        fyo[q] = (ii - g.ib) + NI * (jj - g.jb); fys[q] = row * SP + col + 3;
        fyl[q] = (jj - 1) * ni + (ii - 1);
      }
    }
  }

  auto SV = [&](int kk) -> float {
    float v = LDG(&a.s[kk * planeS + oc]);
    if (a.sadd) v = (LDG(&g.th0[kk]) - 300.0f) + v;
    return v;
  };
  // averaged w of a w-level (zero at the bottom and top boundaries)
  auto WRAW = [&](int kk) -> float { return (kk <= 1 || kk >= nk + 1) ? 0.0f : LDG(&a.rrw[kk * planeS + oc]); };

  // register window of the column: wv[d+3] = s(k+1+d), d = -3..2 (for the top face of level k);
  // the block covers levels kc0..kc1 of its columns (blockIdx.z selects the chunk)
  const int kc0 = 1 + (int)blockIdx.z * KC, kc1 = min(nk, kc0 + KC - 1);
  float wv[6];
#pragma unroll
  for (int d = 0; d < 6; d++) {
    const int kk = kc0 - 2 + d;
    wv[d] = (active && kk >= 0 && kk <= nk + 1) ? SV(kk) : 0.0f;
  }
  float wlo = active ? WRAW(kc0) : 0.0f;       // raw averaged w through the bottom face of the level
  float fwlo = wlo * LDG(&g.rf0[kc0]);
  float fzlo = 0.0f;                            // flux through the bottom face of the level
  if (active && kc0 >= 2) {
    float w0[6];
#pragma unroll
    for (int d = 0; d < 6; d++) {
      const int kk = kc0 - 3 + d;
      w0[d] = (kk >= 0 && kk <= nk + 1) ? SV(kk) : 0.0f;
    }
    fzlo = zflux_win(g, w0, fwlo, kc0, WENO, pdefweno, weps);
  }

  // Every global read of a level (the staged plane, the face velocities, the
  // cell's inputs and the next top of the column window) is issued one level
  // ahead, so it is in flight while the previous level computes.  None of
  // these arrays is written by this kernel.
  float pst[NST], pru[2], prv[2], pwhi = 0.0f, pe0 = 0.0f, pe1 = 0.0f, pe2 = 0.0f, pwtop = 0.0f;
  auto fetch = [&](int kf) {
    const float *sk = a.s + kf * planeS;
#pragma unroll
    for (int q = 0; q < NST; q++) pst[q] = (soff[q] >= 0) ? LDG(&sk[soff[q]]) : 0.0f;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      pru[q] = (fxo[q] >= 0) ? LDG(&a.rru[kf * planeU + fxo[q]]) : 0.0f;
      prv[q] = (fyo[q] >= 0) ? LDG(&a.rrv[kf * planeV + fyo[q]]) : 0.0f;
    }
    if (active) {
      const int o = kf * planeS + oc;
      pwhi = WRAW(kf + 1);
      if (MODE == MODE_UPDATE) {
        pe0 = out.sten_in[o];
        pe1 = LDG(&out.sbase[o]);
        if (a.thterm) pe2 = LDG(&a.thterm[o]);
      } else {
        pe0 = LDG(&a.s0[o]);
      }
      pwtop = (kf + 3 <= nk + 1) ? SV(kf + 3) : 0.0f;   // top of the window of level kf
    }
  };
  fetch(kc0);

  for (int k = kc0; k <= kc1; k++) {
    const float r0k = LDG(&g.rho0[k]);
    const float th0m = a.sadd ? (LDG(&g.th0[k]) - 300.0f) : 0.0f;
    // ---- stage the level with its halo; take the raw face velocities
#pragma unroll
    for (int q = 0; q < NST; q++) {
      if (sidx[q] >= 0) {
        float v = pst[q];
        if (soff[q] >= 0 && a.sadd) v = th0m + v;
        ss[sidx[q]] = v;
      }
    }
    const float ru[2] = {pru[0], pru[1]}, rv[2] = {prv[0], prv[1]};
    const float whi = pwhi, e0 = pe0, e1 = pe1, e2 = pe2;
    if (k < kc1) fetch(k + 1);
    __syncthreads();
    // ---- face values: each x/y face once, each upper z face once per column
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int f = FS::x(tid, q), fy_ = FS::y(tid, q);
      if (fxo[q] >= 0) {
        const float *p = &ss[fxs[q]];
        const float r = ru[q] * r0k;
        float ph = __int_as_float(0x7fc00000);
        if (MODE == MODE_UPDATE && out.ex.phix) ph = out.ex.phix[(k - 1) * (ni + 1) * nj + fxl[q]];
        const float fl = (ph == ph) ? r * ph : hflux5(r, p[0], p[1], p[2], p[3], p[4], p[5], WENO, pdef, weps);
        fx[f] = fl;
        ux[f] = ru[q];
        if (DIFF) {   // face between s(i-1) and s(i): p[2], p[3]
          const int ro = k * planeS + fxr[q];                           // rho(i,j)
          const float fd = diff6_stencil(p[0], p[1], p[2], p[3], p[4], p[5]) * 0.5f *
                           (LDG(&a.df.rho[ro - 1]) + LDG(&a.df.rho[ro]));
          dfx[f] = diff6_limit(fd, p[3], p[2], a.df.mdiff);
        }
        if (MODE == MODE_UPDATE && out.ex.capfx) {
          out.ex.capfx[k * planeU + fxo[q]] = fl;
          out.ex.caprx[k * planeU + fxo[q]] = r;
        }
      }
      if (fyo[q] >= 0) {
        const float *p = &ss[fys[q]];
        const float r = rv[q] * r0k;
        float ph = __int_as_float(0x7fc00000);
        if (MODE == MODE_UPDATE && out.ex.phiy) ph = out.ex.phiy[(k - 1) * ni * (nj + 1) + fyl[q]];
        const float fl = (ph == ph) ? r * ph
                                    : hflux5(r, p[0], p[SP], p[2 * SP], p[3 * SP], p[4 * SP], p[5 * SP], WENO, pdef, weps);
        fy[fy_] = fl;
        vy[fy_] = rv[q];
        if (DIFF) {   // face between s(j-1) and s(j): p[2 SP], p[3 SP]
          const int ro = k * planeS + fyo[q];                           // rho(i,j)
          const float fd = diff6_stencil(p[0], p[SP], p[2 * SP], p[3 * SP], p[4 * SP], p[5 * SP]) * 0.5f *
                           (LDG(&a.df.rho[ro - NI]) + LDG(&a.df.rho[ro]));
          dfy[fy_] = diff6_limit(fd, p[3 * SP], p[2 * SP], a.df.mdiff);
        }
        if (MODE == MODE_UPDATE && out.ex.capfy) {
          out.ex.capfy[k * planeV + fyo[q]] = fl;
          out.ex.capry[k * planeV + fyo[q]] = r;
        }
      }
    }
    const float fwhi = whi * LDG(&g.rf0[k + 1]);
    float fzhi = 0.0f, sc = 0.0f;
    if (active) {
      sc = ss[(ty + 3) * SP + tx + 3];
      if (k + 1 <= nk) fzhi = zflux_win(g, wv, fwhi, k + 1, WENO, pdefweno, weps);
    }
    __syncthreads();
    if (active) {
      const int o = k * planeS + oc;
      const int xi = ty * (TX + 1) + tx, yi = ty * TX + tx;
      float fx0 = fx[xi], fxp = fx[xi + 1], fy0 = fy[yi], fyp = fy[yi + TX];
      const float u0r = ux[xi], u1r = ux[xi + 1], v0r = vy[yi], v1r = vy[yi + TX];
      const float fu0 = u0r * r0k, fu1 = u1r * r0k, fv0 = v0r * r0k, fv1 = v1r * r0k;
      // adv.F:212-268
      if (doitw && i == 1 && fu0 >= 0.0f) fx0 = fxp;
      if (doite && i == ni && fu1 <= 0.0f) fxp = fx0;
      if (doits && j == 1 && fv0 >= 0.0f) fy0 = fyp;
      if (doitn && j == nj && fv1 <= 0.0f) fyp = fy0;
      float advx = -(fxp - fx0) * g.rdx * uh_i;
      float advy = -(fyp - fy0) * g.rdy * vh_j;
      // adv.F:286-335
      if (doitw && i == 1 && fu0 >= 0.0f) advx = advx - sc * (fu1 - fu0) * g.rdx * uh_i;
      if (doite && i == ni && fu1 <= 0.0f) advx = advx - sc * (fu1 - fu0) * g.rdx * uh_i;
      if (doits && j == 1 && fv0 >= 0.0f) advy = advy - sc * (fv1 - fv0) * g.rdy * vh_j;
      if (doitn && j == nj && fv1 <= 0.0f) advy = advy - sc * (fv1 - fv0) * g.rdy * vh_j;
      if (DIFF) {   // adv.F:375-378, 397-400
        const float ri = LDG(&a.df.ri[o]);
        advx = advx + a.df.coef * (dfx[xi + 1] - dfx[xi]) * ri * r0k;
        advy = advy + a.df.coef * (dfy[yi + TX] - dfy[yi]) * ri * r0k;
      }
      const float mhk = LDG(&g.mh[k]);
      float advz;
      if (k == 1) advz = -fzhi * g.rdz * mhk;
      else if (k == nk) advz = +fzlo * g.rdz * mhk;
      else advz = -(fzhi - fzlo) * g.rdz * mhk;
      float div = ((fu1 - fu0) * g.rdx * uh_i + (fv1 - fv0) * g.rdy * vh_j) + (fwhi - fwlo) * g.rdz * mhk;
      if (fabsf(div) < g.smeps) div = 0.0f;
      if (MODE == MODE_UPDATE) {
        float ten = e0;
        if (a.thterm) {   // getdiv of the averaged velocities (misclibs.F:127-136)
          float rd = ((u1r - u0r) * g.rdx * uh_i + (v1r - v0r) * g.rdy * vh_j) + (whi - wlo) * g.rdz * mhk;
          if (fabsf(rd) < g.smeps) rd = 0.0f;
          ten = ten - rd * e2;
        }
        ten = ten + (((advx + advy) + advz) + sc * div) * LDG(&g.rr0[k]);
        float v = e1 + dt * ten;
        if (flush && fabsf(v) < g.smeps) v = 0.0f;
        out.snew[o] = v;
      } else {
        // pdefx1 / pdefy1 / pdefz provisional masses (pdef.F:35-102, 289-340, 478-496)
        out.advx[o] = advx; out.advy[o] = advy; out.advz[o] = advz;
        const float s0 = e0;
        float dx = r0k * s0 + dt * (advx + sc * (fu1 - fu0) * g.rdx * uh_i);
        if (doitw && i == 1 && fu0 >= 0.0f) dx = r0k * s0;
        if (doite && i == ni && fu1 <= 0.0f) dx = r0k * s0;
        float dy = r0k * s0 + dt * (advy + sc * (fv1 - fv0) * g.rdy * vh_j);
        if (doits && j == 1 && fv0 >= 0.0f) dy = r0k * s0;
        if (doitn && j == nj && fv1 <= 0.0f) dy = r0k * s0;
        out.dumx[o] = dx; out.dumy[o] = dy;
        out.dumz[o] = r0k * s0 + dt * (advz + sc * (fwhi - fwlo) * g.rdz * mhk);
      }
      // slide the column window and carry the upper face to the next level
#pragma unroll
      for (int d = 0; d < 5; d++) wv[d] = wv[d + 1];
      wv[5] = pwtop;            // s(k+4), the new top of the window for level k+1
      fzlo = fzhi;
      fwlo = fwhi;
      wlo = whi;
    }
    // no barrier here: the next level's staging writes ss, which nobody reads
    // after the second barrier, and fx/fy/ux/vy are rewritten only after the
    // next level's first barrier, which every thread reaches after this level.
  }
}

// One k_advs_tile launch: WENO and the 6th-order diffusion (a.df.rho set)
// select compile-time variants, so the plain pass carries no diffusion code.
template <int TX, int TY, int KC, int MODE>
static void advs_tile_launch(dim3 grid, dim3 blk, cudaStream_t st, int weno, const DGrid &g, const SAdv &a,
                             const STileOut &o, int pdef, int pdefweno, double weps, float dt, int flush) {
  if (a.df.rho) {
    if (weno) k_advs_tile<TX, TY, KC, MODE, 1, 1><<<grid, blk, 0, st>>>(g, a, o, pdef, pdefweno, weps, dt, flush);
    else k_advs_tile<TX, TY, KC, MODE, 0, 1><<<grid, blk, 0, st>>>(g, a, o, pdef, pdefweno, weps, dt, flush);
  } else {
    if (weno) k_advs_tile<TX, TY, KC, MODE, 1, 0><<<grid, blk, 0, st>>>(g, a, o, pdef, pdefweno, weps, dt, flush);
    else k_advs_tile<TX, TY, KC, MODE, 0, 0><<<grid, blk, 0, st>>>(g, a, o, pdef, pdefweno, weps, dt, flush);
  }
}

// Production scalar pass (MODE_UPDATE, or the pdef two-pass form) with the
// tile shape TX x TY x KC.
template <int TX, int TY, int KC>
static void advs_tiled_shape(const DGrid &g, const SAdv &a, STileOut o, int weno, int pdef, int pdefweno,
                             double weps, float dt, int flush, float *scratch, cudaStream_t st, int64_t *nl) {
  // k_advs_tile: TY cell rows and the row of the tile's extra faces; pass 2
  // (no face evaluations) takes TY + 1 cell rows per block
  dim3 blk(TX, TY + 1), grid((g.ni + TX - 1) / TX, (g.nj + TY - 1) / TY, (g.nk + KC - 1) / KC);
  dim3 grid2((g.ni + TX - 1) / TX, (g.nj + TY) / (TY + 1), (g.nk + KC - 1) / KC);
  if (!pdef) {
    ProfScope _ps("k_advs_tile", st);
    advs_tile_launch<TX, TY, KC, MODE_UPDATE>(grid, blk, st, weno, g, a, o, 0, pdefweno, weps, dt, flush);
    if (nl) *nl += 1;
    return;
  }
  long n = nS(g);
  o.advx = scratch; o.advy = scratch + n; o.advz = scratch + 2 * n;
  o.dumx = scratch + 3 * n; o.dumy = scratch + 4 * n; o.dumz = scratch + 5 * n;
  {
    ProfScope _ps("k_advs_tile_pdef1", st);
    advs_tile_launch<TX, TY, KC, MODE_PDEF1>(grid, blk, st, weno, g, a, o, 1, pdefweno, weps, dt, flush);
  }
  {
    ProfScope _ps("k_advs_pdef2", st);
    k_advs_pdef2_tile<TX, TY + 1, KC><<<grid2, blk, 0, st>>>(g, a, o.advx, o.advy, o.advz, o.dumx, o.dumy, o.dumz,
                                                       o.sten_in, o.snew, o.sbase, dt, flush);
  }
  if (nl) *nl += 2;
}

void launch_advs_tiled(const DGrid &g, const float *rru, const float *rrv, const float *rrw, const float *s,
                       const float *s0, int sadd, const float *ten1, const float *thterm, float *snew, int weno,
                       int pdef, int pdefweno, double weps, float dt, int flush, float *scratch, cudaStream_t st,
                       int64_t *nl, const TileExtras *ex, const Diff6 *diff) {
  SAdv a{rru, rrv, rrw, s, s0, thterm, sadd};
  if (diff) a.df = *diff;
  STileOut o{};
  o.sten_in = ten1; o.sbase = s0; o.snew = snew;
  if (ex) o.ex = *ex;
  static_assert(kNumTileShapes == 5, "one case per tile shape");
#define CM1G_ADVS_SHAPE(n)                                                                                      \
  case n:                                                                                                      \
    advs_tiled_shape<kScalShapes[n][0], kScalShapes[n][1], kScalShapes[n][2]>(g, a, o, weno, pdef, pdefweno,    \
                                                                              weps, dt, flush, scratch, st, nl); \
    break;
  switch (g.tile_adv) {
    CM1G_ADVS_SHAPE(1)
    CM1G_ADVS_SHAPE(2)
    CM1G_ADVS_SHAPE(3)
    CM1G_ADVS_SHAPE(4)
    default: CM1G_ADVS_SHAPE(0)
  }
#undef CM1G_ADVS_SHAPE
}

}  // namespace cm1g
