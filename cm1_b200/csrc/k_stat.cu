// k_stat.cu -- the statistics package (statpack.F:10-658) on the device.
//
// statpack evaluates a fixed list of domain statistics: extrema of fields
// and of derived quantities (maxmin / maxmin2d, maxmin.F:5-228), the CFL
// number (calccfl, misclibs.F:2584-2718), vertical vorticity maxima
// (vertvort, misclibs.F:2424-2576), cloud top and base (cloud,
// misclibs.F:2344-2416) and FP64 budgets (calcmass, totmois, totq, calcener,
// calcmoe, tmf; misclibs.F:3134-3636).  Every one of them is a reduction over
// the points of one model level followed by a reduction over the levels, so
// the device form is three launches:
//
//   k_stat_flow    the statistics of the flow and of water vapour (velocities,
//                  pressure, theta, qv, divergence, humidity, wind speed, CFL,
//                  mass, moisture, momentum and energy budgets), which share
//                  their fields: one block per (level, chunk of rows) reads
//                  each field once and evaluates every expression that is on;
//   k_stat_levels  the remaining quantities (condensate, tracers, single
//                  levels), each of which reads fields of its own: one block
//                  per (quantity, level, chunk of points);
//   k_stat_finish  one block per rstat entry: it combines the chunks and
//                  levels with the reference's tie rule (the value of the
//                  strict comparisons from the same initial values, the
//                  first level holding it) and FP64 sums, and writes rstat
//                  in statpack's order.
//
// Bound by instruction issue (binary64 budgets and conversions, pow and exp):
// both passes issue in 60 % of the cycles, at 14 and 19 % of the DRAM peak.
// 256x256x80 with five tracers, 87 entries: 0.277 ms a call (flow 0.155,
// levels 0.076, finish 0.010) against 0.651 with one block per quantity, level
// and chunk for everything.
//
// The host copies rstat back with one small device-to-host copy.  Point
// expressions keep the reference's operand order and kinds (binary32 where
// the Fortran is real, binary64 where it declares double precision); the
// library is compiled with --fmad=false.
#include <algorithm>
#include "cm1g_common.cuh"
#include "k_stat.cuh"

namespace cm1g {

// rslf (cm1libs.F:16-62): saturation mixing ratio over liquid
__device__ __forceinline__ float st_rslf(float p, float t, const StatConsts &s) {
  if (s.ptype == 4) return 380.00f * expf(17.2693882f - 4097.8531f / (t - 35.86f)) / p;
  float esl = 611.2f * expf(17.67f * (t - 273.15f) / (t - 29.65f));
  esl = fminf(esl, p * 0.5f);
  return s.eps * esl / (p - esl);
}

// value of a max/min quantity of k_stat_levels at (i, j, k)
template <int KIND>
__device__ __forceinline__ float st_value(const DGrid &g, const StatJob &jb, const StatFields &f, const StatConsts &s,
                                          const float *field, int i, int j, int k) {
  if (KIND == SK_FIELD) return LDG(&field[iS(g, i, j, k)]);
  if (KIND == SK_PRATE) return f.prate ? LDG(&f.prate[i2(g, i, j)]) : 0.0f;
  if (KIND == SK_WLEV) {  // statpack.F:180-188; jb.k0 = nkm
    const long o = iS(g, i, j, jb.k0);
    return jb.r1 * LDG(&f.wa[o]) + jb.r2 * LDG(&f.wa[o + (long)g.NI * g.NJ]);
  }
  if (KIND == SK_PSFC) {  // statpack.F:425-430
    const long o = iS(g, i, j, 1), pl = (long)g.NI * g.NJ;
    return (s.cgs1 * LDG(&f.prs[o]) + s.cgs2 * LDG(&f.prs[o + pl])) + s.cgs3 * LDG(&f.prs[o + 2 * pl]);
  }
  if (KIND == SK_VORT) {  // vertvort (misclibs.F:2497-2505), jb.k0 = the level
    const int kk = jb.k0;
    const float dv = LDG(&f.va[iV(g, i, j, kk)]) - LDG(&f.va[iV(g, i - 1, j, kk)]);
    const float du = LDG(&f.ua[iU(g, i, j, kk)]) - LDG(&f.ua[iU(g, i, j - 1, kk)]);
    return dv * g.rdx * LDG(&g.uf[i - g.ib]) - du * g.rdy * LDG(&g.vf[j - g.jb]);
  }
  // SK_CLOUD (statpack.F:406-418): sum of the cloud species
  const long o = iS(g, i, j, k);
  float q = 0.0f;
  for (int n = 0; n < s.numq; n++)
    if (s.cloudmask & (1u << n)) q = q + LDG(&f.qa[(long)n * f.qstride + o]);
  return q;
}

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

static const int ST_NT = 256;                 // threads of a block
static const int ST_NW = ST_NT / 32;
static const int ST_CHUNK = 4096;             // points of one block at most

// Chunks of a level: at most ST_CHUNK points, and on small grids enough
// chunks for four blocks on each of the 148 SMs over all levels (chunks of at
// least two points per thread).
int stat_chunks(int npl, int nlev) {
  if (npl <= 0) return 1;
  const int big = (npl + ST_CHUNK - 1) / ST_CHUNK, fill = (4 * 148 + nlev - 1) / nlev;
  const int most = (npl + 2 * ST_NT - 1) / (2 * ST_NT);
  return big > fill ? big : fill < most ? fill : most;
}

// slots of k_stat_flow's maxima and minima, and of its FP64 sums
enum { FM_U = 0, FM_V, FM_W, FM_PPI, FM_THA, FM_QV, FM_PP, FM_DIV, FM_RH, FM_THE, FM_WSP, FM_CFL, FM_N };
enum { FS_MASS = 0, FS_TMOIS, FS_QMAS, FS_TMF, FS_MOE, FS_ENER, FS_N };
constexpr int FS_ACC = 12;
// a sum job's first component in the accumulators (tmf has 2, moe 3, ener 4)
__device__ __forceinline__ int fs_first(int q) { return q <= FS_TMF ? q : q == FS_MOE ? 5 : q == FS_ENER ? 8 : FS_ACC; }

// jobs of k_stat_flow (-1: off) and the levels of the theta_e job
struct StatFlow {
  int m[FM_N], s[FS_N], the_nlev;
};

// grid: x = chunk of rows, y = level (nk+1: w only).  wpr of the block's warps (1, 2,
// 4 or 8) share a row, so that few long rows occupy all of them.  SUMS: 2 with the
// momentum or energy budgets, 1 with others, 0 with none; EXT: with extrema.  The
// registers of those left out hold one or two more blocks an SM.  Quantities that are
// off cost their branch only; PLAIN (most are on, a row a warp) goes without the
// branches.  256x256x80: w alone 42 us (66 with everything always formed and a row
// always a warp's), dry mass alone 26 (70), momentum alone 68 (122), everything 154
// (158); 1100x960x20: w and the Courant number 302 us a call (686), everything 586
// (875).
template <int SUMS, bool EXT, bool PLAIN>
__global__ void __launch_bounds__(ST_NT, 6 - SUMS - EXT) k_stat_flow(DGrid g, StatFields f, StatConsts s, StatFlow F, StatLev *lev,
                                                            int maxlev, int nch, int wpr) {
  __shared__ float red[2 * FM_N][ST_NW];
  __shared__ double rsum[FS_ACC][ST_NW];
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  const int ni = g.ni, nj = g.nj, nk = g.nk, k = 1 + (int)blockIdx.y;
  const int rpc = (nj + 1 + nch - 1) / nch, j0 = 1 + (int)blockIdx.x * rpc, j1 = min(nj + 1, j0 + rpc - 1);
  const int pl = g.NI * g.NJ, NI = g.NI;      // < 2^31 points (cm1g_init)
  const bool top = k == nk + 1;
  const bool the = F.m[FM_THE] >= 0 && k <= F.the_nlev, rhs = F.m[FM_RH] >= 0 || the;
  const bool moe = SUMS == 2 && F.s[FS_MOE] >= 0, ener = SUMS == 2 && F.s[FS_ENER] >= 0, wsp = PLAIN || F.m[FM_WSP] >= 0;
  const bool liquid = s.imoist && s.nql1 >= 0;
  float mx[FM_N], mn[FM_N];
  double acc[FS_ACC];
#pragma unroll
  for (int q = 0; q < FM_N; q++) { mx[q] = -1.0e30f; mn[q] = 1.0e30f; }
#pragma unroll
  for (int q = 0; q < FS_ACC; q++) acc[q] = 0.0;
  auto put = [&](int q, float v) { if (EXT) { mx[q] = fmaxf(mx[q], v); mn[q] = fminf(mn[q], v); } };

  const int kk = min(k, nk);
  const float th0 = LDG(&g.th0[kk]), pi0 = LDG(&g.pi0[kk]), mh = LDG(&g.mh[kk]), rmh = LDG(&g.rmh[kk]);
  const float r0 = LDG(&g.rho0[kk]), r0p = LDG(&g.rho0[kk + 1]), r0m = LDG(&g.rho0[kk - 1]), zh = s.zh[kk];
  const float pbase = F.m[FM_PP] >= 0 ? s.p00 * powf(pi0, s.cpdrd) : 0.0f;   // statpack.F:236-242
  if (PLAIN) wpr = 1;
  const int rows = ST_NW / wpr, i0 = 1 + 32 * (w & (wpr - 1)) + lane;      // the block's rows at a time; first point
  for (int j = j0 + w / wpr; j <= j1; j += rows) {
    const float vh = LDG(&g.vh[j - g.jb]), rvh = LDG(&g.rvh[j - g.jb]);
    const int orow = k * pl + NI * (j - g.jb) - g.ib;
    const float *ur = f.ua ? f.ua + (long)k * (NI + 1) * g.NJ + (long)(NI + 1) * (j - g.jb) - g.ib : nullptr;
    const float *vr = f.va ? f.va + (long)k * NI * (g.NJ + 1) + (long)NI * (j - g.jb) - g.ib : nullptr;
    for (int i = i0; i <= ni + 1; i += 32 * wpr) {
      if (top) {
        if (f.wa && i <= ni && j <= nj) put(FM_W, LDG(&f.wa[orow + i]));
        continue;
      }
      if (j > nj) {                    // v has one row more, u one column
        if (vr && i <= ni) put(FM_V, LDG(&vr[i]));
        continue;
      }
      const float u1 = ur ? LDG(&ur[i]) : 0.0f;
      put(FM_U, u1);
      if (i > ni) continue;
      const int o = orow + i;
      const float uh = LDG(&g.uh[i - g.ib]), ruh = LDG(&g.ruh[i - g.ib]);
      const float u2 = ur ? LDG(&ur[i + 1]) : 0.0f, v1 = vr ? LDG(&vr[i]) : 0.0f, v2 = vr ? LDG(&vr[i + NI]) : 0.0f;
      const float w1 = f.wa ? LDG(&f.wa[o]) : 0.0f, w2 = f.wa ? LDG(&f.wa[o + pl]) : 0.0f;
      const float ppi = f.ppi ? LDG(&f.ppi[o]) : 0.0f, tha = f.tha ? LDG(&f.tha[o]) : 0.0f;
      const float prs = f.prs ? LDG(&f.prs[o]) : 0.0f, rho = f.rho ? LDG(&f.rho[o]) : 0.0f;
      float qv = 0.0f, ql = 0.0f;
      if (s.imoist && f.qa) {
        qv = LDG(&f.qa[(long)s.nqv * f.qstride + o]);
        for (int n = s.nql1; n >= 0 && n <= s.nql2; n++) ql = ql + LDG(&f.qa[(long)n * f.qstride + o]);
      }
      const float ua = 0.0f + 0.5f * (u1 + u2), va = 0.0f + 0.5f * (v1 + v2), tx = (th0 + tha) * (pi0 + ppi);
      if (EXT) {
        put(FM_V, v1);
        put(FM_W, w1);
        put(FM_PPI, ppi);
        put(FM_THA, tha);
        put(FM_QV, qv);
        put(FM_PP, prs - pbase);
        if (F.m[FM_DIV] >= 0) {          // statpack.F:297-309 (axisymm = 0)
          const float ta = 0.5f * ((r0 + r0) * u2 - (r0 + r0) * u1) * g.rdx * uh;
          const float tb = 0.5f * ((r0 + r0) * v2 - (r0 + r0) * v1) * g.rdy * vh;
          const float tc = 0.5f * ((r0 + r0p) * w2 - (r0 + r0m) * w1) * g.rdz * mh;
          put(FM_DIV, (ta + tb) + tc);
        }
        if (rhs) {                       // statpack.F:364-371; calcthe (misclibs.F:2300-2336), cpm = cp, l0 = 2.555e6
          const float qvs = st_rslf(prs, tx, s);
          const float rh = qv * (1.0f + qvs * s.reps) / (qvs * (1.0f + qv * s.reps));
          put(FM_RH, rh);
          if (the) {
            const float cpm = s.cp;
            put(FM_THE, tx * powf(s.p00 * (1.0f + qv * s.reps) / prs, s.rd / cpm) * powf(rh, -(qv * s.rv / cpm)) *
                            expf(2.555e6f * qv / (cpm * tx)));
          }
        }
        if (wsp) put(FM_WSP, sqrtf(ua * ua + va * va));   // statpack.F:437-441 (umove = vmove = 0)
        if (F.m[FM_CFL] >= 0) {          // calccfl (misclibs.F:2618-2665)
          const float cu = (u1 + u2) * s.dtdx * uh, cv = (v1 + v2) * s.dtdy * vh, cw = (w1 + w2) * s.dtdz * mh;
          float c;
          if (s.nx > 1 && s.ny > 1) c = sqrtf((cu * cu + cv * cv) + cw * cw);
          else if (s.nx > 1) c = sqrtf(cu * cu + cw * cw);
          else c = sqrtf(cv * cv + cw * cw);
          put(FM_CFL, c);
        }
      }
      if (!SUMS) continue;
      // ---- FP64 budgets, in the reference's operand kinds
      if (F.s[FS_MASS] >= 0) acc[0] = acc[0] + (double)(rho * ruh * rvh * rmh);                          // misclibs.F:3160-3166
      if (F.s[FS_TMOIS] >= 0) acc[1] = acc[1] + (double)(rho * ((qv + ql) + 0.0f) * ruh * rvh * rmh);    // :3224-3230, qi = 0
      if (F.s[FS_QMAS] >= 0) acc[2] = acc[2] + (double)(rho * qv * ruh * rvh * rmh);                     // :3297-3303
      if (F.s[FS_TMF] >= 0) {          // :3588-3596: mf is double precision, formed in binary32
        const double mf = (double)(rho * 0.5f * (w1 + w2) * ruh * rvh);
        acc[3] = acc[3] + fmax(mf, 0.0);
        acc[4] = acc[4] + fmin(mf, 0.0);
      }
      if (moe || ener) {
        const double qtot = (double)((qv + ql) + 0.0f), tem = (double)(ruh * rvh * rmh);
        const double rt = (double)rho * tem, rq = rt * (1.0 + qtot);
        // the reference's terms with a factor 0 (vr, qi) are added to a factor of the
        // others: zero, or not a number where a value in them is not finite
        const float wm = __fmaf_rn(0.0f, ql * rho, 0.5f * (w1 + w2));
        if (moe) {                     // calcmoe (misclibs.F:3488-3502), umove = vmove = 0
          acc[5] = acc[5] + rq * (double)ua;
          acc[6] = acc[6] + rq * (double)va;
          acc[7] = acc[7] + rq * (double)wm;
        }
        if (ener) {                    // calcener (misclibs.F:3374-3393), umove = vmove = 0
          const float ke = __fmaf_rn(0.0f, wm, (0.5f * (u1 * u1 + u2 * u2) + 0.5f * (v1 * v1 + v2 * v2)) + 0.5f * (w1 * w1 + w2 * w2));
          acc[8] = acc[8] + rq * 0.5 * (double)ke;
          const double tmp = (double)tx;
          acc[9] = acc[9] + rt * (double)(s.cv + s.cvv * qv) * tmp;
          acc[10] = acc[10] + rq * (double)s.g * (double)zh;
          const float qz = __fmaf_rn(0.0f, rho, __fmaf_rn(0.0f, tx, ql));
          acc[11] = acc[11] + (liquid ? rt * (double)qz * ((double)s.cpl * tmp - (double)s.lv1) : (double)qz);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < (EXT ? FM_N : 0); q++) {
    if (F.m[q] < 0) continue;
    const float a = warp_max(mx[q]), b = warp_min(mn[q]);
    if (lane == 0) { red[2 * q][w] = a; red[2 * q + 1][w] = b; }
  }
#pragma unroll
  for (int q = 0; q < (SUMS == 2 ? FS_ACC : SUMS ? 5 : 0); q++) {
    const int job = q < 3 ? q : q < 5 ? FS_TMF : q < 8 ? FS_MOE : FS_ENER;   // its sum (fs_first)
    if (!PLAIN && F.s[job] < 0) continue;
    const double a = warp_sum(acc[q]);
    if (lane == 0) rsum[q][w] = a;
  }
  __syncthreads();
  auto rec = [&](int job) -> StatLev & { return lev[((long)job * maxlev + (k - 1)) * nch + blockIdx.x]; };
  const int t = (int)threadIdx.x;
  if (EXT && t < FM_N && F.m[t] >= 0 && !(top && t != FM_W) && !(t == FM_THE && !the)) {
    float a = red[2 * t][0], b = red[2 * t + 1][0];
    for (int q = 1; q < ST_NW; q++) { a = fmaxf(a, red[2 * t][q]); b = fminf(b, red[2 * t + 1][q]); }
    rec(F.m[t]).vmax = a;
    rec(F.m[t]).vmin = b;
  }
  if (SUMS && t >= 32 && t < 32 + FS_N && F.s[t - 32] >= 0 && !top) {
    const int q = t - 32;
    for (int c = 0; c < fs_first(q + 1) - fs_first(q); c++) {
      double a = 0.0;
      for (int m = 0; m < ST_NW; m++) a = a + rsum[fs_first(q) + c][m];
      rec(F.s[q]).s[c] = a;
    }
  }
}

// One chunk of one level of one quantity, its kind a constant so that the
// unrolled point loop issues its loads ahead of their use.
template <int KIND>
__device__ __forceinline__ void st_chunk(const DGrid &g, const StatJob &jb, const StatFields &f, const StatConsts &s,
                                         int k, int t0, int t1, int ni, StatLev *out, double (*red)[ST_NW]) {
  float vmax = -1.0e30f, vmin = 1.0e30f;
  double acc = 0.0;
  const float *field = nullptr;
  if (KIND == SK_FIELD || KIND == SK_QMAS)
    field = (KIND == SK_QMAS || jb.src == SF_Q) ? f.qa + (long)jb.qn * f.qstride
            : jb.src == SF_PT ? f.pta + (long)jb.qn * f.qstride : f.prs;
  // (ii, jj): offsets of point t in the level's i-j range, advanced by
  // ST_NT points (dj rows and di points) per step without a division
  const int dj = ST_NT / ni, di = ST_NT - dj * ni;
  const int tt = t0 + (int)threadIdx.x;
  int jj = tt / ni, ii = tt - jj * ni;
#pragma unroll 8
  for (int t = tt; t < t1; t += ST_NT) {
    const int i = jb.i0 + ii, j = jb.j0 + jj;
    ii += di; jj += dj;
    if (ii >= ni) { ii -= ni; jj++; }
    if (KIND == SK_QMAS) {   // totq (misclibs.F:3297-3303)
      const long o = iS(g, i, j, k);
      acc = acc + (double)(LDG(&f.rho[o]) * LDG(&field[o]) * LDG(&g.ruh[i - g.ib]) * LDG(&g.rvh[j - g.jb]) * LDG(&g.rmh[k]));
    } else {
      const float v = st_value<KIND>(g, jb, f, s, field, i, j, k);
      vmax = fmaxf(vmax, v);
      vmin = fminf(vmin, v);
    }
  }
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  if (KIND == SK_QMAS) {
    acc = warp_sum(acc);
    if (lane == 0) red[0][w] = acc;
  } else {
    vmax = warp_max(vmax);
    vmin = warp_min(vmin);
    if (lane == 0) { red[0][w] = (double)vmax; red[1][w] = (double)vmin; }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = red[0][0], b = red[1][0];
    for (int q = 1; q < ST_NW; q++) {
      if (KIND == SK_QMAS) a = a + red[0][q];
      else { a = fmax(a, red[0][q]); b = fmin(b, red[1][q]); }
    }
    if (KIND == SK_QMAS) out->s[0] = a;
    else { out->vmax = (float)a; out->vmin = (float)b; }
  }
}

// grid: x = chunk of a level, y = level of a job: R.first[q] is the first y of
// the list's job q
__global__ void __launch_bounds__(ST_NT) k_stat_levels(DGrid g, StatFields f, StatConsts s, const StatJob *jobs,
                                                       StatRest R, StatLev *lev, int maxlev, int nch) {
  __shared__ double red[2][ST_NW];
  int q = 0;
  while (q + 1 < R.n && (int)blockIdx.y >= R.first[q + 1]) q++;
  const int jx = R.job[q], kl = (int)blockIdx.y - R.first[q];
  const StatJob jb = jobs[jx];
  const int ni = jb.ie - jb.i0 + 1, nj = jb.je - jb.j0 + 1;
  const int npl = (ni > 0 && nj > 0) ? ni * nj : 0;
  const int len = (npl + nch - 1) / nch, t0 = (int)blockIdx.x * len, npt = min(npl, t0 + len);   // an empty chunk writes the neutral record
  const int k = jb.klo + kl;
  StatLev *out = lev + ((long)jx * maxlev + kl) * nch + blockIdx.x;
  switch (jb.kind) {
    case SK_FIELD: st_chunk<SK_FIELD>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    case SK_PRATE: st_chunk<SK_PRATE>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    case SK_WLEV:  st_chunk<SK_WLEV>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    case SK_PSFC:  st_chunk<SK_PSFC>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    case SK_VORT:  st_chunk<SK_VORT>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    case SK_CLOUD: st_chunk<SK_CLOUD>(g, jb, f, s, k, t0, npt, ni, out, red); break;
    default:       st_chunk<SK_QMAS>(g, jb, f, s, k, t0, npt, ni, out, red); break;
  }
}

// Block reductions over the (level, chunk) records of a job: the max/min with
// the first level that holds it, and the sums of one component (the warps'
// sums added in order).
static const int SF_NT = 128, SF_NW = SF_NT / 32;

__device__ __forceinline__ void warp_best(float &v, int &lv, bool is_max) {
  for (int o = 16; o > 0; o >>= 1) {
    const float v2 = __shfl_down_sync(0xffffffffu, v, o);
    const int l2 = __shfl_down_sync(0xffffffffu, lv, o);
    if (is_max ? (v2 > v || (v2 == v && l2 < lv)) : (v2 < v || (v2 == v && l2 < lv))) { v = v2; lv = l2; }
  }
}
struct FinShared { float v[SF_NW]; int l[SF_NW]; double d[SF_NW]; };
__device__ __forceinline__ void block_best(float &v, int &lv, bool is_max, FinShared &S) {
  warp_best(v, lv, is_max);
  if ((threadIdx.x & 31) == 0) { S.v[threadIdx.x >> 5] = v; S.l[threadIdx.x >> 5] = lv; }
  __syncthreads();
  v = S.v[0]; lv = S.l[0];
  for (int q = 1; q < SF_NW; q++)
    if (is_max ? (S.v[q] > v || (S.v[q] == v && S.l[q] < lv)) : (S.v[q] < v || (S.v[q] == v && S.l[q] < lv))) { v = S.v[q]; lv = S.l[q]; }
}
__device__ __forceinline__ double block_total(double t, FinShared &S) {
  t = warp_sum(t);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) S.d[threadIdx.x >> 5] = t;
  __syncthreads();
  t = S.d[0];
  for (int q = 1; q < SF_NW; q++) t = t + S.d[q];
  return t;
}

// The output program: one block per rstat entry, statpack's order.
__global__ void __launch_bounds__(SF_NT) k_stat_finish(DGrid g, StatConsts s, const StatJob *jobs, const StatLev *lev, int maxlev, int nch,
                              const StatOp *ops, int nops, float *rstat) {
  __shared__ FinShared S;
  const int p = (int)blockIdx.x, lane = (int)threadIdx.x;
  const StatOp op = ops[p];
  const int jx = op.job >= 0 ? op.job : 0;
  const StatJob jb = jobs[jx];
  const StatLev *L = lev + (long)jx * maxlev * nch;
  const int nrec = jb.nlev * nch;
  float r = 0.0f;
  switch (op.op) {
    case SO_MAX: case SO_ZF_KMAX: case SO_ZH_KMAX: case SO_CFL: {
      // maxmin.F:62-75: strict comparison from -1e30 in level order, level 1
      // if none; calccfl: cfl(k) from -1, fmax from -99999999
      float v = -1.0e30f; int lv = 0x7fffffff;
      for (int q = lane; q < nrec; q += SF_NT) {
        const float x = L[q].vmax;
        if (x > v) { v = x; lv = q / nch; }
      }
      block_best(v, lv, true, S);
      if (op.op == SO_MAX) r = v;
      else if (op.op == SO_CFL) r = fmaxf(-99999999.0f, v > -1.0f ? v : -1.0f);
      else {
        const int kmax = (lv == 0x7fffffff) ? 1 : jb.klo + lv;
        r = op.op == SO_ZF_KMAX ? s.zf[kmax] : s.zh[kmax];
      }
      break;
    }
    case SO_MIN: case SO_ZF_KMIN: case SO_ZH_KMIN: {
      float v = 1.0e30f; int lv = 0x7fffffff;
      for (int q = lane; q < nrec; q += SF_NT) {
        const float x = L[q].vmin;
        if (x < v) { v = x; lv = q / nch; }
      }
      block_best(v, lv, false, S);
      if (op.op == SO_MIN) r = v;
      else {
        const int kmin = (lv == 0x7fffffff) ? 1 : jb.klo + lv;
        r = op.op == SO_ZF_KMIN ? s.zf[kmin] : s.zh[kmin];
      }
      break;
    }
    case SO_LEVMAX: case SO_VORT: {   // maxmin2d of one level; vertvort: max(-9999999, ...)
      const StatLev *Lk = L + (long)(op.k - jb.klo) * nch;
      if (op.op == SO_VORT) Lk = L;
      float v = -1.0e30f; int lv = 0x7fffffff;
      for (int q = lane; q < nch; q += SF_NT) if (Lk[q].vmax > v) { v = Lk[q].vmax; lv = q; }
      block_best(v, lv, true, S);
      r = op.op == SO_VORT ? fmaxf(-9999999.0f, v) : v;
      break;
    }
    case SO_LEVMIN: {
      const StatLev *Lk = L + (long)(op.k - jb.klo) * nch;
      float v = 1.0e30f; int lv = 0x7fffffff;
      for (int q = lane; q < nch; q += SF_NT) if (Lk[q].vmin < v) { v = Lk[q].vmin; lv = q; }
      block_best(v, lv, false, S);
      r = v;
      break;
    }
    case SO_QCTOP: case SO_QCBOT: {  // cloud (misclibs.F:2364-2400), clwsat = 1e-6
      float top = 0.0f, bot = s.maxz;
      for (int q = lane; q < nrec; q += SF_NT) {
        const bool cl = L[q].vmax >= 1.e-6f;
        const float z = s.zh[jb.klo + q / nch];
        top = fmaxf(top, cl ? z : 0.0f);
        bot = fminf(bot, cl ? z : s.maxz);
      }
      int lt = 0, lb = 0;
      block_best(top, lt, true, S);
      __syncthreads();
      block_best(bot, lb, false, S);
      if (bot == s.maxz) bot = 0.0f;
      r = op.op == SO_QCTOP ? top : bot;
      break;
    }
    case SO_SUM: {  // the levels' sums, then the volume factor of the budget
      double t = 0.0;
      for (int q = lane; q < nrec; q += SF_NT) t = t + L[q].s[op.k];
      t = block_total(t, S);
      if (op.arg == 1) t = t * (double)(g.dx * g.dy * g.dz);
      else if (op.arg == 2) t = t * (double)g.dx * (double)g.dy;
      r = (float)t;
      break;
    }
    case SO_ENER_TOTAL: {  // calcener: et = ek + ei + ep + le of the scaled terms
      double e[4];
      for (int c = 0; c < 4; c++) {
        double t = 0.0;
        for (int q = lane; q < nrec; q += SF_NT) t = t + L[q].s[c];
        e[c] = block_total(t, S) * (double)(g.dx * g.dy * g.dz);
      }
      r = (float)(((e[0] + e[1]) + e[2]) + e[3]);
      break;
    }
    default:  // SO_ZERO, and SO_HOST (filled by the host)
      r = 0.0f;
      break;
  }
  if (lane == 0) rstat[p] = r;
}

void launch_stat(const DGrid &g, const StatFields &f, const StatConsts &s, const StatJob *hjobs, const StatJob *jobs,
                 int njobs, StatLev *lev, int maxlev, int nch, const StatOp *ops, int nops, float *rstat, cudaStream_t st,
                 int64_t *nl) {
  StatFlow F;
  for (int &q : F.m) q = -1;
  for (int &q : F.s) q = -1;
  F.the_nlev = 0;
  StatRest R;
  R.n = 0;
  int flow = 0, nlev = 0;
  auto rest = [&]() {   // the jobs outside k_stat_flow gathered so far
    if (R.n == 0) return;
    dim3 grid((unsigned)nch, (unsigned)nlev);
    { ProfScope _ps("k_stat_levels", st); k_stat_levels<<<grid, ST_NT, 0, st>>>(g, f, s, jobs, R, lev, maxlev, nch); }
    if (nl) *nl += 1;
    R.n = 0;
    nlev = 0;
  };
  for (int q = 0; q < njobs; q++) {
    const StatJob &j = hjobs[q];
    int *slot = nullptr;
    if (j.kind == SK_FIELD) {
      if (j.src == SF_U) slot = &F.m[FM_U];
      else if (j.src == SF_V) slot = &F.m[FM_V];
      else if (j.src == SF_W) slot = &F.m[FM_W];
      else if (j.src == SF_PPI) slot = &F.m[FM_PPI];
      else if (j.src == SF_THA) slot = &F.m[FM_THA];
      else if (j.src == SF_Q && j.qn == s.nqv) slot = &F.m[FM_QV];
    } else if (j.kind == SK_PP) slot = &F.m[FM_PP];
    else if (j.kind == SK_DIV) slot = &F.m[FM_DIV];
    else if (j.kind == SK_RH) slot = &F.m[FM_RH];
    else if (j.kind == SK_THE) { slot = &F.m[FM_THE]; F.the_nlev = j.nlev; }
    else if (j.kind == SK_WSP) slot = &F.m[FM_WSP];
    else if (j.kind == SK_CFL) slot = &F.m[FM_CFL];
    else if (j.kind == SK_MASS) slot = &F.s[FS_MASS];
    else if (j.kind == SK_TMOIS) slot = &F.s[FS_TMOIS];
    else if (j.kind == SK_QMAS && j.qn == s.nqv) slot = &F.s[FS_QMAS];
    else if (j.kind == SK_TMF) slot = &F.s[FS_TMF];
    else if (j.kind == SK_MOE) slot = &F.s[FS_MOE];
    else if (j.kind == SK_ENER) slot = &F.s[FS_ENER];
    if (j.nlev == 0) continue;
    if (slot) { *slot = q; flow = 1; continue; }
    if (R.n == ST_MAXREST || nlev + j.nlev > 65535) rest();   // a launch grid's y extent
    R.first[R.n] = nlev;
    R.job[R.n++] = q;
    nlev += j.nlev;
  }
  rest();
  if (flow) {
    dim3 grid((unsigned)nch, (unsigned)(F.m[FM_W] >= 0 ? g.nk + 1 : g.nk));
    int sums = 0;
    for (int q = 0; q < FS_N; q++)
      if (F.s[q] >= 0) sums = std::max(sums, q == FS_MOE || q == FS_ENER ? 2 : 1);
    // the sharing of rows whose warps take the fewest turns
    const int rpc = (g.nj + 1 + nch - 1) / nch, nseg = (g.ni + 32) / 32;
    int wpr = 1, turns = 0;
    for (int p = 1; p <= ST_NW; p *= 2) {
      const int n = (rpc * p + ST_NW - 1) / ST_NW * ((nseg + p - 1) / p);
      if (p == 1 || n < turns) { wpr = p; turns = n; }
    }
    ProfScope _ps("k_stat_flow", st);
    bool ext = false;
    for (int q : F.m) ext = ext || q >= 0;
    const auto flow_pass = sums == 2 && wpr == 1 && F.m[FM_WSP] >= 0 ? k_stat_flow<2, true, true>
                           : sums == 2 ? (ext ? k_stat_flow<2, true, false> : k_stat_flow<2, false, false>)
                           : sums == 1 ? (ext ? k_stat_flow<1, true, false> : k_stat_flow<1, false, false>)
                                       : k_stat_flow<0, true, false>;
    flow_pass<<<grid, ST_NT, 0, st>>>(g, f, s, F, lev, maxlev, nch, wpr);
    if (nl) *nl += 1;
  }
  if (nops > 0) {
    ProfScope _ps("k_stat_finish", st);
    k_stat_finish<<<(unsigned)nops, SF_NT, 0, st>>>(g, s, jobs, lev, maxlev, nch, ops, nops, rstat);
    if (nl) *nl += 1;
  }
}

}  // namespace cm1g
