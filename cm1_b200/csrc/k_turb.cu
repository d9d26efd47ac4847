// k_turb.cu -- Smagorinsky subgrid turbulence (sgsmodel=2) of an LES,
// Cartesian grid without terrain, periodic lateral boundaries, dry N^2,
// explicit vertical mixing (doimpl=0):
//   calcdef   rho*S_ij and the deformations defv, defh (turb.F:4711-5423)
//   calcnm    dry squared Brunt-Vaisala frequency (turb.F:5432-5480)
//   turbsmag  kmh, kmv for tconfig 1 and 2, bcw's zero rows and periodic
//             halo, khh = kmh/Pr, khv = kmv/Pr (turb.F:3375-3621)
//   gettau    stresses t_ij = 2 K rho S_ij with sfcstress's bbc 1/2 and the
//             top conditions tbc 1/2 (turb.F:4059-4506, 4515-4582)
//   turbu, turbv, turbw, turbs/turbsz   the tendencies solve1 adds to
//             uten1, vten1, wten1, thten1, qten, ptten (turbtend.F:18-692,
//             1052-1424, 1816-2180, 2473-2885; solve1.F:1113-1240)
//
// Two launches, both tiles of columns that march upward with the values of
// the level below in registers:
//   k_les_km    the strains, N^2 and the deformations of a w-level, and from
//               them kmh and kmv (the halo ring is written from its periodic
//               image, which equals bcw's copy)
//   k_les_tend  the strains again, the stresses t_ij, the scalar fluxes' face
//               coefficients, and every tendency
// The strains and stresses live in registers, warp shuffles (x neighbours)
// and a few shared rows (y neighbours) only: forming the strain twice costs
// about 60 binary32 operations a point, storing and re-reading the twelve
// strain, stress and coefficient arrays cost 48 to 100 bytes a point.
// Bound by instruction issue (71 and 61 % of the cycles; 558 and 884 warp
// instructions per 32 points), at 14 and 25 % of the DRAM peak.  256x256x128
// with theta and two tracers: 0.583 ms a call against 1.33 for the four
// point-parallel passes before.  With every neighbour loaded instead of
// shuffled the two passes took 0.81 ms, and without reading a level's
// tendencies ahead of its stores (which may alias for the compiler) 1.03 ms.
// Binary32 in the Fortran's evaluation order (--fmad=false); the logarithm
// of calcnm and the cube root of tconfig=1 are evaluated in binary64 and
// rounded once.
#include "cm1g_common.cuh"
#include "k_turb.cuh"

namespace cm1g {

__device__ __forceinline__ float sq(float x) { return x * x; }

__device__ __forceinline__ float from_west(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float from_east(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Rows of threads of a tile (x: 32 lanes, of which 30 own points).
constexpr int LK_TY = 16, LT_TY = 12;

// calcdef (turb.F:4772-4790, 4880-4893, 5366-5390), calcnm (dry) and kmh/kmv
// of turbsmag.  A block owns 30 x (LK_TY-1) columns: thread (lane, row) is the
// point (30 bx + lane, (LK_TY-1) by + 1 + row); the outer lanes and the last
// row only supply neighbours.  It marches through the w-levels kc0 ..
// kc0+kc-1, the level above loading while a level computes.  The bottom and
// top rows are zero (bcw flag 1, bc.F:1126-1137).
__global__ void __launch_bounds__(32 * LK_TY, 2) k_les_km(DGrid g, TurbArgs a, int kc) {
  __shared__ float s12[2][LK_TY][32], s23s[2][LK_TY][32];
  const int lane = threadIdx.x, row = threadIdx.y;
  const int i = (int)blockIdx.x * 30 + lane, j = 1 + (int)blockIdx.y * (LK_TY - 1) + row;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI;
  const int pl = NI * g.NJ, plU = (NI + 1) * g.NJ, plV = NI * (g.NJ + 1);   // < 2^31 points (cm1g_init)
  const bool valid = i <= ni + 1 && j <= nj + 1;
  const bool owner = lane >= 1 && lane < 31 && row < LK_TY - 1 && i <= ni && j <= nj;
  const int kc0 = 2 + (int)blockIdx.z * kc, kc1 = min(nk, kc0 + kc - 1);
  const float rdx = g.rdx, rdy = g.rdy, rdz = g.rdz;
  // threads outside the arrays' ring follow the column (ib, jb+1) and supply nothing that is used
  const int ic = valid ? i - g.ib : 0, jc = valid ? j - g.jb : 1;
  const float uh = LDG(&g.uh[ic]), vh = LDG(&g.vh[jc]), uf = LDG(&g.uf[ic]), vf = LDG(&g.vf[jc]);
  const int oc = ic + NI * jc, ocu = ic + (NI + 1) * jc;
  const float dxr = g.dx * LDG(&g.ruh[ic]), dyr = g.dy * LDG(&g.rvh[jc]);

  // a value of an owned column and its periodic images on the halo ring
  auto put = [&](float *q, int k, float v) {
    float *r = q + k * pl + oc;
    const int dx = (i == 1) ? ni : (i == ni ? -ni : 0), dy = (j == 1) ? nj * NI : (j == nj ? -nj * NI : 0);
    r[0] = v;
    if (dx) r[dx] = v;
    if (dy) r[dy] = v;
    if (dx && dy) r[dx + dy] = v;
    if (ni == 1 && dx) { r[-dx] = v; if (dy) r[dy - dx] = v; }
    if (nj == 1 && dy) { r[-dy] = v; if (dx) { r[dx - dy] = v; if (ni == 1) r[-dx - dy] = v; } }
  };
  if (owner && kc0 == 2) { put(a.kmh, 1, 0.0f); put(a.kmv, 1, 0.0f); }
  if (owner && kc1 == nk) { put(a.kmh, nk + 1, 0.0f); put(a.kmv, nk + 1, 0.0f); }

  // a level of the column and of its y neighbours (x neighbours come by shuffles)
  struct Lev { float u, us, v, vn, w, ws, r, rs, th; };
  auto load = [&](int k) -> Lev {
    const int o = k * pl + oc, ou = k * plU + ocu, ov = k * plV + oc;
    return Lev{LDG(&a.ua[ou]), LDG(&a.ua[ou - (NI + 1)]), LDG(&a.va[ov]), LDG(&a.va[ov + NI]), LDG(&a.wa[o]),
               LDG(&a.wa[o - NI]), LDG(&a.rho[o]), LDG(&a.rho[o - NI]), LDG(&a.tha[o])};
  };
  // of the level below: u, v, rho, theta, the squared strains, the sum of t12^2 over the four corners
  float u0 = 0, v0 = 0, r0 = 0, rs0 = 0, th_0 = 0, q11 = 0, q22 = 0, q33 = 0, g12 = 0;
  float lastarg = -1.0f, grd1 = 0.0f;   // tconfig 1: the grid scale changes only with the metrics
  Lev c = load(kc0 - 1);
  int b = 0;
  for (int k = kc0 - 1; k <= kc1; k++, b ^= 1) {
    const bool wl = k >= kc0;        // a w-level of this block
    const Lev n = load(k + 1);
    if (k + 3 <= kc1) {              // levels ahead towards L2
      const int o = (k + 3) * pl + oc;
      prefetch_l2(&a.ua[(k + 3) * plU + ocu]); prefetch_l2(&a.va[(k + 3) * plV + oc]);
      prefetch_l2(&a.wa[o]); prefetch_l2(&a.rho[o]); prefetch_l2(&a.tha[o]);
    }
    const float t11 = c.r * (from_east(c.u) - c.u) * rdx * uh;
    const float t22 = c.r * (c.vn - c.v) * rdy * vh;
    const float t33 = c.r * (n.w - c.w) * (rdz * LDG(&g.mh[k]));
    const float t12 = 0.5f * ((c.u - c.us) * rdy * vf + (c.v - from_west(c.v)) * rdx * uf) * 0.25f *
                      ((from_west(c.rs) + c.r) + (from_west(c.r) + c.rs));
    float t13 = 0.0f, t23 = 0.0f, rfc = 1.0f;
    const float c1 = LDG(&g.c1[k]), c2 = LDG(&g.c2[k]), mf = LDG(&g.mf[k]);
    if (wl) {
      rfc = c1 * r0 + c2 * c.r;
      const float rfy = c1 * rs0 + c2 * c.rs;
      t13 = 0.5f * ((c.w - from_west(c.w)) * rdx * uf + (c.u - u0) * rdz * 0.5f * (mf + mf)) * 0.5f * (from_west(rfc) + rfc);
      t23 = 0.5f * ((c.w - c.ws) * rdy * vf + (c.v - v0) * rdz * 0.5f * (mf + mf)) * 0.5f * (rfy + rfc);
    }
    s12[b][row][lane] = t12;
    s23s[b][row][lane] = t23;
    const float t12e = from_east(t12), t13e = from_east(t13);
    __syncthreads();
    if (owner) {
      const float n11 = sq(t11), n22 = sq(t22), n33 = sq(t33);
      const float n12 = (sq(t12) + sq(s12[b][row + 1][lane + 1])) + (sq(s12[b][row + 1][lane]) + sq(t12e));
      if (wl) {
        const float tmp11 = c1 * q11 + c2 * n11, tmp22 = c1 * q22 + c2 * n22, tmp33 = c1 * q33 + c2 * n33;
        const float tmp12 = 0.25f * (c1 * g12 + c2 * n12);
        const float tmp13 = 0.5f * (sq(t13) + sq(t13e));
        const float tmp23 = 0.5f * (sq(t23) + sq(s23s[b][row + 1][lane]));
        const float rrf = 1.0f / sq(rfc);
        const float defv = 4.0f * (tmp13 + tmp23) * rrf;
        const float defh = (2.0f * ((tmp11 + tmp22) + tmp33) + 4.0f * tmp12) * rrf;
        // calcnm, imoist=0 (turb.F:5458-5468)
        const float q = (LDG(&g.th0[k]) + c.th) / (LDG(&g.th0[k - 1]) + th_0);
        const float nm = (float)log((double)q) * g.c.g * rdz * mf;
        const float dmin = 1.0e-10f;
        const float rmf = 1.0f / mf;
        float kmh, kmv;
        if (a.tconfig == 1) {
          const float arg = (dxr * dyr) * (g.dz * rmf);
          if (arg != lastarg) { grd1 = (float)pow((double)arg, (double)0.33333333f); lastarg = arg; }
          kmh = sq(a.csm * grd1) * sqrtf(fmaxf(defv + defh - nm * a.prinv, dmin));
          kmv = kmh;
        } else {
          const float lenh = sqrtf(dxr * dyr);
          const float grd = g.dz * rmf;
          kmh = sq(a.csm * lenh) * sqrtf(fmaxf(defh, dmin));
          kmv = sq(a.csm * grd) * sqrtf(fmaxf(defv - nm * a.prinv, dmin));
        }
        put(a.kmh, k, kmh);
        put(a.kmv, k, kmv);
      }
      q11 = n11; q22 = n22; q33 = n33; g12 = n12;
    }
    u0 = c.u; v0 = c.v; r0 = c.r; rs0 = c.rs; th_0 = c.th;
    c = n;
  }
}

// gettau (Cartesian) with sfcstress's bottom row and the top row (turb.F:
// 4059-4582), then turbu, turbv, turbw (turbtend.F:1101-1104, 1290-1296,
// 1408-1416, 1816-2180, 2473-2885) and turbs/turbsz of the scalars n0 ..
// n0+NS-1 (turbtend.F:66-78, 480-510).  A block owns 30 x (LT_TY-2) points:
// thread (lane, row) is the point (30 bx + lane, (LT_TY-2) by + row); the
// outer lanes and rows only supply neighbours.  It marches through the
// s-levels kc0 .. kc0+kc-1, the level above loading while a level computes.
// MOM: add the momentum tendencies too.
template <int NS, bool MOM>
__global__ void __launch_bounds__(32 * LT_TY, 2) k_les_tend(DGrid g, TurbArgs a, int kc, int n0) {
  __shared__ float s12[2][LT_TY][32], s22[2][LT_TY][32], s23[2][LT_TY][32], scy[2][LT_TY][32];
  const int lane = threadIdx.x, row = threadIdx.y;
  const int i = (int)blockIdx.x * 30 + lane, j = (int)blockIdx.y * (LT_TY - 2) + row;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI;
  const int pl = NI * g.NJ, plU = (NI + 1) * g.NJ, plV = NI * (g.NJ + 1);   // < 2^31 points (cm1g_init)
  const bool valid = i <= ni + 2 && j <= nj + 1;           // the last u point needs the column east of it
  const bool owner = lane >= 1 && lane < 31 && row >= 1 && row < LT_TY - 1 && i <= ni + 1 && j <= nj + 1;
  const bool own_u = owner && j <= nj, own_v = owner && i <= ni, own_s = own_u && own_v;
  const int kc0 = 1 + (int)blockIdx.z * kc, kc1 = min(nk, kc0 + kc - 1);
  const float rdx = g.rdx, rdy = g.rdy, rdz = g.rdz, tem = rdz * 0.5f, pr = a.prinv;
  // threads outside the arrays' ring follow the column (ib, jb+1) and supply nothing that is used
  const int ic = valid ? i - g.ib : 0, jc = valid ? j - g.jb : 1;
  const float uh = LDG(&g.uh[ic]), vh = LDG(&g.vh[jc]), uf = LDG(&g.uf[ic]), vf = LDG(&g.vf[jc]), vfn = LDG(&g.vf[jc + 1]);
  const int oc = ic + NI * jc, ocu = ic + (NI + 1) * jc;

  // a level of the column and of its y neighbours (x neighbours come by shuffles)
  struct Lev { float u, us, v, vn, w, ws, r, rs, kh, khs, kv, kvs; };
  auto load = [&](int k) -> Lev {
    const int o = k * pl + oc, ou = k * plU + ocu, ov = k * plV + oc;
    return Lev{LDG(&a.ua[ou]), LDG(&a.ua[ou - (NI + 1)]), LDG(&a.va[ov]), LDG(&a.va[ov + NI]), LDG(&a.wa[o]),
               LDG(&a.wa[o - NI]), LDG(&a.rho[o]), LDG(&a.rho[o - NI]), LDG(&a.kmh[o]), LDG(&a.kmh[o - NI]),
               LDG(&a.kmv[o]), LDG(&a.kmv[o - NI])};
  };
  // w-level density at the bottom (kk = 1) and top (nk+1) rows, offset d from the column
  auto rf_end = [&](int d, int kk) -> float {
    const float *q = a.rho + kk * pl + oc + d;
    if (kk == 1) return a.cgs1 * q[0] + a.cgs2 * q[pl] + a.cgs3 * q[2 * pl];
    return a.cgt1 * q[-pl] + a.cgt2 * q[-2 * pl] + a.cgt3 * q[-3 * pl];
  };
  struct WLev { float t13, t23, rf; };
  // an inner w-level kk = 2..nk from the s-levels below and above it
  auto inner = [&](const Lev &lo, const Lev &hi, int kk) -> WLev {
    const float c1 = LDG(&g.c1[kk]), c2 = LDG(&g.c2[kk]), mf = LDG(&g.mf[kk]);
    const float rfc = c1 * lo.r + c2 * hi.r, rfy = c1 * lo.rs + c2 * hi.rs;
    const float x13 = 0.5f * ((hi.w - from_west(hi.w)) * rdx * uf + (hi.u - lo.u) * rdz * 0.5f * (mf + mf)) * 0.5f * (from_west(rfc) + rfc);
    const float x23 = 0.5f * ((hi.w - hi.ws) * rdy * vf + (hi.v - lo.v) * rdz * 0.5f * (mf + mf)) * 0.5f * (rfy + rfc);
    return WLev{x13 * (from_west(hi.kv) + hi.kv), x23 * (hi.kvs + hi.kv), rfc};
  };
  // no slip at the bottom or top row kk (turb.F:4407-4419, 4550-4562), ugr = ua,
  // vgr = va: l the s-level beside the row, kv the viscosities of the nearest inner w-level
  auto noslip = [&](const Lev &l, const Lev &kv, int kk) -> WLev {
    const float mf = LDG(&g.mf[kk]), rfc = rf_end(0, kk);
    return WLev{2.0f * l.u * rdz * 0.5f * (mf + mf) * 0.5f * (from_west(rfc) + rfc) * 0.5f * (from_west(kv.kv) + kv.kv),
                2.0f * l.v * rdz * 0.5f * (mf + mf) * 0.5f * (rf_end(-NI, kk) + rfc) * 0.5f * (kv.kvs + kv.kv), rfc};
  };

  Lev c = load(kc0);
  WLev wlo{0.0f, 0.0f, 1.0f};
  float t33m = 0.0f, sc[NS > 0 ? NS : 1], fzl[NS > 0 ? NS : 1];
  const bool theta = NS > 0 && n0 == 0;
  auto SV = [&](int n, int k, int d) -> float {   // the scalar as turbs sees it (solve1.F:1184-1195)
    const float v = LDG(&a.s[n0 + n][k * pl + oc + d]);
    return (n == 0 && theta) ? (LDG(&g.th0[k]) - 300.0f) + v : v;
  };
#pragma unroll
  for (int n = 0; n < NS; n++) { sc[n] = SV(n, kc0, 0); fzl[n] = 0.0f; }
  if (kc0 > 1) {
    const Lev m = load(kc0 - 1);
    wlo = inner(m, c, kc0);
    t33m = m.r * (c.w - m.w) * (rdz * LDG(&g.mh[kc0 - 1])) * (m.kh + c.kh);
#pragma unroll
    for (int n = 0; n < NS; n++) fzl[n] = -(c.kv * pr) * (sc[n] - SV(n, kc0 - 1, 0)) * rdz * LDG(&g.mf[kc0]) * wlo.rf;
  }
  float k40 = (from_west(c.khs) + c.kh) + (from_west(c.kh) + c.khs);
  float hx0 = c.kh * pr + from_west(c.kh) * pr, hy0 = c.kh * pr + c.khs * pr;
  int b = 0;
  for (int k = kc0; k <= kc1; k++, b ^= 1) {
    const int o = k * pl + oc, ou = k * plU + ocu, ov = k * plV + oc;
    // every global read of the level, before anything is stored
    const Lev n = load(k + 1);
    float tu = 0, tv = 0, tw = 0, ts[NS > 0 ? NS : 1], sn[NS > 0 ? NS : 1], ss[NS > 0 ? NS : 1], sno[NS > 0 ? NS : 1];
    if (MOM) {
      if (own_u) tu = a.uten[ou];
      if (own_v) tv = a.vten[ov];
      if (own_s && k >= 2) tw = a.wten[o];
    }
#pragma unroll
    for (int m = 0; m < NS; m++) {
      ts[m] = own_s ? a.sten[n0 + m][o] : 0.0f;
      sn[m] = SV(m, k + 1, 0);
      ss[m] = SV(m, k, -NI);
      sno[m] = SV(m, k, NI);
    }
    if (k + 3 <= kc1) {              // levels ahead towards L2
      const int o3 = o + 3 * pl, o2 = o + 2 * pl;
      prefetch_l2(&a.ua[ou + 3 * plU]); prefetch_l2(&a.va[ov + 3 * plV]);
      prefetch_l2(&a.wa[o3]); prefetch_l2(&a.rho[o3]); prefetch_l2(&a.kmh[o3]); prefetch_l2(&a.kmv[o3]);
      if (MOM) { prefetch_l2(&a.uten[ou + 2 * plU]); prefetch_l2(&a.vten[ov + 2 * plV]); prefetch_l2(&a.wten[o2]); }
#pragma unroll
      for (int m = 0; m < NS; m++) { prefetch_l2(&a.s[n0 + m][o3]); prefetch_l2(&a.sten[n0 + m][o2]); }
    }
    const float mhk = LDG(&g.mh[k]), rx = from_west(c.r), temk = c.kh + n.kh;
    // the w-levels of this s-level's bottom and top
    WLev whi;
    if (k < nk) {
      whi = inner(c, n, k + 1);
      if (k == 1) {
        if (a.bbc == 1) { wlo.t13 = whi.t13; wlo.t23 = whi.t23; }     // free slip: t13(1) = t13(2)
        else wlo = noslip(c, n, 1);
      }
    } else if (a.tbc == 1) {
      whi = wlo;                                                      // t13(nk+1) = t13(nk)
    } else {
      whi = noslip(c, c, nk + 1);
      whi.t13 = -whi.t13;
      whi.t23 = -whi.t23;
    }
    const float hx1 = n.kh * pr + from_west(n.kh) * pr, hy1 = n.kh * pr + n.khs * pr;
    // turbs' face coefficients (turbtend.F:68-77): khh = kmh * prinv at the
    // four points, summed as the Fortran does, times -0.125 (rho + rho)
    const float cx = -0.125f * (c.r + rx) * (hx0 + hx1), cy = -0.125f * (c.r + c.rs) * (hy0 + hy1);
    float t11 = 0, t22 = 0, t33 = 0, t12 = 0, t11w = 0, t12e = 0, t13e = 0;
    const float k41 = (from_west(n.khs) + n.kh) + (from_west(n.kh) + n.khs);
    if (MOM) {
      t11 = c.r * (from_east(c.u) - c.u) * rdx * uh * temk;
      t22 = c.r * (c.vn - c.v) * rdy * vh * temk;
      t33 = c.r * (n.w - c.w) * (rdz * mhk) * temk;
      t12 = 0.5f * ((c.u - c.us) * rdy * vf + (c.v - from_west(c.v)) * rdx * uf) * 0.25f *
            ((from_west(c.rs) + c.r) + (rx + c.rs)) * 0.25f * (k40 + k41);
      s12[b][row][lane] = t12;
      s22[b][row][lane] = t22;
      s23[b][row][lane] = wlo.t23;
      t11w = from_west(t11);
      t12e = from_east(t12);
      t13e = from_east(wlo.t13);
    }
    if (NS > 0) scy[b][row][lane] = cy;
    __syncthreads();
    if (MOM) {
      if (own_u) {   // turbu
        const float tx = (t11 - t11w) * rdx * uf;
        const float ty = (s12[b][row + 1][lane] - t12) * rdy * vh;
        const float tz = (whi.t13 - wlo.t13) * tem * (mhk + mhk);
        const float rru0 = 1.0f / (0.5f * (rx + c.r));
        a.uten[ou] = tu + ((tx + ty) + tz) * rru0;
      }
      if (own_v) {   // turbv
        const float tx = (t12e - t12) * rdx * uh;
        const float ty = (t22 - s22[b][row - 1][lane]) * rdy * vf;
        const float tz = (whi.t23 - wlo.t23) * tem * (mhk + mhk);
        const float rrv0 = 1.0f / (0.5f * (c.rs + c.r));
        a.vten[ov] = tv + ((tx + ty) + tz) * rrv0;
      }
      if (own_s && k >= 2) {   // turbw
        const float tx = (t13e - wlo.t13) * rdx * uh;
        const float ty = (s23[b][row + 1][lane] - wlo.t23) * rdy * vh;
        const float tz = (t33 - t33m) * rdz * LDG(&g.mf[k]);
        a.wten[o] = tw + ((tx + ty) + tz) / wlo.rf;
      }
    }
    if (NS > 0) {
      const float cyn = row < LT_TY - 1 ? scy[b][row + 1][lane] : 0.0f, rr = 1.0f / c.r;
      const float khh = n.kv * pr, mfh = k < nk ? LDG(&g.mf[k + 1]) : 0.0f;
#pragma unroll
      for (int m = 0; m < NS; m++) {
        const float fx0 = cx * (sc[m] - from_west(sc[m])) * rdx * uf, fx1 = from_east(fx0);
        const float fy0 = cy * (sc[m] - ss[m]) * rdy * vf, fy1 = cyn * (sno[m] - sc[m]) * rdy * vfn;
        // vertical fluxes: at the bottom and top boundaries zero (bcturbs 1)
        // or the nearest inner level's flux
        float fz1;
        if (k < nk) fz1 = -khh * (sn[m] - sc[m]) * rdz * mfh * whi.rf;
        else fz1 = a.bcturbs == 1 ? 0.0f : fzl[m];
        const float fz0 = k > 1 ? fzl[m] : (a.bcturbs == 1 ? 0.0f : fz1);
        const float tx = -(fx1 - fx0) * rdx * uh;
        const float ty = -(fy1 - fy0) * rdy * vh;
        const float tz = -(fz1 - fz0) * rdz * mhk;
        if (own_s) a.sten[n0 + m][o] = ts[m] + ((tx + ty) + tz) * rr;
        fzl[m] = fz1;
        sc[m] = sn[m];
      }
    }
    wlo = whi; t33m = t33; k40 = k41; hx0 = hx1; hy0 = hy1;
    c = n;
  }
}

// Levels a block: those whose blocks finish first, from one level on small grids,
// whose blocks then march one step after their first (16x16x20 60 to 48 us a call
// against at least four levels).
template <bool MOM>
static void les_tend(const DGrid &g, const TurbArgs &a, int ns, int n0, cudaStream_t st) {
  dim3 blk(32, LT_TY), grid((g.ni + 1 + 29) / 30, (g.nj + 1 + LT_TY - 3) / (LT_TY - 2));
  const int kc = tile_levels((long)grid.x * grid.y, g.nk, 2 * 148, 3, 1, 128);
  grid.z = (g.nk + kc - 1) / kc;
  ProfScope _ps("k_les_tend", st);
  switch (ns) {
    case 0: k_les_tend<0, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    case 1: k_les_tend<1, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    case 2: k_les_tend<2, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    default: k_les_tend<3, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
  }
}

void launch_turbsmag(const DGrid &g, const TurbArgs &a, cudaStream_t st, int64_t *nl) {
  {
    dim3 grid((g.ni + 29) / 30, (g.nj + LK_TY - 2) / (LK_TY - 1));
    const int kc = tile_levels((long)grid.x * grid.y, g.nk - 1, 2 * 148, 3, 1, 128);
    grid.z = (g.nk - 1 + kc - 1) / kc;
    ProfScope _ps("k_les_km", st);
    k_les_km<<<grid, dim3(32, LK_TY), 0, st>>>(g, a, kc);
  }
  // momentum with up to three scalars, then three scalars a launch
  les_tend<true>(g, a, a.nsc < 3 ? a.nsc : 3, 0, st);
  if (nl) *nl += 2;
  for (int n0 = 3; n0 < a.nsc; n0 += 3) {
    les_tend<false>(g, a, a.nsc - n0 < 3 ? a.nsc - n0 : 3, n0, st);
    if (nl) *nl += 1;
  }
}

}  // namespace cm1g
