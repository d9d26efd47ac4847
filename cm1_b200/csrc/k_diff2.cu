// k_diff2.cu -- 2nd-order diffusion with a fixed viscosity (difforder=2):
// the stress tensor of diff2def (diff2.F:743-1221, Cartesian grid, no
// terrain) and the tendencies diff2u/v/w/s (diff2.F:11-735) that solve1 adds
// to uten1 ... ptten (solve1.F:686-734), with rr = 1/rho and the w-level
// density rf of solve3.F:660-678.
//
// Without lateral walls one launch does it all (k_d2_flow): a tile of columns
// marches upward, the tensor of a point is formed once and passed to the
// neighbours that difference it by warp shuffles (x), shared rows (y) and
// registers (z); 256x256x80 with theta and three tracers takes 0.274 ms (67 %
// of the issue slots, 26 % of the DRAM peak) against 0.438 through memory.  Up to
// three scalars go with the momentum, further ones three a launch.
// Lateral walls (free slip 3, no slip 4) rewrite the tensor
// along the sides in the reference's order, corners included, so grids with
// walls keep it in memory: k_d2_tensor forms rr, rf, divx and the raw
// t11..t33 at every point; k_d2_lateral applies the wall conditions;
// k_d2_column applies the bottom/top conditions and the rf weighting of t13,
// t23 column by column; k_d2_tend adds the momentum tendencies and the scalar
// ones.
// Binary32 throughout in the Fortran's evaluation order (--fmad=false).
#include "cm1g_common.cuh"
#include "k_diff2.cuh"

namespace cm1g {

__global__ void k_d2_tensor(DGrid g, Diff2Args a) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);   // 0 .. ni+1
  const int j = (int)blockIdx.y;                                // 0 .. nj+1
  const int k = 1 + (int)blockIdx.z;                            // 1 .. nk+1
  if (i > g.ni + 1) return;
  const int nk = g.nk;
  const float coef = a.kdiff2;
  const long o = iS(g, i, j, k);
  const long pl = (long)g.NI * g.NJ;
  const float *rho = a.rho, *ua = a.ua, *va = a.va, *wa = a.wa;
  // rr and rf (solve3.F:660-678)
  if (k <= nk) a.rr[o] = 1.0f / rho[o];
  if (k == 1) a.rf[o] = a.cgs1 * rho[o] + a.cgs2 * rho[o + pl] + a.cgs3 * rho[o + 2 * pl];
  else if (k == nk + 1) a.rf[o] = a.cgt1 * rho[o - pl] + a.cgt2 * rho[o - 2 * pl] + a.cgt3 * rho[o - 3 * pl];
  else a.rf[o] = LDG(&g.c1[k]) * rho[o - pl] + LDG(&g.c2[k]) * rho[o];
  if (k <= nk) {
    // diff2def.F:773-795: divx and the stress tensor at s-points and t12
    const long ou = iU(g, i, j, k), ov = iV(g, i, j, k);
    const float uh = LDG(&g.uh[i - g.ib]), vh = LDG(&g.vh[j - g.jb]), mh = LDG(&g.mh[k]);
    float dv = (ua[ou + 1] - ua[ou]) * g.rdx * uh + (va[ov + g.NI] - va[ov]) * g.rdy * vh +
               (wa[o + pl] - wa[o]) * g.rdz * mh;
    if (fabsf(dv) < g.smeps) dv = 0.0f;
    a.divx[o] = dv;
    a.t11[o] = coef * rho[o] * (ua[ou + 1] - ua[ou]) * g.rdx * uh;
    a.t22[o] = coef * rho[o] * (va[ov + g.NI] - va[ov]) * g.rdy * vh;
    a.t33[o] = coef * rho[o] * (wa[o + pl] - wa[o]) * g.rdz * mh;
    const float uf = LDG(&g.uf[i - g.ib]), vf = LDG(&g.vf[j - g.jb]);
    a.t12[o] = coef * ((ua[ou] - ua[ou - (g.NI + 1)]) * g.rdy * vf + (va[ov] - va[ov - 1]) * g.rdx * uf) * 0.25f *
               ((rho[o - 1 - g.NI] + rho[o]) + (rho[o - 1] + rho[o - g.NI]));
  }
  // t13, t23 at k = 2..nk (diff2def.F:852-858)
  if (k >= 2 && k <= nk && i >= 1 && j >= 1) {
    const long ou = iU(g, i, j, k), ov = iV(g, i, j, k);
    const float mf = LDG(&g.mf[k]), uf = LDG(&g.uf[i - g.ib]), vf = LDG(&g.vf[j - g.jb]);
    a.t13[o] = coef * ((ua[ou] - ua[ou - (long)(g.NI + 1) * g.NJ]) * g.rdz * mf + (wa[o] - wa[o - 1]) * g.rdx * uf);
    a.t23[o] = coef * ((va[ov] - va[ov - (long)g.NI * (g.NJ + 1)]) * g.rdz * mf + (wa[o] - wa[o - g.NI]) * g.rdy * vf);
  } else if (k == 1 || k == nk + 1) {
    a.t13[o] = 0.0f;   // set by the bottom/top conditions where the tendencies read them
    a.t23[o] = 0.0f;
  }
}

// Lateral walls (diff2def.F:797-917): one warp per level, the four sides in
// the reference's order (west, east, south, north), lanes along a side.
__global__ void k_d2_lateral(DGrid g, Diff2Args a) {
  const int k = 1 + (int)blockIdx.x;
  const int lane = (int)threadIdx.x;
  const int ni = g.ni, nj = g.nj;
  const float coef = a.kdiff2;
  const float *rho = a.rho;
  auto R4 = [&](int i, int j) {   // (rho(i-1,j-1)+rho(i,j))+(rho(i-1,j)+rho(i,j-1)); the 0.25 is applied before it
    return (rho[iS(g, i - 1, j - 1, k)] + rho[iS(g, i, j, k)]) + (rho[iS(g, i - 1, j, k)] + rho[iS(g, i, j - 1, k)]);
  };
  float *t12 = a.t12, *t13 = a.t13, *t23 = a.t23;
  // t12 at every level 1..nk
  if (g.wbc == 3 && g.ibw) for (int j = 1 + lane; j <= nj + 1; j += 32) t12[iS(g, 1, j, k)] = t12[iS(g, 2, j, k)];
  else if (g.wbc == 4 && g.ibw)
    for (int j = 1 + lane; j <= nj + 1; j += 32)
      t12[iS(g, 1, j, k)] = coef * 2.0f * a.va[iV(g, 1, j, k)] * g.rdx * LDG(&g.uf[1 - g.ib]) * 0.25f * R4(1, j);
  __syncwarp();
  if (g.ebc == 3 && g.ibe) for (int j = 1 + lane; j <= nj + 1; j += 32) t12[iS(g, ni + 1, j, k)] = t12[iS(g, ni, j, k)];
  else if (g.ebc == 4 && g.ibe)
    for (int j = 1 + lane; j <= nj + 1; j += 32)
      t12[iS(g, ni + 1, j, k)] = -coef * 2.0f * a.va[iV(g, ni, j, k)] * g.rdx * LDG(&g.uf[ni + 1 - g.ib]) * 0.25f * R4(ni + 1, j);
  __syncwarp();
  if (g.sbc == 3 && g.ibs) for (int i = 1 + lane; i <= ni + 1; i += 32) t12[iS(g, i, 1, k)] = t12[iS(g, i, 2, k)];
  else if (g.sbc == 4 && g.ibs)
    for (int i = 1 + lane; i <= ni + 1; i += 32)
      t12[iS(g, i, 1, k)] = coef * 2.0f * a.ua[iU(g, i, 1, k)] * g.rdy * LDG(&g.vf[1 - g.jb]) * 0.25f * R4(i, 1);
  __syncwarp();
  if (g.nbc == 3 && g.ibn) for (int i = 1 + lane; i <= ni + 1; i += 32) t12[iS(g, i, nj + 1, k)] = t12[iS(g, i, nj, k)];
  else if (g.nbc == 4 && g.ibn)
    for (int i = 1 + lane; i <= ni + 1; i += 32)
      t12[iS(g, i, nj + 1, k)] = -coef * 2.0f * a.ua[iU(g, i, nj, k)] * g.rdy * LDG(&g.vf[nj + 1 - g.jb]) * 0.25f * R4(i, nj + 1);
  __syncwarp();
  if (k == 1) return;   // t13, t23 at k = 2..nk
  if (g.wbc == 3 && g.ibw) for (int j = 1 + lane; j <= nj; j += 32) t13[iS(g, 1, j, k)] = t13[iS(g, 2, j, k)];
  else if (g.wbc == 4 && g.ibw)
    for (int j = 1 + lane; j <= nj; j += 32) t13[iS(g, 1, j, k)] = coef * 2.0f * a.wa[iS(g, 1, j, k)] * g.rdx * LDG(&g.uf[1 - g.ib]);
  __syncwarp();
  if (g.ebc == 3 && g.ibe) for (int j = 1 + lane; j <= nj; j += 32) t13[iS(g, ni + 1, j, k)] = t13[iS(g, ni, j, k)];
  else if (g.ebc == 4 && g.ibe)
    for (int j = 1 + lane; j <= nj; j += 32)
      t13[iS(g, ni + 1, j, k)] = -coef * 2.0f * a.wa[iS(g, ni, j, k)] * g.rdx * LDG(&g.uf[ni + 1 - g.ib]);
  __syncwarp();
  if (g.sbc == 3 && g.ibs) for (int i = 1 + lane; i <= ni; i += 32) t23[iS(g, i, 1, k)] = t23[iS(g, i, 2, k)];
  else if (g.sbc == 4 && g.ibs)
    for (int i = 1 + lane; i <= ni; i += 32) t23[iS(g, i, 1, k)] = coef * 2.0f * a.wa[iS(g, i, 1, k)] * g.rdy * LDG(&g.vf[1 - g.jb]);
  __syncwarp();
  if (g.nbc == 3 && g.ibn) for (int i = 1 + lane; i <= ni; i += 32) t23[iS(g, i, nj + 1, k)] = t23[iS(g, i, nj, k)];
  else if (g.nbc == 4 && g.ibn)
    for (int i = 1 + lane; i <= ni; i += 32)
      t23[iS(g, i, nj + 1, k)] = -coef * 2.0f * a.wa[iS(g, i, nj, k)] * g.rdy * LDG(&g.vf[nj + 1 - g.jb]);
}

// Bottom/top conditions and the rf weighting of t13, t23 (diff2def.F:926-989)
__global__ void k_d2_column(DGrid g, Diff2Args a) {
  const int i = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);   // 1 .. ni+1
  const int j = 1 + (int)blockIdx.y;                                // 1 .. nj+1
  if (i > g.ni + 1) return;
  const int nk = g.nk;
  const float coef = a.kdiff2;
  float *t13 = a.t13, *t23 = a.t23;
  const bool in13 = j <= g.nj, in23 = i <= g.ni;   // ranges of the t13 and t23 conditions
  const long o1 = iS(g, i, j, 1), o2 = iS(g, i, j, 2), on = iS(g, i, j, nk), on1 = iS(g, i, j, nk + 1);
  const float mf1 = LDG(&g.mf[1]), mfn = LDG(&g.mf[nk + 1]);
  if (a.bbc == 1) {
    if (in13) t13[o1] = t13[o2];
    if (in23) t23[o1] = t23[o2];
  } else if (a.bbc == 2) {
    if (in13) t13[o1] = coef * 2.0f * (a.ua[iU(g, i, j, 1)] + 0.0f) * g.rdz * mf1;
    if (in23) t23[o1] = coef * 2.0f * (a.va[iV(g, i, j, 1)] + 0.0f) * g.rdz * mf1;
  }
  if (a.tbc == 1) {
    if (in13) t13[on1] = t13[on];
    if (in23) t23[on1] = t23[on];
  } else if (a.tbc == 2) {
    if (in13) t13[on1] = -coef * 2.0f * a.ua[iU(g, i, j, nk)] * g.rdz * mfn;
    if (in23) t23[on1] = -coef * 2.0f * a.va[iV(g, i, j, nk)] * g.rdz * mfn;
  }
  for (int k = 1; k <= nk + 1; k++) {
    const long o = iS(g, i, j, k);
    t13[o] = t13[o] * 0.5f * (a.rf[o - 1] + a.rf[o]);
    t23[o] = t23[o] * 0.5f * (a.rf[o - g.NI] + a.rf[o]);
  }
}

// diff2u/v/w (diff2.F:11-532) and diff2s (diff2.F:540-735) for nsc scalars
__global__ void k_d2_tend(DGrid g, Diff2Args a) {
  const int i = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);   // 1 .. ni+1
  const int j = 1 + (int)blockIdx.y;                                // 1 .. nj+1
  const int k = 1 + (int)blockIdx.z;                                // 1 .. nk
  if (i > g.ni + 1) return;
  const int ni = g.ni, nj = g.nj, nk = g.nk;
  const float twdth = 2.0f / 3.0f;
  const long o = iS(g, i, j, k), pl = (long)g.NI * g.NJ;
  const float *rho = a.rho;
  const float rdx = g.rdx, rdy = g.rdy, rdz = g.rdz;
  {
    if (j <= nj) {   // u at (i, j), i = 1..ni+1
      const float d0 = 2.0f * a.t11[o] - rho[o] * twdth * a.divx[o];
      const float dm = 2.0f * a.t11[o - 1] - rho[o - 1] * twdth * a.divx[o - 1];
      const float fx = (d0 - dm) * rdx * LDG(&g.uf[i - g.ib]);
      const float fy = (a.t12[o + g.NI] - a.t12[o]) * rdy * LDG(&g.vh[j - g.jb]);
      const float fz = (a.t13[o + pl] - a.t13[o]) * rdz * LDG(&g.mh[k]);
      const long ou = iU(g, i, j, k);
      a.uten[ou] = a.uten[ou] + ((fx + fy) + fz) / (0.5f * (rho[o - 1] + rho[o]));
    }
    if (i <= ni) {   // v at (i, j), j = 1..nj+1
      const float fx = (a.t12[o + 1] - a.t12[o]) * rdx * LDG(&g.uh[i - g.ib]);
      const float d0 = 2.0f * a.t22[o] - rho[o] * twdth * a.divx[o];
      const float dm = 2.0f * a.t22[o - g.NI] - rho[o - g.NI] * twdth * a.divx[o - g.NI];
      const float fy = (d0 - dm) * rdy * LDG(&g.vf[j - g.jb]);
      const float fz = (a.t23[o + pl] - a.t23[o]) * rdz * LDG(&g.mh[k]);
      const long ov = iV(g, i, j, k);
      a.vten[ov] = a.vten[ov] + ((fx + fy) + fz) / (0.5f * (rho[o - g.NI] + rho[o]));
    }
    if (i <= ni && j <= nj && k >= 2) {   // w at (i, j, k), k = 2..nk
      const float fx = (a.t13[o + 1] - a.t13[o]) * rdx * LDG(&g.uh[i - g.ib]);
      const float fy = (a.t23[o + g.NI] - a.t23[o]) * rdy * LDG(&g.vh[j - g.jb]);
      const float d0 = 2.0f * a.t33[o] - rho[o] * twdth * a.divx[o];
      const float dm = 2.0f * a.t33[o - pl] - rho[o - pl] * twdth * a.divx[o - pl];
      const float fz = (d0 - dm) * rdz * LDG(&g.mf[k]);
      a.wten[o] = a.wten[o] + ((fx + fy) + fz) / a.rf[o];
    }
  }
  if (i > ni || j > nj) return;
  // scalars (diff2s): x, y and z fluxes of each s, sten += (...)*rr
  const float coef = a.kdiff2;
  const float uf0 = LDG(&g.uf[i - g.ib]), uf1 = LDG(&g.uf[i + 1 - g.ib]);
  const float vf0 = LDG(&g.vf[j - g.jb]), vf1 = LDG(&g.vf[j + 1 - g.jb]);
  const float uh = LDG(&g.uh[i - g.ib]), vh = LDG(&g.vh[j - g.jb]), mh = LDG(&g.mh[k]);
  const float mf0 = LDG(&g.mf[k]), mf1 = LDG(&g.mf[k + 1]);
  // rolled: 256x256x160 with five scalars 490 us, 530 as the compiler unrolls it
#pragma unroll 1
  for (int n = 0; n < a.nsc; n++) {
    const float *s = a.s[n];
    const float dxl = 0.5f * (rho[o] + rho[o - 1]) * (s[o] - s[o - 1]) * rdx * uf0;
    const float dxr = 0.5f * (rho[o + 1] + rho[o]) * (s[o + 1] - s[o]) * rdx * uf1;
    const float dfx = coef * (dxr - dxl) * rdx * uh;
    const float dyl = 0.5f * (rho[o] + rho[o - g.NI]) * (s[o] - s[o - g.NI]) * rdy * vf0;
    const float dyr = 0.5f * (rho[o + g.NI] + rho[o]) * (s[o + g.NI] - s[o]) * rdy * vf1;
    const float dfy = coef * (dyr - dyl) * rdy * vh;
    const float dzl = (k == 1) ? 0.0f : (s[o] - s[o - pl]) * rdz * mf0;
    const float dzu = (k == nk) ? 0.0f : (s[o + pl] - s[o]) * rdz * mf1;
    const float dfz = coef * (a.rf[o + pl] * dzu - a.rf[o] * dzl) * rdz * mh;
    a.sten[n][o] = a.sten[n][o] + ((dfx + dfy) + dfz) * a.rr[o];
  }
}

__device__ __forceinline__ float from_west(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float from_east(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }

constexpr int D2_TY = 12;

// A block owns 30 x (D2_TY-2) points: thread (lane, row) is the point (30 bx
// + lane, (D2_TY-2) by + row); the outer lanes and rows only supply
// neighbours.  It marches through the s-levels kc0 .. kc0+kc-1, the level
// above loading while a level computes, and adds the momentum tendencies
// (MOM) and those of the scalars n0 .. n0+NS-1.
template <int NS, bool MOM>
__global__ void __launch_bounds__(32 * D2_TY, 2) k_d2_flow(DGrid g, Diff2Args a, int kc, int n0) {
  __shared__ float s12[2][D2_TY][32], s22[2][D2_TY][32], s23[2][D2_TY][32], shy[2][D2_TY][32];
  const int lane = threadIdx.x, row = threadIdx.y;
  const int i = (int)blockIdx.x * 30 + lane, j = (int)blockIdx.y * (D2_TY - 2) + row;
  const int ni = g.ni, nj = g.nj, nk = g.nk, NI = g.NI;
  const int pl = NI * g.NJ, plU = (NI + 1) * g.NJ, plV = NI * (g.NJ + 1);   // < 2^31 points (cm1g_init)
  const bool valid = i <= ni + 2 && j <= nj + 1;           // the last u point needs the column east of it
  const bool owner = lane >= 1 && lane < 31 && row >= 1 && row < D2_TY - 1 && i <= ni + 1 && j <= nj + 1;
  const bool own_u = owner && j <= nj, own_v = owner && i <= ni, own_s = own_u && own_v;
  const int kc0 = 1 + (int)blockIdx.z * kc, kc1 = min(nk, kc0 + kc - 1);
  const float coef = a.kdiff2, twdth = 2.0f / 3.0f, rdx = g.rdx, rdy = g.rdy, rdz = g.rdz, smeps = g.smeps;
  // threads outside the arrays' ring follow the column (ib, jb+1) and supply nothing that is used
  const int ic = valid ? i - g.ib : 0, jc = valid ? j - g.jb : 1;
  const float uh = LDG(&g.uh[ic]), vh = LDG(&g.vh[jc]), uf = LDG(&g.uf[ic]), vf = LDG(&g.vf[jc]), vfn = LDG(&g.vf[jc + 1]);
  const int oc = ic + NI * jc, ocu = ic + (NI + 1) * jc;

  // a level of the column and of its y neighbours (x neighbours come by shuffles)
  struct Lev { float u, us, v, vn, w, ws, r, rs; };
  auto load = [&](int k) -> Lev {
    const int o = k * pl + oc, ou = k * plU + ocu, ov = k * plV + oc;
    return Lev{LDG(&a.ua[ou]), LDG(&a.ua[ou - (NI + 1)]), LDG(&a.va[ov]), LDG(&a.va[ov + NI]), LDG(&a.wa[o]),
               LDG(&a.wa[o - NI]), LDG(&a.rho[o]), LDG(&a.rho[o - NI])};
  };
  // w-level density at the bottom (kk = 1) and top (nk+1) rows (solve3.F:660-678), offset d from the column
  auto rf_end = [&](int d, int kk) -> float {
    const float *q = a.rho + kk * pl + oc + d;
    if (kk == 1) return a.cgs1 * q[0] + a.cgs2 * q[pl] + a.cgs3 * q[2 * pl];
    return a.cgt1 * q[-pl] + a.cgt2 * q[-2 * pl] + a.cgt3 * q[-3 * pl];
  };
  // a w-level: t13, t23 before the rf weighting (raw) and after it, and rf (diff2def.F:852-858, 926-989)
  struct WLev { float x13, x23, t13, t23, rf; };
  auto weigh = [&](float x13, float x23, float rfc, float rfy) -> WLev {
    return WLev{x13, x23, x13 * 0.5f * (from_west(rfc) + rfc), x23 * 0.5f * (rfy + rfc), rfc};
  };
  auto inner = [&](const Lev &lo, const Lev &hi, int kk) -> WLev {
    const float c1 = LDG(&g.c1[kk]), c2 = LDG(&g.c2[kk]), mf = LDG(&g.mf[kk]);
    return weigh(coef * ((hi.u - lo.u) * rdz * mf + (hi.w - from_west(hi.w)) * rdx * uf),
                 coef * ((hi.v - lo.v) * rdz * mf + (hi.w - hi.ws) * rdy * vf), c1 * lo.r + c2 * hi.r, c1 * lo.rs + c2 * hi.rs);
  };
  auto divx = [&](float du, float dv, float dw, float mh) -> float {   // diff2def.F:773-779
    const float d = du * rdx * uh + dv * rdy * vh + dw * rdz * mh;
    return fabsf(d) < smeps ? 0.0f : d;
  };

  Lev c = load(kc0);
  WLev wlo{0.0f, 0.0f, 0.0f, 0.0f, 1.0f};
  float d33m = 0.0f, sc[NS > 0 ? NS : 1], sm[NS > 0 ? NS : 1];   // the scalars at levels k and k-1
#pragma unroll
  for (int n = 0; n < NS; n++) { sc[n] = LDG(&a.s[n0 + n][kc0 * pl + oc]); sm[n] = LDG(&a.s[n0 + n][(kc0 - 1) * pl + oc]); }
  if (kc0 > 1) {
    const Lev m = load(kc0 - 1);
    wlo = inner(m, c, kc0);
    const float dw = c.w - m.w, mh = LDG(&g.mh[kc0 - 1]);
    d33m = 2.0f * (coef * m.r * dw * rdz * mh) - m.r * twdth * divx(from_east(m.u) - m.u, m.vn - m.v, dw, mh);
  }
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
      const float *s = a.s[n0 + m] + o;
      ts[m] = own_s ? a.sten[n0 + m][o] : 0.0f;
      sn[m] = LDG(s + pl);
      ss[m] = LDG(s - NI);
      sno[m] = LDG(s + NI);
    }
    if (k + 3 <= kc1) {              // levels ahead towards L2
      const int o3 = o + 3 * pl, o2 = o + 2 * pl;
      prefetch_l2(&a.ua[ou + 3 * plU]); prefetch_l2(&a.va[ov + 3 * plV]); prefetch_l2(&a.wa[o3]); prefetch_l2(&a.rho[o3]);
      if (MOM) { prefetch_l2(&a.uten[ou + 2 * plU]); prefetch_l2(&a.vten[ov + 2 * plV]); prefetch_l2(&a.wten[o2]); }
#pragma unroll
      for (int m = 0; m < NS; m++) { prefetch_l2(&a.s[n0 + m][o3]); prefetch_l2(&a.sten[n0 + m][o2]); }
    }
    const float mhk = LDG(&g.mh[k]), rx = from_west(c.r);
    // the w-levels of this s-level's bottom and top
    WLev whi;
    if (k < nk) {
      whi = inner(c, n, k + 1);
    } else {
      float x13 = wlo.x13, x23 = wlo.x23;                             // free slip: the row below
      if (a.tbc == 2) {
        const float mf = LDG(&g.mf[nk + 1]);
        x13 = -coef * 2.0f * c.u * rdz * mf;
        x23 = -coef * 2.0f * c.v * rdz * mf;
      }
      whi = weigh(x13, x23, rf_end(0, nk + 1), rf_end(-NI, nk + 1));
    }
    if (k == 1) {
      float x13 = whi.x13, x23 = whi.x23;                             // free slip: the row above
      if (a.bbc == 2) {
        const float mf = LDG(&g.mf[1]);
        x13 = coef * 2.0f * (c.u + 0.0f) * rdz * mf;
        x23 = coef * 2.0f * (c.v + 0.0f) * rdz * mf;
      }
      wlo = weigh(x13, x23, rf_end(0, 1), rf_end(-NI, 1));
    }
    float d11 = 0, d22 = 0, d33 = 0, t12 = 0, d11w = 0, t12e = 0, t13e = 0;
    const float hy = 0.5f * (c.r + c.rs);
    if (MOM) {
      const float du = from_east(c.u) - c.u, dv = c.vn - c.v, dw = n.w - c.w;
      const float t = c.r * twdth * divx(du, dv, dw, mhk);
      d11 = 2.0f * (coef * c.r * du * rdx * uh) - t;
      d22 = 2.0f * (coef * c.r * dv * rdy * vh) - t;
      d33 = 2.0f * (coef * c.r * dw * rdz * mhk) - t;
      t12 = coef * ((c.u - c.us) * rdy * vf + (c.v - from_west(c.v)) * rdx * uf) * 0.25f *
            ((from_west(c.rs) + c.r) + (rx + c.rs));
      s12[b][row][lane] = t12;
      s22[b][row][lane] = d22;
      s23[b][row][lane] = wlo.t23;
      d11w = from_west(d11);
      t12e = from_east(t12);
      t13e = from_east(wlo.t13);
    }
    if (NS > 0) shy[b][row][lane] = hy;
    __syncthreads();
    if (MOM) {
      if (own_u) {
        const float fx = (d11 - d11w) * rdx * uf;
        const float fy = (s12[b][row + 1][lane] - t12) * rdy * vh;
        const float fz = (whi.t13 - wlo.t13) * rdz * mhk;
        a.uten[ou] = tu + ((fx + fy) + fz) / (0.5f * (rx + c.r));
      }
      if (own_v) {
        const float fx = (t12e - t12) * rdx * uh;
        const float fy = (d22 - s22[b][row - 1][lane]) * rdy * vf;
        const float fz = (whi.t23 - wlo.t23) * rdz * mhk;
        a.vten[ov] = tv + ((fx + fy) + fz) / (0.5f * (c.rs + c.r));
      }
      if (own_s && k >= 2) {
        const float fx = (t13e - wlo.t13) * rdx * uh;
        const float fy = (s23[b][row + 1][lane] - wlo.t23) * rdy * vh;
        const float fz = (d33 - d33m) * rdz * LDG(&g.mf[k]);
        a.wten[o] = tw + ((fx + fy) + fz) / wlo.rf;
      }
    }
    if (NS > 0) {   // diff2s (diff2.F:540-735)
      const float hx = 0.5f * (c.r + rx), hyn = row < D2_TY - 1 ? shy[b][row + 1][lane] : 0.0f, rr = 1.0f / c.r;
      const float mf0 = LDG(&g.mf[k]), mf1 = LDG(&g.mf[k + 1]);
#pragma unroll
      for (int m = 0; m < NS; m++) {
        const float fx0 = hx * (sc[m] - from_west(sc[m])) * rdx * uf, fx1 = from_east(fx0);
        const float dfx = coef * (fx1 - fx0) * rdx * uh;
        const float dfy = coef * (hyn * (sno[m] - sc[m]) * rdy * vfn - hy * (sc[m] - ss[m]) * rdy * vf) * rdy * vh;
        const float dzl = (k == 1) ? 0.0f : (sc[m] - sm[m]) * rdz * mf0;
        const float dzu = (k == nk) ? 0.0f : (sn[m] - sc[m]) * rdz * mf1;
        const float dfz = coef * (whi.rf * dzu - wlo.rf * dzl) * rdz * mhk;
        if (own_s) a.sten[n0 + m][o] = ts[m] + ((dfx + dfy) + dfz) * rr;
        sm[m] = sc[m];
        sc[m] = sn[m];
      }
    }
    wlo = whi; d33m = d33;
    c = n;
  }
}

template <bool MOM>
static void d2_flow(const DGrid &g, const Diff2Args &a, int ns, int n0, cudaStream_t st) {
  dim3 blk(32, D2_TY), grid((g.ni + 1 + 29) / 30, (g.nj + 1 + D2_TY - 3) / (D2_TY - 2));
  const int kc = tile_levels((long)grid.x * grid.y, g.nk, 2 * 148, 3, 4, 128);
  grid.z = (g.nk + kc - 1) / kc;
  ProfScope _ps("k_d2_flow", st);
  switch (ns) {
    case 0: k_d2_flow<0, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    case 1: k_d2_flow<1, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    case 2: k_d2_flow<2, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
    default: k_d2_flow<3, MOM><<<grid, blk, 0, st>>>(g, a, kc, n0); break;
  }
}

bool diff2_walls(const DGrid &g) {
  return (g.ibw && (g.wbc == 3 || g.wbc == 4)) || (g.ibe && (g.ebc == 3 || g.ebc == 4)) ||
         (g.ibs && (g.sbc == 3 || g.sbc == 4)) || (g.ibn && (g.nbc == 3 || g.nbc == 4));
}

void launch_diff2(const DGrid &g, const Diff2Args &a, cudaStream_t st, int64_t *nl) {
  if (!diff2_walls(g)) {
    // momentum with up to three scalars, then three scalars a launch
    d2_flow<true>(g, a, a.nsc < 3 ? a.nsc : 3, 0, st);
    if (nl) *nl += 1;
    for (int n0 = 3; n0 < a.nsc; n0 += 3) {
      d2_flow<false>(g, a, a.nsc - n0 < 3 ? a.nsc - n0 : 3, n0, st);
      if (nl) *nl += 1;
    }
    return;
  }
  {
    dim3 grid((g.ni + 2 + 127) / 128, g.nj + 2, g.nk + 1);
    ProfScope _ps("k_d2_tensor", st);
    k_d2_tensor<<<grid, 128, 0, st>>>(g, a);
  }
  {
    ProfScope _ps("k_d2_lateral", st);
    k_d2_lateral<<<g.nk, 32, 0, st>>>(g, a);
  }
  {
    dim3 grid((g.ni + 1 + 127) / 128, g.nj + 1);
    ProfScope _ps("k_d2_column", st);
    k_d2_column<<<grid, 128, 0, st>>>(g, a);
  }
  {
    dim3 grid((g.ni + 1 + 127) / 128, g.nj + 1, g.nk);
    ProfScope _ps("k_d2_tend", st);
    k_d2_tend<<<grid, 128, 0, st>>>(g, a);
  }
  if (nl) *nl += 4;
}

}  // namespace cm1g
