// cm1g_common.cuh -- device-side grid descriptor, Fortran-layout indexing and
// the face-value functions shared by the large-step kernels.
//
// All fields use the reference's Fortran layout (i fastest) with lower
// bounds ib=1-ngxy, jb=1-ngxy, kb=0.  Without terrain the base state and the
// vertical metrics are horizontally uniform, so the kernels read them as
// 1-D profiles indexed by k (checked when the context is created).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cm1g {

struct Consts {
  float g, rd, rv, cp, cv, cpv, cvv, cpl, cpi;
  float rovcp, rddcv, cpdrd, reps, repsm1;
};

// Everything a kernel needs to know about the grid; passed by value.
struct DGrid {
  int ni, nj, nk, ngxy;
  int ib, jb;                 // kb = 0
  int NI, NJ, NK;             // extents of s-arrays
  float dx, dy, dz, rdx, rdy, rdz;
  int wbc, ebc, sbc, nbc;
  int ibw, ibe, ibs, ibn;
  float smeps, alph, kdiv;
  int irbc;                   // open-boundary phase speeds: 1 and 2 Klemp-Wilhelmson, 4 Durran-Klemp
  float cstar;                // the Klemp-Wilhelmson gravity-wave speed of irbc 1 and 2
  int roflux;                 // 1: the open boundaries' outflow is restricted to the inflow at every acoustic step
  Consts c;
  // vertical profiles (index k, k = 0..nk+1; w-profiles to nk+2)
  const float *mh, *rmh, *mf, *rho0, *rr0, *rf0, *rrf0, *c1, *c2, *pi0, *th0, *rth0, *qv0, *qc0, *qi0;
  const float *prs0;          // base-state pressure profile (output only; null when not given)
  // horizontal metrics (index i-ib / j-jb)
  const float *uh, *ruh, *uf, *ruf, *vh, *rvh, *vf, *rvf;
  const float *dtu0, *dtv0;   // (ib:ie, jb:je)
  const float *u0, *v0;       // base-state winds, full u-/v-arrays (Rayleigh damping)
  // launch shapes (cm1g_set_tune / cm1g_autotune): index into the tile-shape
  // table of the scalar and momentum passes, and the acoustic kernel's form
  // (-1: the default, form 0)
  int tile_adv, tile_mom, sound_cfg;
};

// Launch shapes of the momentum pass.  With the 6th-order diffusion (k_mom_tile):
// x and y threads of a block and the levels it marches through.  Without it k_mom
// owns 31 x 8 points a block whatever the entry, and takes the entry's levels only
// (entry 0: levels chosen by the grid's size).  Entry 0 is the default; the others
// are the autotuner's candidates.
constexpr int kNumTileShapes = 5;
constexpr int kTileShapes[kNumTileShapes][3] = {{32, 8, 16}, {32, 8, 8}, {32, 4, 16}, {64, 4, 16}, {32, 8, 32}};
// Tile shapes of the scalar passes (k_scal_tile, k_advs_tile), indexed like
// kTileShapes: TX x TY cells and KC levels per block; the block has one more
// row of TX threads than the tile has cell rows (the row that evaluates the
// tile's north and east faces), so a block is TX x (TY + 1) threads.  k_scal_tile
// chooses the levels of entry 0 by the grid's size; k_advs_tile takes all as listed.
constexpr int kScalShapes[kNumTileShapes][3] = {{32, 7, 16}, {32, 7, 8}, {32, 3, 16}, {64, 3, 16}, {32, 7, 32}};
// Forms of the acoustic kernel: 0 tile (32 columns, the warps over the levels
// chosen by the grid's size), 1 tile with 16 explicit warps, 2 column sweep
// 32 x 4 columns, 3 column sweep 32 x 2 columns.
constexpr int kNumSoundCfgs = 4;

// Fortran-layout offsets.  s and w arrays share the plane (NI*NJ); u arrays
// have NI+1 points in x, v arrays NJ+1 rows.
__host__ __device__ __forceinline__ long iS(const DGrid &g, int i, int j, int k) {
  return (long)(i - g.ib) + (long)g.NI * ((long)(j - g.jb) + (long)g.NJ * (long)k);
}
__host__ __device__ __forceinline__ long iW(const DGrid &g, int i, int j, int k) { return iS(g, i, j, k); }
__host__ __device__ __forceinline__ long iU(const DGrid &g, int i, int j, int k) {
  return (long)(i - g.ib) + (long)(g.NI + 1) * ((long)(j - g.jb) + (long)g.NJ * (long)k);
}
__host__ __device__ __forceinline__ long iV(const DGrid &g, int i, int j, int k) {
  return (long)(i - g.ib) + (long)g.NI * ((long)(j - g.jb) + (long)(g.NJ + 1) * (long)k);
}
__host__ __device__ __forceinline__ long i2(const DGrid &g, int i, int j) {
  return (long)(i - g.ib) + (long)g.NI * (long)(j - g.jb);
}
__host__ __device__ __forceinline__ long nS(const DGrid &g) { return (long)g.NI * g.NJ * g.NK; }
__host__ __device__ __forceinline__ long nU(const DGrid &g) { return (long)(g.NI + 1) * g.NJ * g.NK; }
__host__ __device__ __forceinline__ long nV(const DGrid &g) { return (long)g.NI * (g.NJ + 1) * g.NK; }
__host__ __device__ __forceinline__ long nW(const DGrid &g) { return (long)g.NI * g.NJ * (g.NK + 1); }

#define LDG(p) __ldg(p)

// The physical point that the fills of a scalar copy to the halo point at n
// of 1..N along one direction (bc.F:180-518: periodic, open, or a wall's
// mirror image; a single row beyond the edge copies the edge in every
// non-periodic case).
__device__ __forceinline__ int bc_source(int n, int N, int lo, int hi) {
  if (n < 1) return lo == 1 ? n + N : lo == 2 ? 1 : 1 - n;
  if (n > N) return hi == 1 ? n - N : hi == 2 ? N : 2 * N + 1 - n;
  return n;
}

// brings the line of p into L2; the marching kernels call it for the levels ahead
__device__ __forceinline__ void prefetch_l2(const float *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---------------------------------------------------------------------
// Face values (binary32 arithmetic in the reference's evaluation order;
// adv_routines.F:5971-6205, 6331-6355).  The library is compiled with
// --fmad=false so that each product and sum rounds as the Fortran does.
// ---------------------------------------------------------------------
__device__ __forceinline__ float flx3(float s1, float s2, float s3) {
  return ((-1.0f / 6.0f) * s1 + (5.0f / 6.0f) * s2) + (2.0f / 6.0f) * s3;
}
__device__ __forceinline__ float flx5(float s1, float s2, float s3, float s4, float s5) {
  return ((((2.0f / 60.0f) * s1 + (-13.0f / 60.0f) * s2) + (47.0f / 60.0f) * s3) +
          (27.0f / 60.0f) * s4) + (-3.0f / 60.0f) * s5;
}

// WENO5 with Borges et al. (2008) weights.  Smoothness indicators in
// binary32 (as the Fortran evaluates them), weights and quotient in binary64.
//
// The reference (adv_routines.F:6166-6205) forms each weight with its own
// binary64 division, w_i = c_i (1 + min(1e30, tau/(b_i+weps))^2), and the
// face value as (w1 q1 + w2 q2 + w3 q3)/(w1 + w2 + w3) rounded to binary32
// (weno5_exact).  weno5_fast folds the three divisions into one over the common
// denominator d1^2 d2^2 d3^2.  The weights are positive and each has a
// relative error of a few units of the last binary64 place, so both binary64
// results lie within 17 such units, times A = (w1 |q1| + w2 |q2| + w3 |q3|) /
// (w1 + w2 + w3), of the exact weighted average: they differ by less than
// 2^-46 A.  Where the folded value v, in [2^E, 2^(E+1)), is within a factor
// 1024 of A, that is less than 2^17 units of its last place 2^(E-52); binary32
// rounding discards v's last 29 bits and changes where they are 2^28, so when
// they are farther than 2^17 from that, the reference's value rounds to the
// same binary32 number.  Otherwise (one face in two thousand, and values a
// thousand times smaller than their terms) v - 2^-46 A and v + 2^-46 A are both
// rounded: where they agree, the reference's value between them does too.  Where
// not (a tie to 14 digits, which the nominal weights make of neighbouring
// candidate values; a weight at its bound), weno5_fast returns NaN and its caller
// evaluates the face with weno5_exact, from the stencil where it lies, so that a
// kernel's main loop holds nothing for it.
//
// Products by 2, 4 and 0.25 are exact while they stay in the normal range, so
// fusing them with the addition that follows gives the binary32 value of the
// separate operations but for a subnormal indicator's last bit (2^-149).
// weno5_fast takes the fused form, and decides only where every denominator
// b_i + weps is above 2^-90: that bit is then far below the denominators' own
// rounding, and no product of theirs or of their squares leaves binary64's normal
// range.  Smaller denominators (weps = 0 or below 2^-90, in a field of tiny or
// equal values) go to weno5_exact, which rounds every operation.
// smoothness indicators and the three candidate values of a stencil
struct Weno5Terms { float f1, f2, f3, q1, q2, q3; };
template <bool FUSED>
__device__ __forceinline__ Weno5Terms weno5_terms(float s1, float s2, float s3, float s4, float s5) {
  const float c1312 = 13.0f / 12.0f;
  Weno5Terms w;
  float t, u;
  auto add = [](float c, float x, float y) { return FUSED ? __fmaf_rn(c, x, y) : c * x + y; };
  t = add(-2.0f, s2, s1) + s3; u = add(-4.0f, s2, s1) + 3.0f * s3;
  w.f1 = add(0.25f, u * u, c1312 * (t * t));
  t = add(-2.0f, s3, s2) + s4; u = s2 - s4;
  w.f2 = add(0.25f, u * u, c1312 * (t * t));
  t = add(-2.0f, s4, s3) + s5; u = add(-4.0f, s4, 3.0f * s3) + s5;
  w.f3 = add(0.25f, u * u, c1312 * (t * t));
  w.q1 = ((2.0f / 6.0f) * s1 + (-7.0f / 6.0f) * s2) + (11.0f / 6.0f) * s3;
  w.q2 = ((-1.0f / 6.0f) * s2 + (5.0f / 6.0f) * s3) + (2.0f / 6.0f) * s4;
  w.q3 = ((2.0f / 6.0f) * s3 + (5.0f / 6.0f) * s4) + (-1.0f / 6.0f) * s5;
  return w;
}
// n/d, d >= 0, rounded to nearest by Markstein's method (IBM J. Res. Dev. 34,
// 1990): Newton's iteration gives 1/d to the last place, and one correction of n/d
// by its exact residual rounds correctly, for d between 1e-60 and 1e200 and
// quotients and operands below 1e200.  Where that gives no number (d zero or
// infinite, n infinite, an operand not a number) the quotient is n times the
// approximate reciprocal 0 or infinity of d, or n's infinity.  Unlike the operator
// it has no subroutine for the extremes of the range, whose call would cost the
// main loop registers.
__device__ __forceinline__ double div_rn(double n, double d) {
  double y, y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(d));
  y = __fma_rn(y0, __fma_rn(-d, y0, 1.0), y0);
  y = __fma_rn(y, __fma_rn(-d, y, 1.0), y);
  y = __fma_rn(y, __fma_rn(-d, y, 1.0), y);
  const double q = n * y, r = __fma_rn(__fma_rn(-d, q, n), y, q);
  return r == r ? r : n * y0;
}
__device__ __forceinline__ float weno5_exact(float s1, float s2, float s3, float s4, float s5, double weps) {
  const Weno5Terms w = weno5_terms<false>(s1, s2, s3, s4, s5);
  if (w.q1 == 0.0f && w.q2 == 0.0f && w.q3 == 0.0f) return 0.0f;
  const double b1 = (double)w.f1, b2 = (double)w.f2, b3 = (double)w.f3;
  const double tau = fabs(b1 - b3);
  double r;
  r = fmin(1.0e30, div_rn(tau, b1 + weps)); const double w1 = (double)0.1f * (1.0 + r * r);
  r = fmin(1.0e30, div_rn(tau, b2 + weps)); const double w2 = (double)0.6f * (1.0 + r * r);
  r = fmin(1.0e30, div_rn(tau, b3 + weps)); const double w3 = (double)0.3f * (1.0 + r * r);
  const double num = (w1 * (double)w.q1 + w2 * (double)w.q2) + w3 * (double)w.q3;
  return (float)div_rn(num, (w1 + w2) + w3);
}
__device__ __forceinline__ float weno5_fast(float s1, float s2, float s3, float s4, float s5, double weps) {
  // a stencil of zeros, which fills most of a tracer's or a hydrometeor's field
  const int any = __float_as_int(s1) | __float_as_int(s2) | __float_as_int(s3) | __float_as_int(s4) | __float_as_int(s5);
  if ((any << 1) == 0) return 0.0f;
  const Weno5Terms w = weno5_terms<true>(s1, s2, s3, s4, s5);
  const double b1 = (double)w.f1, b2 = (double)w.f2, b3 = (double)w.f3;
  const double tau = fabs(b1 - b3);
  const double d1 = b1 + weps, d2 = b2 + weps, d3 = b3 + weps;
  const double tt = tau * tau, e1 = d1 * d1, e2 = d2 * d2, e3 = d3 * d3;
  const double a1 = (double)0.1f * (e1 + tt) * (e2 * e3);
  const double a2 = (double)0.6f * (e2 + tt) * (e1 * e3);
  const double a3 = (double)0.3f * (e3 + tt) * (e1 * e2);
  const double p1 = (double)w.q1, p2 = (double)w.q2, p3 = (double)w.q3;
  const double num = __fma_rn(a3, p3, __fma_rn(a2, p2, a1 * p1));
  const double A = __fma_rn(a3, fabs(p3), __fma_rn(a2, fabs(p2), a1 * fabs(p1)));   // times the denominator
  const double den = (a1 + a2) + a3;
  // num/den to a few units of the last place: Newton's iteration for 1/den from
  // the 20 bits of rcp.approx.ftz.f64 (once: 40 bits), then one correction of
  // the quotient by its residual; not a number where den has no normal reciprocal
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
  y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
  const double v0 = num * y, v = __fma_rn(__fma_rn(-den, v0, num), y, v0);
  const float f = (float)v;
  // v's last 29 bits against 2^28 -+ 2^17, without the bits above them
  const unsigned off = 8u * (unsigned)__double2loint(v) - 8u * ((1u << 28) - (1u << 17));
  // no weight reaches its bound 1e30 where tau < 2^98 (b_i + weps), by exponent,
  // and b_i + weps is above 2^-90; the floor 1.2e-35 keeps f a normal binary32 number
  const int ht = max(__double2hiint(tau) - (98 << 20), (1023 - 90) << 20);
  if (ht < __double2hiint(weps) && off > 8u << 18 && fabs(num) * 1024.0 >= A && fabsf(f) >= 1.2e-35f) return f;
  const double e = A * y * 0x1p-46;
  const float lo = (float)(v - e), hi = (float)(v + e);
  if (ht < __double2hiint((double)fminf(fminf(w.f1, w.f2), w.f3) + weps) && lo == hi &&
      __float_as_int(lo) == __float_as_int(hi))
    return f;
  return __int_as_float(0x7fffffff);
}
__device__ __forceinline__ float weno5(float s1, float s2, float s3, float s4, float s5, double weps) {
  const float f = weno5_fast(s1, s2, s3, s4, s5, weps);
  return f != f ? weno5_exact(s1, s2, s3, s4, s5, weps) : f;
}

__device__ __forceinline__ float upstrpd(float s1, float s2, float s3, double weps) {
  float dd = s2 - s1;
  float rr = (s3 - s2) / (copysignf((float)weps, dd) + dd);
  float phi = fmaxf(0.0f, fminf(rr, fminf((1.0f / 6.0f) + (2.0f / 6.0f) * rr, 1.0f)));
  return s2 + phi * (s2 - s1);
}

__device__ __forceinline__ float absmax5(float a, float b, float c, float d, float e) {
  return fmaxf(fmaxf(fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c)), fabsf(d)), fabsf(e));
}

// Optional extras of the scalar tile (k_advs_tile, update mode):
//  phix/phiy  learned face values of the horizontal faces (NaN: use WENO5),
//             indexed f = (k-1)*nfx*nfy + (j-1)*nfx + (i-1) with
//             nfx x nfy = (ni+1) x nj for x-faces and ni x (nj+1) for y-faces;
//  cap*       capture of the x/y face fluxes and face mass fluxes the
//             kernel used (u-/v-array layout), for building training targets.
struct TileExtras {
  const float *phix = nullptr, *phiy = nullptr;
  float *capfx = nullptr, *capfy = nullptr, *caprx = nullptr, *capry = nullptr;
};

// 6th-order horizontal diffusion inside the advection passes (idiff=1,
// difforder=6; adv.F:342-406, 1177-1236, 2115-2174, 3109-3170).  rho null:
// no diffusion.  ri is 1/rho as the scalar form uses it (rr of solve2; it
// may lag rho by one stage), coef = kdiff6/64/dt, mdiff the limiter.
struct Diff6 {
  const float *rho = nullptr, *ri = nullptr;
  float coef = 0.0f;
  int mdiff = 0;
};

// The difference stencil of a face between a(-1) and a(0), as the Fortran
// evaluates it: (10 (a0 - am1) - 5 (ap1 - am2)) + (ap2 - am3).
__device__ __forceinline__ float diff6_stencil(float am3, float am2, float am1, float a0, float ap1, float ap2) {
  return (10.0f * (a0 - am1) - 5.0f * (ap1 - am2)) + (ap2 - am3);
}
// the mdiff limiter: no flux against the local gradient
__device__ __forceinline__ float diff6_limit(float f, float a0, float am1, int mdiff) {
  return (mdiff == 1 && f * (a0 - am1) <= 0.0f) ? 0.0f : f;
}

// One advected field of the fused scalar pass of an RK stage (k_scal.cu).
struct ScalField {
  const float *s;               // stage input (full halo)
  const float *sbase;           // RK base value (tha, qa, pta)
  const float *ten1;            // fixed tendency (thten1, qten, ptten)
  float *snew;                  // stage output
  double weps;                  // WENO epsilon of the field (solve2.F:1391, 1472-1514, 1941)
  int sadd;                     // theta: advect th0(k) - 300 + s (solve2.F:1365-1372)
  int flush;                    // |snew| < smeps -> 0 (theta and moisture)
  int pdefweno;                 // pdef form of the vertical WENO (adv_routines.F:2386-2421)
};

// Liquid water of the stage set-up (ptype=1): the RK-stage input of each
// liquid species (at most two: Kessler's qc, qr) and the buoyancy array
// that the stage set-up writes for the w tendency (null without liquid).
struct LiquidIn {
  const float *q[2] = {nullptr, nullptr};
  int n = 0;
  float *b8 = nullptr;
};

// Inputs of the solve1 tendency initialisation and of calcener (k_misc.cu).
struct TendIn {
  int irdamp;
  float rdalpha;
  const float *tauh, *taus, *tauf, *uavg, *vavg, *thavg, *ua, *va, *wa, *tha;
  float *uten1, *vten1, *wten1, *thten1, *qten, *ptten;
  int nq;     // moisture + tracer arrays to zero (qten first, then ptten)
  int numq;
};
struct EnerIn {
  const float *zh, *rho, *ua, *va, *wa, *ppi, *tha, *qv, *ql, *qi, *vr;
  float lv1, ls1;
};

// Levels that a block of a marching tile kernel owns, kcmin to kcmax: the
// choice whose blocks, handed to `slots` resident blocks in launch order,
// finish first (a block costs its levels plus `over` for its first ones).
int tile_levels(long tiles, int nk, int slots, int over, int kcmin, int kcmax);

// Records a message for cm1g_last_error() and returns code (C++ linkage,
// not part of the C-ABI).
int report_error(int code, const char *msg);

// Per-kernel device timing (the library's counterpart of the reference's
// timestats, input.F:359-387).  When a profile is active every kernel launch
// site brackets its launch with a pair of CUDA events on the launch stream;
// the elapsed times are summed per kernel name when the profile is read.
struct Profile;
extern thread_local Profile *g_profile;
void prof_record(const char *name, cudaStream_t st, bool begin);

struct ProfScope {
  const char *name;
  cudaStream_t st;
  ProfScope(const char *n, cudaStream_t s) : name(n), st(s) { if (g_profile) prof_record(name, st, true); }
  ~ProfScope() { if (g_profile) prof_record(name, st, false); }
};

}  // namespace cm1g
