// k_face.cuh -- face values of the scalar passes, the spread of a tile's faces
// over its threads (FaceSlots) and the exchange of the positive-definite scheme,
// shared by the per-scalar tile (k_adv.cu) and the fused multi-scalar pass
// (k_scal.cu) so that both use the same binary32/binary64 operations.
#pragma once
#include "cm1g_common.cuh"

namespace cm1g {

// Face loop of the tiles: each thread owns face `tid` of each direction
// (none where tid is past the level's faces), and the faces past one per
// thread (NFX - NT x-faces, NFY - NT y-faces, when a level has more faces
// than the block has threads) go to the threads from warp 1 (x) and the
// warps after those (y), so that the second pass of the loop is spread over
// other warps than the first.  A block with one thread row more than the
// tile has cell rows has at most one face of each direction per thread.
template <int NT, int NFX, int NFY>
struct FaceSlots {
  static constexpr int EX = NFX > NT ? NFX - NT : 0, EY = NFY > NT ? NFY - NT : 0;
  static constexpr int X1 = 32;
  static constexpr int Y1 = 32 * (1 + (EX + 31) / 32);
  static_assert(X1 + EX <= NT && Y1 + EY <= NT, "the extra faces fit the block");
  // face index of slot q (0 or 1) of thread tid; >= NFX / NFY: none
  __device__ static __forceinline__ int x(int tid, int q) {
    return q == 0 ? (tid < NFX ? tid : NFX) : ((tid >= X1 && tid < X1 + EX) ? NT + tid - X1 : NFX);
  }
  __device__ static __forceinline__ int y(int tid, int q) {
    return q == 0 ? (tid < NFY ? tid : NFY) : ((tid >= Y1 && tid < Y1 + EY) ? NT + tid - Y1 : NFY);
  }
};

// vertical face flux at level kk from wv[d+3] = s(kk+d), d = -3..2, with the
// interpolation weights c1(kk), c2(kk) of the 2nd-order pieces given
__device__ __forceinline__ float zflux_core(const float *wv, float r, int kk, int nk, float c1k, float c2k, int weno,
                                            int pdefweno, double weps) {
  auto A = [&](int d) { return wv[d + 3]; };
  if (!weno) {
    if (kk >= 4 && kk <= nk - 2) {
      const bool up = (r >= 0.0f);
      return r * flx5(up ? A(-3) : A(2), up ? A(-2) : A(1), up ? A(-1) : A(0), up ? A(0) : A(-1), up ? A(1) : A(-2));
    }
    if (kk == 2) {
      if (r >= 0.0f) return r * (c1k * A(-1) + c2k * A(0));
      return r * flx3(A(1), A(0), A(-1));
    }
    if (kk == nk) {
      if (r >= 0.0f) return r * flx3(A(-2), A(-1), A(0));
      return r * (c1k * A(-1) + c2k * A(0));
    }
    if (kk == 3) {
      if (r >= 0.0f) return r * flx3(A(-2), A(-1), A(0));
      return r * flx5(A(2), A(1), A(0), A(-1), A(-2));
    }
    if (r >= 0.0f) return r * flx5(A(-3), A(-2), A(-1), A(0), A(1));
    return r * flx3(A(1), A(0), A(-1));
  }
  if (kk == 2) {
    if (r >= 0.0f) return r * (c1k * A(-1) + c2k * A(0));
    return r * upstrpd(A(1), A(0), A(-1), weps);
  }
  if (kk == nk) {
    if (r > 0.0f) return r * upstrpd(A(-2), A(-1), A(0), weps);
    return r * (c1k * A(-1) + c2k * A(0));
  }
  if (pdefweno == 1) {
    if (kk == 3 && r > 0.0f) return r * upstrpd(A(-2), A(-1), A(0), weps);
    if (kk == nk - 1 && r < 0.0f) return r * upstrpd(A(1), A(0), A(-1), weps);
    float s1, s2, s3, s4, s5;
    if (r >= 0.0f) { s1 = A(-3); s2 = A(-2); s3 = A(-1); s4 = A(0); s5 = A(1); }
    else { s1 = A(2); s2 = A(1); s3 = A(0); s4 = A(-1); s5 = A(-2); }
    return (absmax5(s1, s2, s3, s4, s5) > (float)weps) ? r * weno5(s1, s2, s3, s4, s5, weps) : 0.0f;
  }
  if (kk >= 4 && kk <= nk - 2) {
    // upwind-ordered stencil first, so a warp with both signs evaluates one WENO
    const bool up = (r >= 0.0f);
    return r * weno5(up ? A(-3) : A(2), up ? A(-2) : A(1), up ? A(-1) : A(0), up ? A(0) : A(-1), up ? A(1) : A(-2),
                     weps);
  }
  if (kk == 3) {
    if (r >= 0.0f) return r * upstrpd(A(-2), A(-1), A(0), weps);
    return r * weno5(A(2), A(1), A(0), A(-1), A(-2), weps);
  }
  if (r >= 0.0f) return r * weno5(A(-3), A(-2), A(-1), A(0), A(1), weps);
  return r * upstrpd(A(1), A(0), A(-1), weps);
}
__device__ __forceinline__ float zflux_win(const DGrid &g, const float *wv, float r, int kk, int weno, int pdefweno,
                                           double weps) {
  return zflux_core(wv, r, kk, g.nk, LDG(&g.c1[kk]), LDG(&g.c2[kk]), weno, pdefweno, weps);
}
// A face value in the reference's upwind order with the full 5-point stencil on
// both sides; NaN where weno5_fast leaves it undecided.  sm3..sp2 are the values
// around the face between sm1 and s0.  pdef: stencils below weps give 0
// (adv_routines.F:2386-2421).
__device__ __forceinline__ float face5(float r, float sm3, float sm2, float sm1, float s0, float sp1, float sp2, int weno,
                                       int pdef, double weps) {
  const bool up = (r >= 0.0f);
  const float s1 = up ? sm3 : sp2, s2 = up ? sm2 : sp1, s3 = up ? sm1 : s0, s4 = up ? s0 : sm1, s5 = up ? sp1 : sm2;
  if (!weno) return r * flx5(s1, s2, s3, s4, s5);
  if (pdef == 1 && !(absmax5(s1, s2, s3, s4, s5) > (float)weps)) return 0.0f;
  return r * weno5_fast(s1, s2, s3, s4, s5, weps);
}
// horizontal face flux, every value decided (weno5)
__device__ __forceinline__ float hflux5(float r, float sm3, float sm2, float sm1, float s0, float sp1, float sp2, int weno,
                                        int pdef, double weps) {
  const bool up = (r >= 0.0f);
  const float s1 = up ? sm3 : sp2, s2 = up ? sm2 : sp1, s3 = up ? sm1 : s0, s4 = up ? s0 : sm1, s5 = up ? sp1 : sm2;
  if (!weno) return r * flx5(s1, s2, s3, s4, s5);
  if (pdef == 1 && !(absmax5(s1, s2, s3, s4, s5) > (float)weps)) return 0.0f;
  return r * weno5(s1, s2, s3, s4, s5, weps);
}
// the same face with weno5_exact
__device__ __forceinline__ float face5_exact(float r, float sm3, float sm2, float sm1, float s0, float sp1, float sp2,
                                             double weps) {
  const bool up = (r >= 0.0f);
  return r * weno5_exact(up ? sm3 : sp2, up ? sm2 : sp1, up ? sm1 : s0, up ? s0 : sm1, up ? sp1 : sm2, weps);
}
// The vertical face at level kk (2..nk) of a column, wv[d+3] = s(kk+d): fz is
// face5's value, which the two lowest and the two highest faces replace where
// the 5-point stencil does not fit (zflux_core's cases).
__device__ __forceinline__ float zface_edge(float fz, const float *wv, float r, int kk, int nk, const float *c1,
                                            const float *c2, int weno, int pdefweno, double weps) {
  if (kk == 2 || kk == nk) {
    const bool lin = kk == 2 ? r >= 0.0f : weno ? !(r > 0.0f) : !(r >= 0.0f);
    if (lin) return r * (LDG(&c1[kk]) * wv[2] + LDG(&c2[kk]) * wv[3]);
  } else if (kk == 3) {
    if (!(weno && pdefweno == 1 ? r > 0.0f : r >= 0.0f)) return fz;
  } else {
    if (r >= 0.0f || (weno && pdefweno == 1 && !(r < 0.0f))) return fz;
  }
  const bool hi = kk == nk || kk == 3;   // upwind from below
  const float s1 = hi ? wv[1] : wv[4], s2 = hi ? wv[2] : wv[3], s3 = hi ? wv[3] : wv[2];
  return r * (weno ? upstrpd(s1, s2, s3, weps) : flx3(s1, s2, s3));
}

// Mass moved into point c by the pdef scatter of pdefx2/pdefy2/pdefz
// (pdef.F:158-174), gathered in the scatter's loop order: contribution from
// the lower neighbour, then the point itself, then the upper neighbour.
__device__ __forceinline__ void pdef_gather(float dm2, float dm1, float d0, float dp1, float dp2, float smeps, float *mass,
                                            bool *flag) {
  float m = 0.0f;
  bool f = false;
  if (dm1 < 0.0f) {  // the point below scatters: we are its upper neighbour
    float foo1 = fmaxf(0.0f, dm2), foo2 = fmaxf(0.0f, d0);
    if (foo1 + foo2 > smeps) {
      float foo3 = fmaxf(dm1, -(foo1 + foo2)) / (foo1 + foo2);
      m = m + foo2 * foo3;
      if (d0 > smeps) f = true;
    }
  }
  if (d0 < 0.0f) {
    float foo1 = fmaxf(0.0f, dm1), foo2 = fmaxf(0.0f, dp1);
    if (foo1 + foo2 > smeps) {
      float foo3 = fmaxf(d0, -(foo1 + foo2)) / (foo1 + foo2);
      m = m - (foo1 + foo2) * foo3;
      f = true;
    }
  }
  if (dp1 < 0.0f) {
    float foo1 = fmaxf(0.0f, d0), foo2 = fmaxf(0.0f, dp2);
    if (foo1 + foo2 > smeps) {
      float foo3 = fmaxf(dp1, -(foo1 + foo2)) / (foo1 + foo2);
      m = m + foo1 * foo3;
      if (d0 > smeps) f = true;
    }
  }
  *mass = m; *flag = f;
}

}  // namespace cm1g
