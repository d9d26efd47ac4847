// k_turb.cuh -- arguments of the Smagorinsky LES kernels (k_turb.cu).
#pragma once
#include "cm1g_common.cuh"

namespace cm1g {

constexpr int kTurbMaxScalars = 1 + 2 * 8;   // theta, up to 8 q arrays and 8 tracers

struct TurbArgs {
  float csm;                                  // Smagorinsky constant (uniform csm of turbsmag)
  float prinv;                                // 1/Prandtl number (turb.F:3421-3422)
  float cgs1, cgs2, cgs3, cgt1, cgt2, cgt3;   // rf extrapolation to the bottom and top w-levels
  int tconfig, bcturbs, bbc, tbc;
  const float *ua, *va, *wa, *rho, *tha;
  float *uten, *vten, *wten;
  // scalars of the tendencies: theta first (s = th0 - th0r + tha), then the
  // tracers; none when nsc is 0
  int nsc;
  const float *s[kTurbMaxScalars];
  float *sten[kTurbMaxScalars];
  float *kmh, *kmv;                           // eddy viscosities (w-shaped; the halo ring is written)
};

void launch_turbsmag(const DGrid &g, const TurbArgs &a, cudaStream_t st, int64_t *nl);

}  // namespace cm1g
