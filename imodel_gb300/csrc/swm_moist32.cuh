// FP32 sources of the moist shallow-water model (internal header), shared by
// its separate kernels (swm_moist.cu) and its fused stage (swm_stage32.cu).
#pragma once
#include "swm_k32_body.cuh"

namespace imodel {

// the thermal momentum source g/2 grad(h h theta) / h_e + g theta_e grad(b)
// (moist_swm.f90:1299-1315) of an edge from its cells' depth deviations and
// h theta; gr = 1 / (l erad), gthb the second term
__device__ __forceinline__ float thermal32(float hd1, float hd2, float Q1, float Q2, float h_ref,
                                           float gr, float grav, float gthb, int *flags) {
  const float h1 = h_ref + hd1, h2 = h_ref + hd2;
  const float g = ((hd2 - hd1) * (Q1 + Q2) * 0.5f + (Q2 - Q1) * (h1 + h2) * 0.5f) * gr;
  // scalar_hx2ed of h
  const float hed = h_ref + 0.5f * (hd1 + hd2);
  float gpi_oh = 0.0f;
  if (fabsf(hed) < 1.1920928955078125e-12f)
    atomicOr(flags, 1);
  else
    gpi_oh = g / hed;
  return (grav * 0.5f) * gpi_oh + gthb;
}

// condensation, evaporation and precipitation (source, moist_swm.f90:
// 1317-1351) at a cell of depth hi: the sources of h theta, h qv, h qc, h qr
__device__ __forceinline__ void sources32(float hi, float bt, float q0ex, float qv, float qc,
                                          float dt, float grav, float (&hs)[4]) {
  constexpr float L = static_cast<float>(kLscale);
  const float qs = q0ex / ((hi + bt) * grav);
  const float gamma_v = 1.0f / (1.0f + L * (20.0f * qs));
  const float r = gamma_v * (qv - qs);
  const float dqv = fmaxf(r, 0.0f) / dt;
  const float dqc = fminf(qc, fmaxf(-r, 0.0f)) / dt;
  const float dqr =
      fmaxf(static_cast<float>(kGammaR) * (qc - static_cast<float>(kQprecip)), 0.0f) / dt;
  hs[1] = hi * (dqc - dqv);
  hs[2] = hi * (dqv - dqc - dqr);
  hs[3] = hi * dqr;
  hs[0] = hi * (L * (dqv - dqc));
}

}  // namespace imodel
