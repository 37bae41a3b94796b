// Pieces of the FP64 kernels (internal header): the RK stage, and the moist
// model's terms (moist_swm.f90) that ride in the shallow-water kernels of
// swm_k64.cu.  Included by units compiled with --fmad=false only, and in the
// reference's operation order.
#pragma once
#include "swm_common.cuh"
#include "swm_div.cuh"

namespace imodel {

// constants.f90:45 -- eps = epsilon(1.) (float epsilon)
constexpr double kEps = 1.1920928955078125e-07;

// ode_rk4, swm.f90:2647-2678.  dt is half the time step in stages 0 and 1: dt
// k / 2 and (dt / 2) k are the same rounding (a power of two), and acc + 2 k
// is one fused operation with an exact product.
__device__ __forceinline__ double rk_stage(int stage, double k, double yn, double *acc,
                                           double dt) {
  if (stage == 0) {
    *acc = k;
    return yn + dt * k;
  } else if (stage == 1) {
    *acc = __fma_rn(2.0, k, *acc);
    return yn + dt * k;
  } else if (stage == 2) {
    *acc = __fma_rn(2.0, k, *acc);
    return yn + dt * k;
  }
  return yn + div_by(dt * (*acc + k), 6.0, kSixth);
}

// Fortran max(0, x) / min(a, b) as std::max / std::min evaluate them
__device__ __forceinline__ double fmax0(double x) { return (0.0 < x) ? x : 0.0; }
__device__ __forceinline__ double fminq(double a, double b) { return (b < a) ? b : a; }

// in place of MoistArgs: the shallow-water kernels alone
struct NoMoist {};

// twice u q_e times d of edge e for every advanced tracer with advmtd = "trsk"
// (scalar_hx2ed + scalar_elem_product, divhx, and div_hx's product with the
// edge length, which both cells form alike up to the sign; "upw1" forms its
// fluxes at the cells)
__device__ __forceinline__ void moist_flux64(const DevMesh64 &M, const MoistArgs &A, int e) {
  if (A.upw1) return;
  const int ne = M.ne, v1 = M.e_v[e], v2 = M.e_v[ne + e];
  const double ue = A.u_in[e], dl = M.e_dleng[e];
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if ((A.active >> k) & 1)
      A.uphi[static_cast<size_t>(k) * ne + e] = ue * (A.q_in[k][v1] + A.q_in[k][v2]) * dl;
}

// the thermal momentum source (source, moist_swm.f90:1299-1315) added to the
// momentum tendency of edge e, and u's RK stage
__device__ __forceinline__ void moist_edge64(const DevMesh64 &M, const MoistArgs &A, int e,
                                             double tend) {
  const int v1 = M.e_v[e], v2 = M.e_v[M.ne + e];
  const double h1 = A.h_in[v1], h2 = A.h_in[v2];
  double g = h2 * A.q_in[0][v2] - h1 * A.q_in[0][v1];
  g = div_by(div_by(g, M.e_leng[e], M.e_rleng[e]), M.erad, M.rerad);
  const double hed = (h1 + h2) * 0.5;
  double gpi_oh = 0.0;
  if (fabs(hed) < kEps / 100000.0)
    atomicOr(A.flags, 1);
  else
    gpi_oh = g / hed;
  const double su = A.hgrav * gpi_oh + A.gthb[e];
  A.u_out[e] = rk_stage(A.stage, tend + su, A.yn_u[e], A.acc_u + e, A.dts);
}

// Cell i: the divergence of each advected tracer's flux (div_hx, or div_hx_upw1
// with the upwind fluxes formed here), with kSwm the condensation, evaporation
// and precipitation sources (source, :1317-1351), and the RK stages of h (with
// the mass tendency tend) and the tracers.
template <bool kSwm>
__device__ __forceinline__ void moist_cell64(const DevMesh64 &M, const MoistArgs &A, int i,
                                             double tend) {
  const int nv = M.nv, ne = M.ne;
  double hs[4] = {0.0, 0.0, 0.0, 0.0};
  if (kSwm) {
    A.h_out[i] = rk_stage(A.stage, tend, A.yn_h[i], A.acc_h + i, A.dts);
    const double hi = A.h_in[i];
    const double qs = A.q0ex[i] / ((hi + M.c_bt[i]) * M.grav);
    double gamma_v = 1.0 + kLscale * (20.0 * qs);
    gamma_v = 1.0 / gamma_v;
    const double qv = A.qv[i], qc = A.qc[i];
    const double r = gamma_v * (qv - qs);
    const double dqv = div_by(fmax0(r), A.dt, A.rdt);
    const double dqc = div_by(fminq(qc, fmax0(-r)), A.dt, A.rdt);
    const double dqr = div_by(fmax0(kGammaR * (qc - kQprecip)), A.dt, A.rdt);
    hs[1] = hi * (dqc - dqv);
    hs[2] = hi * (dqv - dqc - dqr);
    hs[3] = hi * dqr;
    hs[0] = hi * (kLscale * (dqv - dqc));
  }
  const int n = M.c_nnb[i];
  const double A_i = M.c_areag[i], rA = M.c_rareag[i];
  // the slots' edges with ttgout < 0 in bit 31 (unused slots: edge 0)
  uint32_t es[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) es[j] = M.c_eds[j * nv + i];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    if (!((A.active >> k) & 1)) continue;
    double d = 0.0;
    if (A.upw1) {
      // div_hx_upw1: c_sd = ttgout l_e, so (u c_sd) q is the reference's
      // ((ttgout u) l_e) q bit for bit; the cell's own value where the
      // flux leaves it (ttgout u > 0), the neighbour's where it enters
      for (int j = 0; j < n; ++j) {
        const int e = M.c_ed[j * nv + i];
        const double sd = M.c_sd[j * nv + i], ue = A.u_in[e];
        const double out = sd > 0.0 ? ue : -ue;
        // the neighbour across slot j: the other end of edge e (mesh%v(i)%nb(j))
        const int a = M.e_v[e], b = M.e_v[ne + e];
        const double qu = out > 0.0 ? A.q_in[k][i] : A.q_in[k][a == i ? b : a];
        d = d + ue * sd * qu;
      }
    } else {
      const double *uphi = A.uphi + static_cast<size_t>(k) * ne;
      double f[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const double x = uphi[es[j] & 0x7FFFFFFFu];
        f[j] = __hiloint2double(__double2hiint(x) ^ (es[j] & 0x80000000u), __double2loint(x));
      }
      d = f[0];
#pragma unroll
      for (int j = 1; j < 6; ++j)
        if (j < n) d = d + f[j];
      d = d * 0.5;
    }
    double t = -div_by(div_by(d, A_i, rA), M.erad, M.rerad);
    if (kSwm && k < 4) t = t + hs[k];
    A.q_out[k][i] = rk_stage(A.stage, t, A.q_yn[k][i], A.q_acc[k] + i, A.dts);
  }
}

}  // namespace imodel
