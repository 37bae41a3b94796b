// Kernels of the moist shallow-water model (moist_swm.f90) that are not part of
// the shallow-water step's own: constants of a run, a tracer alone, qv, qc and
// qr after a step, and the FP32 model beside the FP32 step.  FP64: the other
// terms are in swm_k64.cuh.
//
// Compiled with --fmad=false and in the reference's operation order, so that
// the GPU equals the CPU oracle bit for bit.  The one transcendental of the
// sources, exp(20 theta) in qsat, is formed once on the host (theta keeps its
// initial value in the reference's RK4 path) and read here.
#include "swm_common.cuh"
#include "swm_k64.cuh"
#include "swm_moist32.cuh"

namespace imodel {
namespace {

// what the sources read that stays fixed in a run: g theta_e grad(b) of
// moist_swm.f90:1299-1315 at the edges, q0 exp(20 theta) of qsat at the cells
__global__ void __launch_bounds__(256) k_moist_consts(DevMesh64 M, const double *__restrict__ th,
                                                      double *__restrict__ ex20, double q0,
                                                      double *__restrict__ gthb) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < M.nv) ex20[e] = q0 * ex20[e];
  if (e >= M.ne) return;
  const int v1 = M.e_v[e], v2 = M.e_v[M.ne + e];
  double gb = M.c_bt[v2] - M.c_bt[v1];
  gb = gb / M.e_leng[e] / M.erad;
  const double th_ed = (th[v1] + th[v2]) * 0.5;
  gthb[e] = M.grav * (th_ed * gb);
}

// A tracer alone (test case 1: the flow stands still): its fluxes, then its
// cells; the shallow-water cases form both in the kernels of swm_k64.cu
__global__ void __launch_bounds__(256) k_moist_edge(DevMesh64 M, MoistArgs A) {
  after_prior<false>();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < M.ne) moist_flux64(M, A, e);
}
__global__ void __launch_bounds__(256) k_moist_cell(DevMesh64 M, MoistArgs A) {
  after_prior<false>();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < M.nv) moist_cell64<false>(M, A, i, 0.0);
}

// after a step: qv, qc, qr = h qv / h etc. (scalar_elem_divide, with its
// guard), the fields the next step's sources read; one reciprocal (rounded
// to nearest) serves the three divisions where it is normal
__global__ void k_moist_q(int nv, const double *__restrict__ h, const double *__restrict__ hqv,
                          const double *__restrict__ hqc, const double *__restrict__ hqr,
                          double *__restrict__ qv, double *__restrict__ qc,
                          double *__restrict__ qr, int *flags) {
  after_prior<false>(h, hqv, hqc, hqr, qv, qc, qr);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const double hi = h[i];
  if (fabs(hi) < kEps / 100000.0) {
    atomicOr(flags, 1);
    return;
  }
  const double r = fabs(hi) <= kRecipHigh ? 1.0 / hi : __longlong_as_double(0x7FF8000000000000LL);
  qv[i] = div_by(hqv[i], hi, r);
  qc[i] = div_by(hqc[i], hi, r);
  qr[i] = div_by(hqr[i], hi, r);
}

// ---- FP32 --------------------------------------------------------------------
// The same model beside the FP32 step (any of its variants, tendencies
// only): h is stored as h - h_ref, so h itself is h_ref + h_d where the
// sources and the thermal term need it; the gradient of h (h theta) is
// formed as
//   h2 Q2 - h1 Q1 = (h_d2 - h_d1) (Q1 + Q2) / 2 + (Q2 - Q1) (h1 + h2) / 2
// (exact in real arithmetic), which keeps the difference of the depths free
// of h_ref's rounding.  The divergences use the cells' folded coefficients
// c_div32 = ttgout l_e / (A erad), the gradients e_grad32 = 1 / (l erad).
// Each cell forms the tracer flux of its edges itself from its neighbour
// across the edge (c_nb): u_e (q_i + q_nb) / 2 with "trsk", the upwind
// value with "upw1"; the two cells of an edge form the same flux, since
// q_i + q_nb and q_nb + q_i round alike, so no flux array goes through
// memory.

// what the sources read that stays fixed in a run: g theta_e grad(b) at the
// edges, q0 exp(20 theta) at the cells
__global__ void __launch_bounds__(256) k_moist_consts32(DevMesh M, const float *__restrict__ th,
                                                        float *__restrict__ ex20, float q0,
                                                        float *__restrict__ gthb) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < M.nv) ex20[e] = q0 * ex20[e];
  if (e >= M.ne) return;
  const int v1 = M.e_v[e], v2 = M.e_v[M.ne + e];
  const float gb = (M.c_bt32[v2] - M.c_bt32[v1]) * M.e_grad32[e];
  const float th_ed = (th[v1] + th[v2]) * 0.5f;
  gthb[e] = static_cast<float>(M.grav) * (th_ed * gb);
}

// the thermal momentum source and u's RK stage (shallow-water cases only)
__global__ void __launch_bounds__(256) k_moist_edge32(DevMesh M, MoistArgs32 A) {
  after_prior<true>();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne;
  if (e >= ne) return;
  const int v1 = __ldg(&M.e_v[e]), v2 = __ldg(&M.e_v[ne + e]);
  const float gr = __ldg(&M.e_grad32[e]), grav = static_cast<float>(M.grav);
  const float su = thermal32(A.h_in[v1], A.h_in[v2], A.q_in[0][v1], A.q_in[0][v2], A.h_ref, gr,
                             grav, A.gthb[e], A.flags);
  const float momeq = A.tend_u[e] + su;
  A.u_out[e] = rk_stage32(A.stage, momeq, A.yn_u[e], A.acc_u + e, A.dt);
}

__global__ void __launch_bounds__(256) k_moist_cell32(DevMesh M, MoistArgs32 A) {
  after_prior<true>();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nv = M.nv;
  if (i >= nv) return;
  float hs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (A.swm) {
    A.h_out[i] = rk_stage32(A.stage, A.tend_h[i], A.yn_h[i], A.acc_h + i, A.dt);
    sources32(A.h_ref + A.h_in[i], __ldg(&M.c_bt32[i]), A.q0ex[i], A.qv[i], A.qc[i], A.dt,
              static_cast<float>(M.grav), hs);
  }
  // the cell's edges: the normal velocity times c_div32, and the neighbour
  const int n = M.c_nnb[i];
  float w[6];
  int nb[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    w[j] = 0.0f;
    nb[j] = i;
    if (j < n) {
      w[j] = A.u_in[__ldg(&M.c_ed[j * nv + i])] * __ldg(&M.c_div32[j * nv + i]);
      nb[j] = __ldg(&M.c_nb[j * nv + i]);
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    if (!((A.active >> k) & 1)) continue;
    const float *q = A.q_in[k];
    const float qi = q[i];
    float d = 0.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      if (j >= n) continue;
      const float qn = q[nb[j]];
      // "upw1": the cell's own value where the flux leaves it (w > 0)
      const float qf = A.upw1 ? (w[j] > 0.0f ? qi : qn) : (qi + qn) * 0.5f;
      d += w[j] * qf;
    }
    float t = -d;
    if (A.swm && k < 4) t = t + hs[k];
    A.q_out[k][i] = rk_stage32(A.stage, t, A.q_yn[k][i], A.q_acc[k] + i, A.dt);
  }
}

__global__ void k_moist_q32(int nv, const float *__restrict__ hd, float h_ref,
                            const float *__restrict__ hqv, const float *__restrict__ hqc,
                            const float *__restrict__ hqr, float *__restrict__ qv,
                            float *__restrict__ qc, float *__restrict__ qr, int *flags) {
  after_prior<true>(hd, hqv, hqc, hqr, qv, qc, qr);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const float hi = h_ref + hd[i];
  if (fabsf(hi) < 1.1920928955078125e-12f) {
    atomicOr(flags, 1);
    return;
  }
  qv[i] = hqv[i] / hi;
  qc[i] = hqc[i] / hi;
  qr[i] = hqr[i] / hi;
}

inline int nblocks(int n, int t) { return (n + t - 1) / t; }

}  // namespace

void launch_moist_stage32(const DevMesh &M, const MoistArgs32 &A, cudaStream_t s) {
  if (A.swm) launch_pdl(k_moist_edge32, nblocks(M.ne, 256), 256, s, M, A);
  launch_pdl(k_moist_cell32, nblocks(M.nv, 256), 256, s, M, A);
}

void launch_moist_q32(int nv, const float *hd, float h_ref, const float *hqv, const float *hqc,
                      const float *hqr, float *qv, float *qc, float *qr, int *flags,
                      cudaStream_t s) {
  launch_pdl(k_moist_q32, nblocks(nv, 256), 256, s, nv, hd, h_ref, hqv, hqc, hqr, qv, qc, qr,
             flags);
}

void launch_moist_consts(const DevMesh64 &M, const double *th, double *ex20, double q0,
                         double *gthb, cudaStream_t s) {
  // every cell has at least three edges on these grids, two cells an edge, so
  // ne >= nv; the larger count covers both either way
  const int n = M.ne > M.nv ? M.ne : M.nv;
  k_moist_consts<<<nblocks(n, 256), 256, 0, s>>>(M, th, ex20, q0, gthb);
}

void launch_moist_consts32(const DevMesh &M, const float *th, float *ex20, float q0, float *gthb,
                           cudaStream_t s) {
  const int n = M.ne > M.nv ? M.ne : M.nv;
  k_moist_consts32<<<nblocks(n, 256), 256, 0, s>>>(M, th, ex20, q0, gthb);
}

void launch_moist_tracer(const DevMesh64 &M, const MoistArgs &A, cudaStream_t s) {
  const int be = block64(M.ne), bc = block64(M.nv);
  launch_pdl(k_moist_edge, nblocks(M.ne, be), be, s, M, A);
  launch_pdl(k_moist_cell, nblocks(M.nv, bc), bc, s, M, A);
}

void launch_moist_q(int nv, const double *h, const double *hqv, const double *hqc,
                    const double *hqr, double *qv, double *qc, double *qr, int *flags,
                    cudaStream_t s) {
  launch_pdl(k_moist_q, nblocks(nv, 256), 256, s, nv, h, hqv, hqc, hqr, qv, qc, qr, flags);
}

}  // namespace imodel
