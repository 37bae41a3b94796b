// FP64 kernels in the reference's operation order, plus the layout
// permutations and the compensated FP64 integrals.
//
// This translation unit is compiled with --fmad=false: every product and sum
// below is rounded on its own, as in the Fortran built without contraction,
// so that the FP64 step reproduces the reference arithmetic of
// src/swm.f90:2416-2683 and src/swm_operators.f90 bit for bit.
#include <cmath>
#include <type_traits>

#include "imodel_swm.h"
#include "swm_common.cuh"
#include "swm_k64.cuh"

namespace imodel {
namespace {

// What bounds the FP64 step: GB300's FP64 pipe (2 operations per cycle and
// SM), not memory -- the kernels below are counted in FP64 operations.  Three
// things keep the count low without changing a bit of the results:
//  * divisions by what is known in advance (areas, lengths, the earth's
//    radius, 6) are three operations instead of about ten (div_by);
//  * factors of two are left out of the per-edge fields and put into
//    constants: uh2 = 2 u h_e = u (h_1 + h_2), q2 = 2 q_e, and the stencil's
//    d / 8 takes the product's 8 back (scaling by a power of two commutes
//    with rounding);
//  * products that both cells of an edge form alike are formed once per edge
//    (2 u h_e d and the kinetic-energy term) and added with the cell's sign;
//  * sums begin with their first term (0 + x is x but for the sign of a zero).

// Edge e's fluxes: uh2 = 2 u h_e (scalar_hx2ed :89-97, scalar_elem_product
// :1546), fe = {2 u h_e d, (l d / 4) u^2}
__device__ __forceinline__ void edge_flux64(const DevMesh64 &M, int e, const double *__restrict__ h,
                                            const double *__restrict__ u,
                                            double *__restrict__ uh2,
                                            double2 *__restrict__ fe) {
  const int ne = M.ne;
  const double ue = u[e];
  const double f = ue * (h[M.e_v[e]] + h[M.e_v[ne + e]]);
  uh2[e] = f;
  fe[e] = make_double2(f * M.e_dleng[e], M.e_kew[e] * (ue * ue));
}

// Blocks [0, nbt): vort_tr (:551-611) + scalar_hx2tr (:229-284) +
// scalar_elem_divide (:1579); the depth at the triangle by the scheme's
// interpolation (swm.f90:2459-2464): kite areas (trsk), barycentric weights
// of the circumcentre (bary, pxt16) or scalar_edtr2trcc of h_ed (:286-343,
// gass18, which also keeps eta and h_tr for the rhombus PV).  The blocks
// after: the edges' fluxes, which the next launch reads beside q.
template <class Moist>
__global__ void __launch_bounds__(256) k_tri64(DevMesh64 M, const double *__restrict__ h,
                                               const double *__restrict__ u,
                                               double *__restrict__ q_tr, int pv_on,
                                               int *flags, const double *__restrict__ kt,
                                               double *__restrict__ coefvort, int scheme,
                                               double *__restrict__ eta_t,
                                               double *__restrict__ h_trs,
                                               double *__restrict__ uh2,
                                               double2 *__restrict__ fe, int nbt, Moist Q) {
  after_prior<false>(h, u, q_tr, coefvort, eta_t, h_trs, uh2, fe);
  if (static_cast<int>(blockIdx.x) >= nbt) {
    const int e = (blockIdx.x - nbt) * blockDim.x + threadIdx.x;
    if (e >= M.ne) return;
    edge_flux64(M, e, h, u, uh2, fe);
    if constexpr (std::is_same<Moist, MoistArgs>::value) moist_flux64(M, Q, e);
    return;
  }
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = M.nt;
  if (t >= nt) return;
  double e = u[M.t_ed[t]] * M.t_lt[t];
#pragma unroll
  for (int s = 1; s < 3; ++s) e = e + u[M.t_ed[s * nt + t]] * M.t_lt[s * nt + t];
  const double A = M.t_areag[t], rA = M.t_rareag[t];
  e = div_by(div_by(e, A, rA), M.erad, M.rerad);
  // with diffusion on: rel_vort_tr(u) (:780-827) is this sum before f is
  // added; diffusion_ed's K_tr zeta
  if (coefvort) coefvort[t] = kt[t] * e;
  e = e + M.t_f[t];
  double ht = 0.0;
  if (scheme == IMODEL_SWM_PXT16) {
#pragma unroll
    for (int s = 0; s < 3; ++s) ht = ht + M.t_bary[s * nt + t] * h[M.t_v[s * nt + t]];
  } else if (scheme == IMODEL_SWM_GASS18) {
    const int ne = M.ne;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int ed = M.t_ed[s * nt + t];
      const double he = (h[M.e_v[ed]] + h[M.e_v[ne + ed]]) * 0.5;
      ht = ht + M.t_edarea[s * nt + t] * he;
    }
    ht = div_by(ht, A, rA);
    eta_t[t] = e;
    h_trs[t] = ht;
  } else {
    ht = M.t_kite[t] * h[M.t_v[t]];
#pragma unroll
    for (int s = 1; s < 3; ++s) ht = ht + M.t_kite[s * nt + t] * h[M.t_v[s * nt + t]];
    ht = div_by(ht, A, rA);
  }
  double q = 0.0;
  if (pv_on) {
    if (fabs(ht) < kEps / 100000.0)
      atomicOr(flags, 1);
    else
      q = e / ht;
  }
  q_tr[t] = q;
}

// proj_vec_sphere (smeshpack.f90:4419-4433): v - (v . p) p / |p|, with |p|
// and its reciprocal from the layout
__device__ __forceinline__ void proj_sphere(double &v0, double &v1, double &v2, double p0,
                                            double p1, double p2, double np, double rnp) {
  const double vp = v0 * p0 + v1 * p1 + v2 * p2;
  v0 = v0 - div_by(vp * p0, np, rnp);
  v1 = v1 - div_by(vp * p1, np, rnp);
  v2 = v2 - div_by(vp * p2, np, rnp);
}

// +-x by the sign of s (a sign flip on the integer pipe instead of a
// comparison and a product on the FP64 pipe)
__device__ __forceinline__ double sign_of(double s, double x) {
  return __hiloint2double(__double2hiint(x) ^ (__double2hiint(s) & 0x80000000),
                          __double2loint(x));
}

// x with its sign changed where bit 31 of es is set
__device__ __forceinline__ double flip(uint32_t es, double x) {
  return __hiloint2double(__double2hiint(x) ^ (es & 0x80000000u), __double2loint(x));
}

// grad_tr2ed(q_tr) (:1427-1463), the PV gradient across each edge
__global__ void __launch_bounds__(256) k_qgrad64(DevMesh64 M, const double *__restrict__ q_tr,
                                                 double *__restrict__ qge) {
  after_prior<false>(q_tr, qge);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne;
  if (e >= ne) return;
  const double g = M.e_sgtg[e] * (q_tr[M.e_sh[ne + e]] - q_tr[M.e_sh[e]]);
  qge[e] = div_by(div_by(g, M.e_dleng[e], M.e_rdleng[e]), M.erad, M.rerad);
}

// The two reconstructions apvm (:1465-1543) reads.  Blocks [0, nbt): the
// PV gradient at the triangles, vector_edtr2tr_perot (:408-452) of qge;
// dsign(1, tr%nr) = -tr%tg (smeshpack.f90:853-859), the sign of t_lt.
// The blocks after: the velocity at the cells, vector_edhx2hx_perot
// (:454-509, HTC, hx%areag); ttgout is the sign of c_sd.
__global__ void __launch_bounds__(256) k_apvm64(DevMesh64 M, const double *__restrict__ qge,
                                                const double *__restrict__ u,
                                                double *__restrict__ qg,
                                                double *__restrict__ vhx, int nbt) {
  after_prior<false>(qge, u, qg, vhx);
  const int ne = M.ne;
  if (static_cast<int>(blockIdx.x) < nbt) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nt = M.nt;
    if (t >= nt) return;
    const double c0 = M.t_c[t], c1 = M.t_c[nt + t], c2 = M.t_c[2 * nt + t];
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int ed = M.t_ed[s * nt + t];
      const double sg = sign_of(-M.t_lt[s * nt + t], qge[ed]);
      const double l = M.e_leng[ed];
      v0 = v0 + sg * (M.e_c[ed] - c0) * l;
      v1 = v1 + sg * (M.e_c[ne + ed] - c1) * l;
      v2 = v2 + sg * (M.e_c[2 * ne + ed] - c2) * l;
    }
    const double A = M.t_areag[t], rA = M.t_rareag[t];
    v0 = div_by(v0, A, rA);
    v1 = div_by(v1, A, rA);
    v2 = div_by(v2, A, rA);
    proj_sphere(v0, v1, v2, c0, c1, c2, M.t_nrm[t], M.t_rnrm[t]);
    qg[t] = v0;
    qg[nt + t] = v1;
    qg[2 * nt + t] = v2;
  } else {
    const int i = (blockIdx.x - nbt) * blockDim.x + threadIdx.x;
    const int nv = M.nv;
    if (i >= nv) return;
    const double p0 = M.c_p[i], p1 = M.c_p[nv + i], p2 = M.c_p[2 * nv + i];
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    const int n = M.c_nnb[i];
    for (int j = 0; j < n; ++j) {
      const int ed = M.c_ed[j * nv + i];
      const double su = sign_of(M.c_sd[j * nv + i], u[ed]);
      const double d = M.e_dleng[ed];
      v0 = v0 + su * (M.e_c[ed] - p0) * d;
      v1 = v1 + su * (M.e_c[ne + ed] - p1) * d;
      v2 = v2 + su * (M.e_c[2 * ne + ed] - p2) * d;
    }
    const double A = M.c_areag[i], rA = M.c_rareag[i];
    v0 = div_by(v0, A, rA);
    v1 = div_by(v1, A, rA);
    v2 = div_by(v2, A, rA);
    proj_sphere(v0, v1, v2, p0, p1, p2, M.c_nrm[i], M.c_rnrm[i]);
    vhx[i] = v0;
    vhx[nv + i] = v1;
    vhx[2 * nv + i] = v2;
  }
}

// Twice the PV of edge e: scalar_tr2ed (:124-176: the plain average for trsk,
// circumcentre-distance weights for bary) or, for gass18, scalar_elem_divide
// of the rhombus averages of eta and h_tr (swm.f90:2475-2480); with qg !=
// NULL the apvm correction of q_ed (:1495-1502), coef = pvspar dt
__device__ __forceinline__ double edge_pv2(const DevMesh64 &M, int e,
                                           const double *__restrict__ q_tr,
                                           const double *__restrict__ qg,
                                           const double *__restrict__ vhx, double coef,
                                           int scheme, const double *__restrict__ eta_t,
                                           const double *__restrict__ h_trs, int pv_on,
                                           int *flags) {
  const int ne = M.ne;
  const int t1 = M.e_sh[e], t2 = M.e_sh[ne + e];
  double q;
  if (scheme == IMODEL_SWM_PXT16) {
    const double d1 = M.e_dist[e], d2 = M.e_dist[ne + e];
    q = div_by(d2 * q_tr[t1] + d1 * q_tr[t2], M.e_dsum[e], M.e_rdsum[e]);
  } else if (scheme == IMODEL_SWM_GASS18) {
    const double a1 = M.t_areag[t1], a2 = M.t_areag[t2];
    const double eta_ed = (a1 * eta_t[t1] + a2 * eta_t[t2]) / (a1 + a2);
    const double h_rhb = (a1 * h_trs[t1] + a2 * h_trs[t2]) / (a1 + a2);
    q = 0.0;
    if (pv_on) {
      if (fabs(h_rhb) < kEps / 100000.0)
        atomicOr(flags, 1);
      else
        q = eta_ed / h_rhb;
    }
  } else {
    const double q2 = q_tr[t1] + q_tr[t2];
    if (!qg) return q2;
    q = 0.5 * q2;
  }
  if (qg) {
    const int nt = M.nt, nv = M.nv;
    const int c1 = M.e_v[e], c2 = M.e_v[ne + e];
    const double a0 = qg[t1] + qg[t2], a1 = qg[nt + t1] + qg[nt + t2],
                 a2 = qg[2 * nt + t1] + qg[2 * nt + t2];
    const double b0 = vhx[c1] + vhx[c2], b1 = vhx[nv + c1] + vhx[nv + c2],
                 b2 = vhx[2 * nv + c1] + vhx[2 * nv + c2];
    q = q - coef * (a0 * b0 + a1 * b1 + a2 * b2);
  }
  return q + q;
}

// Blocks [0, nbc): div_hx(uh) (:613-661), kinetic_energy_hx trsk
// (:1162-1171), Bernoulli potential (swm.f90:2533-2536) and the
// mass-equation RK stage.  The blocks after: q2, twice the edges' PV.  The
// two do not read each other; sharing a launch fills the chip on small grids.
template <class Moist>
__global__ void __launch_bounds__(256)
    k_cell64(DevMesh64 M, const double *__restrict__ h, const double *__restrict__ u,
             const double2 *__restrict__ fe, double *__restrict__ bern,
             const double *__restrict__ yn, double *__restrict__ acc, double *__restrict__ yout,
             double *__restrict__ tend, int stage, double dt, const double *__restrict__ kcv,
             double *__restrict__ coefdiv, int nbc, double *__restrict__ q2,
             const double *__restrict__ q_tr, const double *__restrict__ qg,
             const double *__restrict__ vhx, double coef, int scheme,
             const double *__restrict__ eta_t, const double *__restrict__ h_trs, int pv_on,
             int *flags, Moist Q) {
  if (static_cast<int>(blockIdx.x) >= nbc) {
    after_prior<false>(q2, q_tr, qg, vhx, eta_t, h_trs);
    const int e = (blockIdx.x - nbc) * blockDim.x + threadIdx.x;
    if (e < M.ne) q2[e] = edge_pv2(M, e, q_tr, qg, vhx, coef, scheme, eta_t, h_trs, pv_on, flags);
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nv = M.nv;
  if (i >= nv) return;
  const int n = M.c_nnb[i];
  const double A = M.c_areag[i], rA = M.c_rareag[i];
  // c_eds: the slot's edge with ttgout < 0 in bit 31 (unused slots: edge 0);
  // all slots are read before the sums, so that the loads wait once and not
  // slot by slot (a guarded loop took 7.6 us at level 5).  d is twice the sum
  uint32_t es[6];
  double2 f[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) es[j] = M.c_eds[j * nv + i];
  after_prior<false>(h, u, fe, bern, yn, acc, yout, tend, coefdiv);
#pragma unroll
  for (int j = 0; j < 6; ++j) f[j] = fe[es[j] & 0x7FFFFFFFu];
  double d = flip(es[0], f[0].x), k = f[0].y;
#pragma unroll
  for (int j = 1; j < 6; ++j)
    if (j < n) {
      d = d + flip(es[j], f[j].x);
      k = k + f[j].y;
    }
  // with diffusion on: div_hx(u) (:613-661), diffusion_ed's K div u
  if (coefdiv) {
    double du = 0.0;
    for (int j = 0; j < n; ++j) du = du + u[M.c_ed[j * nv + i]] * M.c_sd[j * nv + i];
    coefdiv[i] = kcv[i] * div_by(div_by(du, A, rA), M.erad, M.rerad);
  }
  const double divuh = div_by(div_by(d * 0.5, A, rA), M.erad, M.rerad);
  double ke;
  if (scheme == IMODEL_SWM_PXT16) {
    // kinetic_energy_hx, perhx branch (:1172-1173): half the squared
    // vector_edhx2hx_perot (:454-509, HTC) of u; c_off = ed%c%p - v%p
    double su[6], dl[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const int ed = static_cast<int>(es[j] & 0x7FFFFFFFu);
      su[j] = flip(es[j], u[ed]);
      dl[j] = M.e_dleng[ed];
    }
    double v0 = su[0] * M.c_off[i] * dl[0], v1 = su[0] * M.c_off[nv + i] * dl[0],
           v2 = su[0] * M.c_off[2 * nv + i] * dl[0];
#pragma unroll
    for (int j = 1; j < 6; ++j)
      if (j < n) {
        v0 = v0 + su[j] * M.c_off[(3 * j) * nv + i] * dl[j];
        v1 = v1 + su[j] * M.c_off[(3 * j + 1) * nv + i] * dl[j];
        v2 = v2 + su[j] * M.c_off[(3 * j + 2) * nv + i] * dl[j];
      }
    v0 = div_by(v0, A, rA);
    v1 = div_by(v1, A, rA);
    v2 = div_by(v2, A, rA);
    proj_sphere(v0, v1, v2, M.c_p[i], M.c_p[nv + i], M.c_p[2 * nv + i], M.c_nrm[i], M.c_rnrm[i]);
    ke = (v0 * v0 + v1 * v1 + v2 * v2) * 0.5;
  } else {
    ke = div_by(k, M.c_cellarea[i], M.c_rcellarea[i]);
  }
  bern[i] = M.grav * (h[i] + M.c_bt[i]) + ke;
  const double masseq = -divuh;
  if constexpr (std::is_same<Moist, MoistArgs>::value) {
    moist_cell64<true>(M, Q, i, masseq);
    return;
  }
  if (stage < 0)
    tend[i] = masseq;
  else
    yout[i] = rk_stage(stage, masseq, yn[i], acc + i, dt);
}

// the momentum tendency from its two terms (swm.f90:2578-2594) and the RK
// stage
template <class Moist = NoMoist>
__device__ __forceinline__ void edge_update64(const DevMesh64 &M, int e, double g, double q,
                                              const double *__restrict__ yn,
                                              double *__restrict__ acc,
                                              double *__restrict__ yout,
                                              double *__restrict__ tend, int stage, double dt,
                                              int mom_on, const double *__restrict__ dif1,
                                              const double *__restrict__ dif2,
                                              const Moist &Q = Moist{}) {
  double momeq = -g - q;
  // diffusion, then hyperdiffusion (swm.f90:2578-2589)
  if (dif1) momeq = momeq + dif1[e];
  if (dif2) momeq = momeq - dif2[e];
  if (!mom_on) momeq = 0.0;
  if constexpr (std::is_same<Moist, MoistArgs>::value)
    moist_edge64(M, Q, e, momeq);
  else if (stage < 0)
    tend[e] = momeq;
  else
    yout[e] = rk_stage(stage, momeq, yn[e], acc + e, dt);
}

// grad_ed (:511-548) + coriolis_ed TRSK (:1283-1308) and the momentum RK stage
template <class Moist>
__global__ void __launch_bounds__(256) k_edge64(DevMesh64 M, const double *__restrict__ bern,
                                                const double *__restrict__ uh2,
                                                const double *__restrict__ q2,
                                                const double *__restrict__ yn,
                                                double *__restrict__ acc,
                                                double *__restrict__ yout,
                                                double *__restrict__ tend, int stage,
                                                double dt, int mom_on,
                                                const double *__restrict__ dif1,
                                                const double *__restrict__ dif2,
                                                const int32_t *__restrict__ stq, Moist Q) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne;
  if (e >= ne) return;
  const double l = M.e_leng[e], rl = M.e_rleng[e];
  const int v1 = M.e_v[e], v2 = M.e_v[ne + e];
  const int ns = M.e_nst[e];
  // slots past ns hold edge 0 and weight 0 and are left out of the sum; all
  // are read at once, the fixed ones before the wait for the cells' kernel
  int k[kMaxStencil];
  double w[kMaxStencil], d8[kMaxStencil];
#pragma unroll
  for (int s = 0; s < kMaxStencil; ++s) {
    k[s] = M.e_stk[s * ne + e];
    w[s] = M.e_stw[s * ne + e];
  }
#pragma unroll
  for (int s = 0; s < kMaxStencil; ++s) d8[s] = M.e_d8[k[s]];
  after_prior<false>(bern, uh2, q2, yn, acc, yout, tend, dif1, dif2);
  double g = bern[v2] - bern[v1];
  g = div_by(div_by(g, l, rl), M.erad, M.rerad);
  const double qe = q2[e];
  double q = 0.0;
  // per slot: F_k (q_e + q_k) / 2 d_k w, in that order; 2 F, 2 q and d / 8
#pragma unroll
  for (int s = 0; s < kMaxStencil; ++s) {
    // gass18 (:1378-1410): the PV of the edge connecting e and k when there
    // is one (stq != NULL), else the TRSK average
    const int c3 = stq ? stq[s * ne + e] : -1;
    const double qs = c3 >= 0 ? q2[c3] + q2[c3] : qe + q2[k[s]];
    const double t = uh2[k[s]] * qs * d8[s] * w[s];
    if (s < ns) q = s == 0 ? t : q + t;
  }
  q = div_by(q, l, rl);
  edge_update64(M, e, g, q, yn, acc, yout, tend, stage, dt, mom_on, dif1, dif2, Q);
}

// dtred: vector_edhx2tr_perot (:345-406, HTC) of uh at the triangle
// circumcentres, cross(tr%c, v) / tr%areag, times q_tr (vector_elem_product,
// :1617-1649); signcor = dsign(1, tr%tg) is the sign of t_lt
__global__ void __launch_bounds__(256) k_vhq64(DevMesh64 M, const double *__restrict__ uh2,
                                               const double *__restrict__ q_tr,
                                               double *__restrict__ vhq) {
  after_prior<false>(uh2, q_tr, vhq);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = M.nt, ne = M.ne;
  if (t >= nt) return;
  const double c0 = M.t_c[t], c1 = M.t_c[nt + t], c2 = M.t_c[2 * nt + t];
  double v0 = 0.0, v1 = 0.0, v2 = 0.0;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int ed = M.t_ed[s * nt + t];
    const double su = sign_of(M.t_lt[s * nt + t], uh2[ed]) * 0.5;
    const double l = M.e_leng[ed];
    v0 = v0 + su * (M.e_c[ed] - c0) * l;
    v1 = v1 + su * (M.e_c[ne + ed] - c1) * l;
    v2 = v2 + su * (M.e_c[2 * ne + ed] - c2) * l;
  }
  const double w0 = c1 * v2 - c2 * v1, w1 = c2 * v0 - c0 * v2, w2 = c0 * v1 - c1 * v0;
  const double A = M.t_areag[t], rA = M.t_rareag[t], q = q_tr[t];
  vhq[t] = div_by(w0, A, rA) * q;
  vhq[nt + t] = div_by(w1, A, rA) * q;
  vhq[2 * nt + t] = div_by(w2, A, rA) * q;
}

// grad_ed (:511-548) + coriolis_ed's dtred (:1310-1329) or pered
// (:1330-1377) branch, HTC, and the momentum RK stage
__global__ void __launch_bounds__(256) k_edge64r(DevMesh64 M, const double *__restrict__ bern,
                                                 const double *__restrict__ uh2,
                                                 const double *__restrict__ q2,
                                                 const double *__restrict__ vhq,
                                                 const double *__restrict__ yn,
                                                 double *__restrict__ acc,
                                                 double *__restrict__ yout,
                                                 double *__restrict__ tend, int stage,
                                                 double dt, int mom_on,
                                                 const double *__restrict__ dif1,
                                                 const double *__restrict__ dif2, int scheme) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne, nv = M.nv, nt = M.nt;
  if (e >= ne) return;
  after_prior<false>(bern, uh2, q2, vhq, yn, acc, yout, tend, dif1, dif2);
  double g = bern[M.e_v[ne + e]] - bern[M.e_v[e]];
  g = div_by(div_by(g, M.e_leng[e], M.e_rleng[e]), M.erad, M.rerad);
  double v0, v1, v2;
  if (scheme == IMODEL_SWM_DTRED) {
    // the dual-triangle reconstructions of the edge's two triangles,
    // weighted by the other triangle's circumcentre distance
    const int k1 = M.e_sh[e], k2 = M.e_sh[ne + e];
    const double d1 = M.e_dist[e], d2 = M.e_dist[ne + e];
    const double ds = M.e_dsum[e], rds = M.e_rdsum[e];
    v0 = div_by(d2 * vhq[k1] + d1 * vhq[k2], ds, rds);
    v1 = div_by(d2 * vhq[nt + k1] + d1 * vhq[nt + k2], ds, rds);
    v2 = div_by(d2 * vhq[2 * nt + k1] + d1 * vhq[2 * nt + k2], ds, rds);
  } else {
    // pered: at each of the edge's cells the Perot reconstruction of
    // uh (q_e + q_k) / 2 over the cell's edges, projected on the tangent
    // plane; twice their average (0.5 x + 0.5 y and 0.5 (x + y) are the same
    // rounding, and the projection is linear in powers of two)
    const double qe = q2[e];
    double vc[2][3];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = M.e_v[i * ne + e];
      const int n = M.c_nnb[c];
      double f[6], d[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const uint32_t es = M.c_eds[j * nv + c];
        const int l2 = static_cast<int>(es & 0x7FFFFFFFu);
        f[j] = flip(es, uh2[l2]) * (qe + q2[l2]);
        d[j] = M.e_d8[l2];
      }
      double a0 = f[0] * M.c_off[c] * d[0], a1 = f[0] * M.c_off[nv + c] * d[0],
             a2 = f[0] * M.c_off[2 * nv + c] * d[0];
#pragma unroll
      for (int j = 1; j < 6; ++j)
        if (j < n) {
          a0 = a0 + f[j] * M.c_off[(3 * j) * nv + c] * d[j];
          a1 = a1 + f[j] * M.c_off[(3 * j + 1) * nv + c] * d[j];
          a2 = a2 + f[j] * M.c_off[(3 * j + 2) * nv + c] * d[j];
        }
      const double A = M.c_areag[c], rA = M.c_rareag[c];
      a0 = div_by(a0, A, rA);
      a1 = div_by(a1, A, rA);
      a2 = div_by(a2, A, rA);
      proj_sphere(a0, a1, a2, M.c_p[c], M.c_p[nv + c], M.c_p[2 * nv + c], M.c_nrm[c],
                  M.c_rnrm[c]);
      vc[i][0] = a0;
      vc[i][1] = a1;
      vc[i][2] = a2;
    }
    v0 = vc[0][0] + vc[1][0];
    v1 = vc[0][1] + vc[1][1];
    v2 = vc[0][2] + vc[1][2];
  }
  proj_sphere(v0, v1, v2, M.e_c[e], M.e_c[ne + e], M.e_c[2 * ne + e], M.e_nrm[e], M.e_rnrm[e]);
  double q = -(v0 * M.e_nr[e] + v1 * M.e_nr[ne + e] + v2 * M.e_nr[2 * ne + e]);
  if (scheme != IMODEL_SWM_DTRED) q = 0.5 * q;
  edge_update64(M, e, g, q, yn, acc, yout, tend, stage, dt, mom_on, dif1, dif2);
}

// diffusion_ed (swm_operators.f90:855-895), first half: coefdiv = K
// div_hx(x) at the cells (blocks [0, nbc)), coefvort = K_tr rel_vort_tr(x)
// at the triangles (the blocks after), HTC branches of div_hx (:613-661) and
// rel_vort_tr (:780-827)
__global__ void __launch_bounds__(256) k_difcv64(DevMesh64 M, const double *__restrict__ x,
                                                 const double *__restrict__ kcv,
                                                 const double *__restrict__ kt,
                                                 double *__restrict__ coefdiv,
                                                 double *__restrict__ coefvort, int nbc) {
  after_prior<false>(x, coefdiv, coefvort);
  if (static_cast<int>(blockIdx.x) < nbc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nv = M.nv;
    if (i >= nv) return;
    const int n = M.c_nnb[i];
    double d = 0.0;
    for (int j = 0; j < n; ++j) d = d + x[M.c_ed[j * nv + i]] * M.c_sd[j * nv + i];
    const double divx = div_by(div_by(d, M.c_areag[i], M.c_rareag[i]), M.erad, M.rerad);
    coefdiv[i] = kcv[i] * divx;
  } else {
    const int t = (blockIdx.x - nbc) * blockDim.x + threadIdx.x;
    const int nt = M.nt;
    if (t >= nt) return;
    double z = 0.0;
#pragma unroll
    for (int s = 0; s < 3; ++s) z = z + x[M.t_ed[s * nt + t]] * M.t_lt[s * nt + t];
    z = div_by(div_by(z, M.t_areag[t], M.t_rareag[t]), M.erad, M.rerad);
    coefvort[t] = kt[t] * z;
  }
}

// second half: lap = grad_ed(coefdiv) - grad_ed_tg(coefvort) (grad_ed
// :511-548, grad_ed_tg :738-777, HTC)
__global__ void __launch_bounds__(256) k_diflap64(DevMesh64 M, const double *__restrict__ coefdiv,
                                                  const double *__restrict__ coefvort,
                                                  double *__restrict__ lap) {
  after_prior<false>(coefdiv, coefvort, lap);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne;
  if (e >= ne) return;
  double g = coefdiv[M.e_v[ne + e]] - coefdiv[M.e_v[e]];
  g = div_by(div_by(g, M.e_leng[e], M.e_rleng[e]), M.erad, M.rerad);
  double gt = M.e_sgtg[e] * (coefvort[M.e_sh[ne + e]] - coefvort[M.e_sh[e]]);
  gt = div_by(gt, M.e_dlerad[e], M.e_rdlerad[e]);
  lap[e] = g - gt;
}

// the coefficients swm.f90:169-205 sets: at the cells the coefficient field
// kf (device order; NULL: the constant k), at the triangles its
// scalar_hx2tr (:258-263); both then sqrt for hyperdiffusion
__global__ void k_dif_coefs(DevMesh M, const double *__restrict__ kf, double k, int take_sqrt,
                            double *__restrict__ kc64, float *__restrict__ kc32,
                            double *__restrict__ kt64, float *__restrict__ kt32, int nbc) {
  if (static_cast<int>(blockIdx.x) < nbc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.nv) return;
    double f = kf ? kf[i] : k;
    if (take_sqrt) f = sqrt(f);
    kc64[i] = f;
    if (kc32) kc32[i] = static_cast<float>(f);
  } else {
    const int t = (blockIdx.x - nbc) * blockDim.x + threadIdx.x;
    const int nt = M.nt;
    if (t >= nt) return;
    double f = 0.0;
#pragma unroll
    for (int s = 0; s < 3; ++s) f = f + M.t_kite[s * nt + t] * (kf ? kf[M.t_v[s * nt + t]] : k);
    f = f / M.t_areag[t];
    if (take_sqrt) f = sqrt(f);
    kt64[t] = f;
    if (kt32) kt32[t] = static_cast<float>(f);
  }
}

// RN(1 / b) for div_by, NaN where its three operations could leave the
// normal range
__device__ __forceinline__ double recip(double b) {
  const double a = fabs(b);
  return a >= kRecipLow && a <= kRecipHigh ? 1.0 / b : __longlong_as_double(0x7FF8000000000000LL);
}
__device__ __forceinline__ double norm3(const double *p, int n, int i) {
  const double p0 = p[i], p1 = p[n + i], p2 = p[2 * n + i];
  return sqrt(p0 * p0 + p1 * p1 + p2 * p2);
}

// the derived constants of DevMesh (entity i of each kind)
__global__ void __launch_bounds__(256) k_consts64(DevMesh64 M) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nv = M.nv, ne = M.ne, nt = M.nt;
  auto w = [](const double *p, int k, double v) { const_cast<double *>(p)[k] = v; };
  if (i < nv) {
    w(M.c_rareag, i, recip(M.c_areag[i]));
    w(M.c_rcellarea, i, recip(M.c_cellarea[i]));
    for (int j = 0; j < 6; ++j) {
      const int k = j * nv + i;
      const bool live = j < M.c_nnb[i];
      const int e = live ? M.c_ed[k] : 0;
      // c_sd = ttgout d
      const bool neg = live && (M.c_sd[k] < 0.0) != (M.e_dleng[e] < 0.0);
      const_cast<uint32_t *>(M.c_eds)[k] = static_cast<uint32_t>(e) | (neg ? 0x80000000u : 0u);
      if (M.c_off)
        for (int c = 0; c < 3; ++c)
          w(M.c_off, (3 * j + c) * nv + i, live ? M.e_c[c * ne + e] - M.c_p[c * nv + i] : 0.0);
    }
    if (M.c_nrm) {
      w(M.c_nrm, i, norm3(M.c_p, nv, i));
      w(M.c_rnrm, i, recip(M.c_nrm[i]));
    }
  }
  if (i < nt) {
    w(M.t_rareag, i, recip(M.t_areag[i]));
    if (M.t_nrm) {
      w(M.t_nrm, i, norm3(M.t_c, nt, i));
      w(M.t_rnrm, i, recip(M.t_nrm[i]));
    }
  }
  if (i < ne) {
    const double d = M.e_dleng[i], dr = d * M.erad;
    w(M.e_rleng, i, recip(M.e_leng[i]));
    w(M.e_rdleng, i, recip(d));
    w(M.e_d8, i, d * 0.125);
    w(M.e_dlerad, i, dr);
    w(M.e_rdlerad, i, recip(dr));
    if (M.e_nrm) {
      w(M.e_nrm, i, norm3(M.e_c, ne, i));
      w(M.e_rnrm, i, recip(M.e_nrm[i]));
    }
    if (M.e_dsum) {
      const double ds = M.e_dist[i] + M.e_dist[ne + i];
      w(M.e_dsum, i, ds);
      w(M.e_rdsum, i, recip(ds));
    }
  }
}

template <class T>
__global__ void k_gather_in(int n, const int32_t *__restrict__ n2o, const double *__restrict__ src,
                            T *__restrict__ dst, double shift) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = static_cast<T>(src[n2o[i]] - shift);
}

// scatter back to reference order; bit 1 of *flags marks a NaN/Inf value
template <class T>
__global__ void k_scatter_out(int n, const int32_t *__restrict__ n2o, const T *__restrict__ src,
                              double *__restrict__ dst, double shift, int *flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const double v = static_cast<double>(src[i]) + shift;
    dst[n2o[i]] = v;
    if (flags && !isfinite(v)) atomicOr(flags, 2);
  }
}

// j runs over the reference order (h, then u), so that the host arrays are read
// (or written) in order; the device side takes the permutation
template <class T>
__global__ void k_load_host(HostMap N, const double *__restrict__ h, const double *__restrict__ u,
                            HostTo<T> to_h, HostTo<T> to_u, double shift) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const bool cell = j < N.nv;
  if (j >= N.nv + N.ne) return;
  const int k = cell ? j : j - N.nv;
  const int i = cell ? N.cell[k] : N.edge[k];
  // the caller's arrays may be what the work in front writes
  after_prior<true>(h, u);
  const T v = static_cast<T>(cell ? h[k] - shift : u[k]);
  const HostTo<T> to = cell ? to_h : to_u;
  if (to.yn) to.yn[i] = v;
  to.ya[i] = v;
  if (to.ck) to.ck[i] = v;
}

template <class T>
__global__ void k_store_host(HostMap N, const T *__restrict__ src_h, const T *__restrict__ src_u,
                             double *__restrict__ h, double *__restrict__ u, double shift,
                             int *flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const bool cell = j < N.nv;
  if (j >= N.nv + N.ne) return;
  const int k = cell ? j : j - N.nv;
  const int i = cell ? N.cell[k] : N.edge[k];
  after_prior<true>(src_h, src_u, h, u);
  const double v = cell ? static_cast<double>(src_h[i]) + shift : static_cast<double>(src_u[i]);
  (cell ? h : u)[k] = v;
  if (flags && !isfinite(v)) atomicOr(flags, 2);
}

__global__ void k_take_flags(int *flags, int *host) {
  after_prior<true>(flags, host);
  *host = *flags;
  *flags = 0;
}

// vecrecon_trsk_tg, interpack.f90:3852-3976 (var%pos == 6)
__global__ void k_trsk_tangent(DevMesh M, const double *__restrict__ u, double *__restrict__ utg) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = M.ne;
  if (e >= ne) return;
  const int ns = M.e_nst[e];
  double t = 0.0;
  for (int s = 0; s < ns; ++s) {
    const int k = M.e_stk[s * ne + e];
    t = t + u[k] * M.e_dleng[k] * M.e_stw[s * ne + e];
  }
  utg[e] = -t / M.e_leng[e];
}

// ---- compensated summation (Neumaier) -------------------------------------
struct KSum {
  double s, c;
  __device__ void add(double x) {
    const double t = s + x;
    if (fabs(s) >= fabs(x))
      c = c + ((s - t) + x);
    else
      c = c + ((x - t) + s);
    s = t;
  }
  __device__ void merge(const KSum &o) {
    add(o.s);
    c = c + o.c;
  }
};

template <int NQ>
__device__ void block_reduce_store(KSum (&acc)[NQ], double *__restrict__ scratch) {
  // warp level: plain sums of the sums and of the compensations (32 terms,
  // error ~1e-15 relative; FP64 operations are slow on this GPU, and a
  // Neumaier merge costs four times a plain add)
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    for (int off = 16; off > 0; off >>= 1) {
      acc[q].s += __shfl_down_sync(0xffffffffu, acc[q].s, off);
      acc[q].c += __shfl_down_sync(0xffffffffu, acc[q].c, off);
    }
  }
  __shared__ double sh[kRedThreads / 32][NQ][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      sh[warp][q][0] = acc[q].s;
      sh[warp][q][1] = acc[q].c;
    }
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x;
    KSum t{0.0, 0.0};
    for (int w = 0; w < kRedThreads / 32; ++w) {
      KSum o{sh[w][q][0], sh[w][q][1]};
      t.merge(o);
    }
    scratch[(q * gridDim.x + blockIdx.x) * 2] = t.s;
    scratch[(q * gridDim.x + blockIdx.x) * 2 + 1] = t.c;
  }
}

// one block: quantity q summed over nblk partials; "max" quantities use max
__global__ void k_finalize(const double *__restrict__ scratch, int nblk, int nq,
                           unsigned maxmask, double *__restrict__ result) {
  // one block per quantity; the partials are combined as a tree (a few
  // dependent compensated merges per thread, then 5 shuffle levels per warp
  // and 3 across the warps) rather than by one thread in a row: FP64
  // operations have a long latency on this GPU
  const int q = blockIdx.x;
  after_prior<true>(scratch, result);
  if (q >= nq) return;
  static_assert(kRedThreads == 256, "8 warps per block");
  __shared__ double ss[8], sc[8];
  const bool is_max = (maxmask >> q) & 1u;
  KSum a{0.0, 0.0};
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    const double s = scratch[(q * nblk + b) * 2], c = scratch[(q * nblk + b) * 2 + 1];
    if (is_max) {
      a.s = fmax(a.s, s);
    } else {
      KSum o{s, c};
      a.merge(o);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int level = 0; level < 2; ++level) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      KSum o{__shfl_down_sync(0xffffffffu, a.s, off), __shfl_down_sync(0xffffffffu, a.c, off)};
      if (is_max)
        a.s = fmax(a.s, o.s);
      else
        a.merge(o);
    }
    if (level == 1) break;
    if (lane == 0) {
      ss[warp] = a.s;
      sc[warp] = a.c;
    }
    __syncthreads();
    if (warp != 0) return;
    a = lane < 8 ? KSum{ss[lane], sc[lane]} : KSum{0.0, 0.0};
  }
  if (threadIdx.x == 0) result[q] = is_max ? a.s : a.s + a.c;
}

// a / b for the diagnostics: FP64 division is slow on GB300's FP64 pipe, so
// the reciprocal starts from the FP32 one (relative error < 2^-22) and takes
// two Newton-Raphson steps r <- r (2 - b r), which square the error each
// (< 2^-44, then below FP64 rounding); b must be a normal FP32-range number
// (areas, depths)
__device__ __forceinline__ double diag_div(double a, double b) {
  double r = static_cast<double>(__frcp_rn(static_cast<float>(b)));
  r = r * (2.0 - b * r);
  r = r * (2.0 - b * r);
  return a * r;
}

// calc_energies (swm.f90:2686-2752), sumf_areas (:3394), potential enstrophy,
// RMS divergence of the last stage input (hs, us), NaN scan.  FULL = false
// computes the two energies only (the learned correction's drift guard).
// Each thread sums its few dozen terms in plain FP64 (relative error ~1e-14);
// threads, warps, blocks and the grid are combined with Neumaier-compensated
// sums.
template <class T, bool FULL>
__global__ void __launch_bounds__(kRedThreads) k_diag(DevMesh M, const T *__restrict__ h,
                                                      const T *__restrict__ u,
                                                      const T *__restrict__ hs,
                                                      const T *__restrict__ us,
                                                      double h_ref,
                                                      double *__restrict__ scratch) {
  double part[kDiagQ];
#pragma unroll
  for (int q = 0; q < kDiagQ; ++q) part[q] = 0.0;
  const int stride = gridDim.x * blockDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const double g = M.grav, erad = M.erad;
  double maxdiv = 0.0, umax = 0.0;
  double nan = 0.0;
  if (!FULL) {
    // energies for the learned correction's drift check: terms and each
    // thread's few dozen-term sums in FP32 (the check compares with a value
    // computed the same way, against a bound of 1e-3; FP64 operations are
    // slow on this GPU), the thread sums merged in FP64
    // (FP32 handles read FP32 copies of the weights: even the conversions
    // from FP64 would load the FP64 pipe)
    constexpr bool f32 = sizeof(T) == sizeof(float);
    const float gf = static_cast<float>(g), hr = static_cast<float>(h_ref);
    float pe = 0.0f, ke = 0.0f, um = 0.0f;
    for (int i = tid; i < M.nv; i += stride) {
      const float hi = static_cast<float>(h[i]) + hr;
      if (!isfinite(hi)) nan = 1.0;
      const float A = f32 ? M.c_area32[i] : static_cast<float>(M.c_areag[i]);
      const float b = f32 ? M.c_bt32[i] : static_cast<float>(M.c_bt[i]);
      pe += A * gf * hi * (hi * 0.5f + b);
    }
    for (int e = tid; e < M.ne; e += stride) {
      const float ue = static_cast<float>(u[e]);
      if (!isfinite(ue)) nan = 1.0;
      um = fmaxf(um, fabsf(ue));
      const float he = (static_cast<float>(hs[M.e_v[e]]) +
                        static_cast<float>(hs[M.e_v[M.ne + e]])) * 0.5f + hr;
      const float Ae = f32 ? M.e_area32[e] : static_cast<float>(M.e_area[e]);
      ke += Ae * he * (ue * ue);
    }
    // warp sums in FP32, the block's warps in FP64; the other quantities'
    // partials are zero
    float ne = nan;
    for (int off = 16; off > 0; off >>= 1) {
      pe += __shfl_down_sync(0xffffffffu, pe, off);
      ke += __shfl_down_sync(0xffffffffu, ke, off);
      um = fmaxf(um, __shfl_down_sync(0xffffffffu, um, off));
      ne = fmaxf(ne, __shfl_down_sync(0xffffffffu, ne, off));
    }
    __shared__ float se[4][kRedThreads / 32];
    const int ln = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (ln == 0) {
      se[0][wp] = pe;
      se[1][wp] = ke;
      se[2][wp] = um;
      se[3][wp] = ne;
    }
    __syncthreads();
    if (threadIdx.x < kDiagQ) {
      const int q = threadIdx.x;
      double v = 0.0;
      for (int w = 0; w < kRedThreads / 32; ++w) {
        if (q == Q_PE) v += static_cast<double>(se[0][w]);
        if (q == Q_KE) v += static_cast<double>(se[1][w]);
        if (q == Q_UMAX) v = fmax(v, static_cast<double>(se[2][w]));
        if (q == Q_NAN) v = fmax(v, static_cast<double>(se[3][w]));
      }
      scratch[(q * gridDim.x + blockIdx.x) * 2] = v;
      scratch[(q * gridDim.x + blockIdx.x) * 2 + 1] = 0.0;
    }
    return;
  }
  for (int i = tid; FULL && i < M.nv; i += stride) {
    const double A = M.c_areag[i];
    const double hi = static_cast<double>(h[i]) + h_ref;
    const double b = M.c_bt[i];
    if (!isfinite(hi)) nan = 1.0;
    part[Q_PE] += A * g * hi * (hi * 0.5 + b);
    part[Q_AREA] += A;
    part[Q_AH] += A * hi;
    part[Q_AHB] += A * (hi + b);
    part[Q_AB2] += A * b * b;
    // div_hx(u) of the last stage input (diagnostic in tendency, :2570)
    const int n = M.c_nnb[i];
    double d = 0.0;
    for (int j = 0; j < n; ++j) {
      const int e = M.c_ed[j * M.nv + i];
      d = d + static_cast<double>(us[e]) * M.c_sd[j * M.nv + i];
    }
    d = diag_div(d, A * erad);
    part[Q_ADIV2] += A * (d * d);
    maxdiv = fmax(maxdiv, fabs(d));
  }
  for (int e = tid; FULL && e < M.ne; e += stride) {
    const double ue = static_cast<double>(u[e]);
    if (!isfinite(ue)) nan = 1.0;
    umax = fmax(umax, fabs(ue));
    // h_ed of the last stage input, as calc_energies uses (swm.f90:2738)
    const double he =
        (static_cast<double>(hs[M.e_v[e]]) + static_cast<double>(hs[M.e_v[M.ne + e]])) * 0.5 + h_ref;
    part[Q_KE] += M.e_area[e] * he * (ue * ue);
  }
  for (int t = tid; FULL && t < M.nt; t += stride) {
    double eta = 0.0, ht = 0.0;
    for (int s = 0; s < 3; ++s) {
      eta = eta + static_cast<double>(us[M.t_ed[s * M.nt + t]]) * M.t_lt[s * M.nt + t];
      ht = ht + M.t_kite[s * M.nt + t] * (static_cast<double>(hs[M.t_v[s * M.nt + t]]) + h_ref);
    }
    const double A = M.t_areag[t];
    eta = diag_div(eta, A * erad);
    eta = eta + M.t_f[t];
    ht = diag_div(ht, A);
    const double q = ht != 0.0 ? diag_div(eta, ht) : 0.0;
    part[Q_ENS] += A * ht * (q * q) * 0.5;
  }
  // The block's sums, with few FP64 operations, which bound a small grid's call
  // (608 blocks; with 12 compensated sums a warp and the maxima in FP64 a call
  // took 65 us at level 5, 114 at level 7, with these 40 and 90): eight sums go
  // down the warp by halves, nine additions where a sum of its own for each takes
  // 40, in the same tree; the maxima, none of them negative, as integers.
  static_assert(Q_ADIV2 == 7 && Q_MAXDIV == 8 && Q_NAN == 9 && Q_UMAX == 10 && kDiagQ == 12, "");
  __shared__ double sh[kRedThreads / 32][8];
  __shared__ long long smax[3][kRedThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16, n = 4; off >= 4; off >>= 1, n >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const double keep = up ? part[k + n] : part[k], send = up ? part[k] : part[k + n];
      part[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  part[0] += __shfl_xor_sync(0xffffffffu, part[0], 2);
  part[0] += __shfl_xor_sync(0xffffffffu, part[0], 1);
  if ((lane & 3) == 0) sh[warp][lane >> 2] = part[0];
  const double mx[3] = {maxdiv, nan, umax};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    long long m = __double_as_longlong(mx[k]);
    for (int off = 16; off > 0; off >>= 1)
      m = max(m, __shfl_down_sync(0xffffffffu, m, off));
    if (lane == 0) smax[k][warp] = m;
  }
  __syncthreads();
  if (threadIdx.x < kDiagQ) {
    const int q = threadIdx.x;
    KSum t{0.0, 0.0};
    if (q <= Q_ADIV2) {
      for (int w = 0; w < kRedThreads / 32; ++w) t.merge(KSum{sh[w][q], 0.0});
    } else if (q <= Q_UMAX) {
      long long m = 0;
      for (int w = 0; w < kRedThreads / 32; ++w) m = max(m, smax[q - Q_MAXDIV][w]);
      t.s = __longlong_as_double(m);
    }
    scratch[(q * gridDim.x + blockIdx.x) * 2] = t.s;
    scratch[(q * gridDim.x + blockIdx.x) * 2 + 1] = t.c;
  }
}

// error_calc partials (swm.f90:3492-3543): weights A_i (cells) and l*d/2
// (edges, sumfsq_areas :3468-3474)
template <class T>
__global__ void __launch_bounds__(kRedThreads) k_errors(DevMesh M, const T *__restrict__ h,
                                                        const T *__restrict__ u, double h_ref,
                                                        const double *__restrict__ href,
                                                        const double *__restrict__ uref,
                                                        double *__restrict__ scratch) {
  constexpr int NQ = 8;
  KSum acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) acc[q] = KSum{0.0, 0.0};
  const int stride = gridDim.x * blockDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  double mdh = 0.0, mrh = 0.0, mdu = 0.0, mru = 0.0;
  for (int i = tid; i < M.nv; i += stride) {
    const double A = M.c_areag[i];
    const double r = href[i];
    const double dif = (static_cast<double>(h[i]) + h_ref) - r;
    acc[0].add(A * (dif * dif));
    acc[1].add(A * (r * r));
    mdh = fmax(mdh, fabs(dif));
    mrh = fmax(mrh, fabs(r));
  }
  for (int e = tid; e < M.ne; e += stride) {
    const double w = M.e_area[e];
    const double r = uref[e];
    const double dif = static_cast<double>(u[e]) - r;
    acc[4].add(w * (dif * dif));
    acc[5].add(w * (r * r));
    mdu = fmax(mdu, fabs(dif));
    mru = fmax(mru, fabs(r));
  }
  double mx[4] = {mdh, mrh, mdu, mru};
  for (int k = 0; k < 4; ++k)
    for (int off = 16; off > 0; off >>= 1) mx[k] = fmax(mx[k], __shfl_down_sync(0xffffffffu, mx[k], off));
  __shared__ double smax[4][kRedThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int k = 0; k < 4; ++k) smax[k][warp] = mx[k];
  __syncthreads();
  double bm[4] = {0, 0, 0, 0};
  for (int k = 0; k < 4; ++k)
    for (int w = 0; w < kRedThreads / 32; ++w) bm[k] = fmax(bm[k], smax[k][w]);
  block_reduce_store<NQ>(acc, scratch);
  __syncthreads();
  if (threadIdx.x == 0) {
    scratch[(2 * gridDim.x + blockIdx.x) * 2] = bm[0];
    scratch[(3 * gridDim.x + blockIdx.x) * 2] = bm[1];
    scratch[(6 * gridDim.x + blockIdx.x) * 2] = bm[2];
    scratch[(7 * gridDim.x + blockIdx.x) * 2] = bm[3];
  }
}

inline int nblocks(int n, int t) { return (n + t - 1) / t; }

}  // namespace

void launch_stage64(const DevMesh64 &M, const Work<double> &W, const double *h_in,
                    const double *u_in, double *h_out, double *u_out, int stage, double dt,
                    cudaStream_t s, cudaEvent_t *ev, const MoistArgs *moist) {
  if (ev) cudaEventRecord(ev[0], s);
  // diffusion: the triangle and cell kernels also write K_tr zeta(u) and
  // K div u; the edge gradients follow them (and, with hyperdiffusion, the
  // second application), before the edge kernel
  const Diffusion<double> &D = W.dif;
  const int sch = W.scheme;
  if (stage == 0 || stage == 1) dt = dt * 0.5;  // rk_stage
  const int bt = block64(M.nt), bc = block64(M.nv), be = block64(M.ne);
  const int nbt = nblocks(M.nt, bt);
  auto tri = [&](auto kernel, const auto &Q) {
    launch_pdl(kernel, nbt + nblocks(M.ne, bt), bt, s, M, h_in, u_in, W.q_tr, W.pv_on, W.flags,
               D.kt, D.on ? D.coefvort : nullptr, sch, W.eta_t, W.h_trs, W.uh, W.fe, nbt, Q);
  };
  if (moist)
    tri(k_tri64<MoistArgs>, *moist);
  else
    tri(k_tri64<NoMoist>, NoMoist{});
  if (ev) cudaEventRecord(ev[1], s);
  const Apvm<double> &A = W.apvm;
  if (A.on) {
    launch_pdl(k_qgrad64, nblocks(M.ne, be), be, s, M, W.q_tr, A.qge);
    launch_pdl(k_apvm64, nbt + nblocks(M.nv, bt), bt, s, M, A.qge, u_in, A.qg, A.vhx, nbt);
  }
  if (sch == IMODEL_SWM_DTRED)
    launch_pdl(k_vhq64, nblocks(M.nt, bt), bt, s, M, W.uh, W.q_tr, W.vhq);
  if (ev) cudaEventRecord(ev[2], s);
  const int nbc = nblocks(M.nv, bc);
  auto cell = [&](auto kernel, const auto &Q) {
    launch_pdl(kernel, nbc + nblocks(M.ne, bc), bc, s, M, h_in, u_in, W.fe, W.bern, W.yn_h,
               W.acc_h, h_out, W.tend_h, stage, dt, D.kcv, D.on ? D.coefdiv : nullptr, nbc,
               W.q_ed, W.q_tr, A.on ? A.qg : nullptr, A.vhx, A.coef, sch, W.eta_t, W.h_trs,
               W.pv_on, W.flags, Q);
  };
  if (moist)
    cell(k_cell64<MoistArgs>, *moist);
  else
    cell(k_cell64<NoMoist>, NoMoist{});
  if (D.on) {
    launch_pdl(k_diflap64, nblocks(M.ne, be), be, s, M, D.coefdiv, D.coefvort, D.lap);
    if (D.k4) {
      launch_pdl(k_difcv64, nbc + nblocks(M.nt, bc), bc, s, M, D.lap, D.kcv, D.kt, D.coefdiv,
                 D.coefvort, nbc);
      launch_pdl(k_diflap64, nblocks(M.ne, be), be, s, M, D.coefdiv, D.coefvort, D.lap2);
    }
  }
  if (ev) cudaEventRecord(ev[3], s);
  if (sch == IMODEL_SWM_PXT16 || sch == IMODEL_SWM_DTRED)
    launch_pdl(k_edge64r, nblocks(M.ne, be), be, s, M, W.bern, W.uh, W.q_ed, W.vhq, W.yn_u,
               W.acc_u, u_out, W.tend_u, stage, dt, W.mom_on, D.k2 ? D.lap : nullptr, D.k4 ?
               D.lap2 : nullptr, sch);
  else {
    auto edge = [&](auto kernel, const auto &Q) {
      launch_pdl(kernel, nblocks(M.ne, be), be, s, M, W.bern, W.uh, W.q_ed, W.yn_u, W.acc_u, u_out,
                 W.tend_u, stage, dt, W.mom_on, D.k2 ? D.lap : nullptr, D.k4 ? D.lap2 : nullptr,
                 sch == IMODEL_SWM_GASS18 ? M.e_stq : nullptr, Q);
    };
    if (moist)
      edge(k_edge64<MoistArgs>, *moist);
    else
      edge(k_edge64<NoMoist>, NoMoist{});
  }
  if (ev) cudaEventRecord(ev[4], s);
}

size_t consts64_size(const DevMesh64 &M) {
  const size_t nv = M.nv, ne = M.ne, nt = M.nt;
  return nv * 5 + ne * 5 + nt + (M.t_c ? 2 * (nv + ne + nt) : 0) + (M.e_dist ? 2 * ne : 0) +
         (M.t_bary ? 18 * nv : 0);
}

void launch_consts64(DevMesh64 &M, double *p, cudaStream_t s) {
  const size_t nv = M.nv, ne = M.ne, nt = M.nt;
  auto take = [&p](size_t n) {
    double *q = p;
    p += n;
    return q;
  };
  M.rerad = M.erad >= kRecipLow && M.erad <= kRecipHigh ? 1.0 / M.erad : std::nan("");
  M.c_rareag = take(nv);
  M.c_rcellarea = take(nv);
  M.c_eds = reinterpret_cast<const uint32_t *>(take(3 * nv));
  M.e_rleng = take(ne);
  M.e_rdleng = take(ne);
  M.e_d8 = take(ne);
  M.e_dlerad = take(ne);
  M.e_rdlerad = take(ne);
  M.t_rareag = take(nt);
  if (M.t_c) {
    M.c_nrm = take(nv);
    M.c_rnrm = take(nv);
    M.e_nrm = take(ne);
    M.e_rnrm = take(ne);
    M.t_nrm = take(nt);
    M.t_rnrm = take(nt);
  }
  if (M.e_dist) {
    M.e_dsum = take(ne);
    M.e_rdsum = take(ne);
  }
  if (M.t_bary) M.c_off = take(18 * nv);
  int n = M.nv > M.ne ? M.nv : M.ne;
  if (M.nt > n) n = M.nt;
  k_consts64<<<nblocks(n, 256), 256, 0, s>>>(M);
}

void launch_dif_coefs(const DevMesh &M, const double *kf, double k, bool take_sqrt, double *kc64,
                      float *kc32, double *kt64, float *kt32, cudaStream_t s) {
  const int nbc = nblocks(M.nv, 256);
  k_dif_coefs<<<nbc + nblocks(M.nt, 256), 256, 0, s>>>(M, kf, k, take_sqrt ? 1 : 0, kc64, kc32,
                                                        kt64, kt32, nbc);
}

void launch_gather_in(int n, const int32_t *n2o, const double *src, double *dst, double shift,
                      cudaStream_t s) {
  k_gather_in<double><<<nblocks(n, 256), 256, 0, s>>>(n, n2o, src, dst, shift);
}
void launch_gather_in32(int n, const int32_t *n2o, const double *src, float *dst, double shift,
                        cudaStream_t s) {
  k_gather_in<float><<<nblocks(n, 256), 256, 0, s>>>(n, n2o, src, dst, shift);
}
void launch_scatter_out(int n, const int32_t *n2o, const double *src, double *dst, double shift,
                        int *flags, cudaStream_t s) {
  k_scatter_out<double><<<nblocks(n, 256), 256, 0, s>>>(n, n2o, src, dst, shift, flags);
}
void launch_scatter_out32(int n, const int32_t *n2o, const float *src, double *dst,
                          double shift, int *flags, cudaStream_t s) {
  k_scatter_out<float><<<nblocks(n, 256), 256, 0, s>>>(n, n2o, src, dst, shift, flags);
}

template <class T>
void launch_load_host(const HostMap &N, const double *h, const double *u, HostTo<T> to_h,
                      HostTo<T> to_u, double shift, cudaStream_t s) {
  launch_pdl(k_load_host<T>, nblocks(N.nv + N.ne, 256), 256, s, N, h, u, to_h, to_u, shift);
}
template <class T>
void launch_store_host(const HostMap &N, const T *src_h, const T *src_u, double *h, double *u,
                       double shift, int *flags, cudaStream_t s) {
  launch_pdl(k_store_host<T>, nblocks(N.nv + N.ne, 256), 256, s, N, src_h, src_u, h, u, shift,
             flags);
}
template void launch_load_host<double>(const HostMap &, const double *, const double *,
                                       HostTo<double>, HostTo<double>, double, cudaStream_t);
template void launch_load_host<float>(const HostMap &, const double *, const double *,
                                      HostTo<float>, HostTo<float>, double, cudaStream_t);
template void launch_store_host<double>(const HostMap &, const double *, const double *, double *,
                                        double *, double, int *, cudaStream_t);
template void launch_store_host<float>(const HostMap &, const float *, const float *, double *,
                                       double *, double, int *, cudaStream_t);
cudaError_t launch_take_flags(int *flags, int *host, cudaStream_t s) {
  return launch_pdl(k_take_flags, 1, 1, s, flags, host);
}

void launch_trsk_tangent(const DevMesh &M, const double *u, double *utg, cudaStream_t s) {
  k_trsk_tangent<<<nblocks(M.ne, 256), 256, 0, s>>>(M, u, utg);
}

template <class T>
void launch_diag(const DevMesh &M, const Work<T> &W, const T *h, const T *u, const T *hs,
                 const T *us, double *scratch, double *result, cudaStream_t s,
                 bool energy_only) {
  if (energy_only)
    k_diag<T, false><<<kRedBlocks, kRedThreads, 0, s>>>(M, h, u, hs, us,
                                                         static_cast<double>(W.h_ref), scratch);
  else
    k_diag<T, true><<<kRedBlocks, kRedThreads, 0, s>>>(M, h, u, hs, us,
                                                        static_cast<double>(W.h_ref), scratch);
  const unsigned maxmask = (1u << Q_MAXDIV) | (1u << Q_NAN) | (1u << Q_UMAX);
  launch_pdl(k_finalize, kDiagQ, kRedThreads, s, scratch, kRedBlocks, kDiagQ, maxmask, result);
}
template void launch_diag<double>(const DevMesh &, const Work<double> &, const double *,
                                  const double *, const double *, const double *, double *,
                                  double *, cudaStream_t, bool);
template void launch_diag<float>(const DevMesh &, const Work<float> &, const float *,
                                 const float *, const float *, const float *, double *,
                                 double *, cudaStream_t, bool);

template <class T>
void launch_errors(const DevMesh &M, const T *h, const T *u, double h_ref, const double *href,
                   const double *uref, double *scratch, double *result, cudaStream_t s) {
  k_errors<T><<<kRedBlocks, kRedThreads, 0, s>>>(M, h, u, h_ref, href, uref, scratch);
  const unsigned maxmask = (1u << 2) | (1u << 3) | (1u << 6) | (1u << 7);
  launch_pdl(k_finalize, 8, kRedThreads, s, scratch, kRedBlocks, 8, maxmask, result);
}
template void launch_errors<double>(const DevMesh &, const double *, const double *, double,
                                    const double *, const double *, double *, double *,
                                    cudaStream_t);
template void launch_errors<float>(const DevMesh &, const float *, const float *, double,
                                   const double *, const double *, double *, double *,
                                   cudaStream_t);

}  // namespace imodel
