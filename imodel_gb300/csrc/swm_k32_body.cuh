// Per-entity bodies of the FP32 cell-centred TRSK stage (internal header).
//
// Shared by the single-run kernels (swm_k32.cu) and the tiles of the fused
// stage and the ensemble kernel (swm_tile.cuh).
#pragma once
#include "swm_common.cuh"
#include "swm_pair.cuh"

namespace imodel {

// Between the loads of the fixed records and the first load of a changing
// field: the wait for the kernel before (after_prior), or nothing.
struct NoWait {
  static constexpr bool kWaits = false;
};
struct PriorWait {
  static constexpr bool kWaits = true;
};
// (discarded without a wait: taking the pointers by reference alone made the
// cell kernel 2 % slower at level 9)
#define IMODEL_WAIT(Wait, ...) \
  if constexpr (Wait::kWaits) after_prior<true>(__VA_ARGS__)

// Which products are fused into a sum is written out in the functions below,
// not left to the compiler: the separate kernels, the fused stage and the
// ensemble kernel give the same bits.  V: float, or Pair for two members.

// ode_rk4 stage update (swm.f90:2647-2678) in FP32
template <class V>
__device__ __forceinline__ V rk_stage32(int stage, V k, V yn, V *acc, float dt) {
  if (stage == 0) {
    *acc = k;
    return vfma(all<V>(0.5f * dt), k, yn);
  } else if (stage == 1) {
    *acc = vfma(all<V>(2.0f), k, *acc);
    return vfma(all<V>(0.5f * dt), k, yn);
  } else if (stage == 2) {
    *acc = vfma(all<V>(2.0f), k, *acc);
    return vfma(all<V>(dt), k, yn);
  }
  return vfma(vmul(all<V>(dt), vadd(*acc, k)), all<V>(1.0f / 6.0f), yn);
}

// scalar_elem_divide with its guard, swm_operators.f90:1604-1606
__device__ __forceinline__ float guarded_div(float a, float b, int *flags) {
  if (fabsf(b) < 1.1920928955078125e-12f) {
    atomicOr(flags, 1);
    return 0.0f;
  }
  return a / b;
}
__device__ __forceinline__ Pair guarded_div(Pair a, Pair b, int *flags) {
  return Pair{guarded_div(a.x, b.x, flags), guarded_div(a.y, b.y, flags)};
}

// q_t = (curl u / A + f) / h_t  (vort_tr + scalar_hx2tr + scalar_elem_divide)
// from a triangle's decoded record: edges, cells, circulation and kite
// coefficients, Coriolis parameter; the sums run in slot order 0, 1, 2
template <class Wait, class V>
__device__ __forceinline__ void tri_core(int t, const int (&ed)[3], const int (&cv)[3],
                                         const float (&circ)[3], const float (&kite)[3],
                                         float f, const V *__restrict__ hd,
                                         const V *__restrict__ u, V *__restrict__ q_tr,
                                         float h_ref, int pv_on, int *flags,
                                         const float *__restrict__ kt = nullptr,
                                         typename ValueOf<V>::type *__restrict__ coefvort =
                                             nullptr,
                                         typename ValueOf<V>::type *__restrict__ ht_out =
                                             nullptr) {
  IMODEL_WAIT(Wait, hd, u, q_tr, coefvort, ht_out);
  V eta = all<V>(f);
  V ht = all<V>(0.0f), z = all<V>(0.0f);
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const V us = u[ed[s]], c = all<V>(circ[s]);
    eta = vfma(c, us, eta);
    z = vfma(c, us, z);
    ht = vfma(all<V>(kite[s]), hd[cv[s]], ht);
  }
  // with diffusion on: K_tr times the relative vorticity
  if (coefvort) coefvort[t] = vmul(all<V>(kt[t]), z);
  ht = padd(ht, all<V>(h_ref));
  // gass18: the depth at the triangle for the rhombus PV of the edges
  if (ht_out) ht_out[t] = ht;
  V q = all<V>(0.0f);
  if (pv_on) q = guarded_div(eta, ht, flags);
  q_tr[t] = q;
}

template <class Wait>
__device__ __forceinline__ void tri_body(const DevMesh &M, int t,
                                         const float *__restrict__ hd,
                                         const float *__restrict__ u, float *__restrict__ q_tr,
                                         float h_ref, int pv_on, int *flags,
                                         const float *__restrict__ kt = nullptr,
                                         float *__restrict__ coefvort = nullptr,
                                         float *__restrict__ ht_out = nullptr) {
  // three 16-byte records instead of 12 scalar streams (fewer load
  // instructions in flight per SM)
  const int4 a = __ldg(&M.t_recA[t]), b = __ldg(&M.t_recB[t]);
  const float4 c = __ldg(&M.t_recC[t]);
  const int ed[3] = {a.x, a.y, a.z}, cv[3] = {a.w, b.x, b.y};
  const float circ[3] = {__int_as_float(b.z), __int_as_float(b.w), c.x};
  const float kite[3] = {c.y, c.z, c.w};
  tri_core<Wait>(t, ed, cv, circ, kite, __ldg(&M.t_f32[t]), hd, u, q_tr, h_ref, pv_on,
                   flags, kt, coefvort, ht_out);
}

// the same from 40-byte records with 16-bit indices (single runs): a warp of
// 32 triangles shares one base per index kind (t_wb); a warp whose indices
// span more than 65,536 takes its indices from the 32-bit records instead
// (warp-uniform branch).  The records and the bases are loaded together, so
// that the gathers wait for one round trip, as with the 32-bit records.
template <class Wait>
__device__ __forceinline__ void tri_body16(const DevMesh &M, int t, const float *__restrict__ hd,
                                           const float *__restrict__ u,
                                           float *__restrict__ q_tr, float h_ref, int pv_on,
                                           int *flags, const float *__restrict__ kt,
                                           float *__restrict__ coefvort) {
  const int2 wb = __ldg(&M.t_wb[t >> 5]);
  const uint4 a = __ldg(&M.t_c16A[t]);
  const float4 b = __ldg(&M.t_c16B[t]);
  const float2 c = __ldg(&M.t_c16C[t]);
  int ed[3], cv[3];
  if (wb.y >= 0) {
    ed[0] = wb.x + static_cast<int>(a.x & 0xFFFFu);
    ed[1] = wb.x + static_cast<int>(a.x >> 16);
    ed[2] = wb.x + static_cast<int>(a.y & 0xFFFFu);
    cv[0] = wb.y + static_cast<int>(a.y >> 16);
    cv[1] = wb.y + static_cast<int>(a.z & 0xFFFFu);
    cv[2] = wb.y + static_cast<int>(a.z >> 16);
  } else {
    const int4 ra = __ldg(&M.t_recA[t]), rb = __ldg(&M.t_recB[t]);
    ed[0] = ra.x;
    ed[1] = ra.y;
    ed[2] = ra.z;
    cv[0] = ra.w;
    cv[1] = rb.x;
    cv[2] = rb.y;
  }
  const float circ[3] = {__uint_as_float(a.w), b.x, b.y};
  const float kite[3] = {b.z, b.w, c.x};
  tri_core<Wait>(t, ed, cv, circ, kite, c.y, hd, u, q_tr, h_ref, pv_on,
                            flags, kt, coefvort);
}

// coriolis_ed (swm_operators.f90:1283-1308) sums, for edge e and each of its
// two cells c, over the other edges k_j of c:
//     F_k * (q_e + q_k)/2 * d_k * w_c(i_e, j) * ttgout_c(j) * tnrccw_c(i_e)
// with w_c(i, j) = sum_{k=i}^{j-1} R_c(k) - 1/2 (calc_trisk_weights,
// interpack.f90:4046-4095).  Every factor but q_e lives on cell c, so each
// cell computes the contribution Z_c(i) of all its n edges at once from its n
// kite fractions R_c; the edge kernel adds the two cells' Z and divides by
// l_e.  The 10-entry stencil (40 B of indices and 40 B of weights per edge)
// becomes n fractions per cell.
//
// The fractions sum to one, so w_c(j, i) = -w_c(i, j): a pair of edges
// shares its weight and q_i + q_j between both its terms (five operations a
// pair, where summing each edge's row took ten), and the pair's work cancels
// exactly in the weight.  S(j) = R(0) + ... + R(j - 1), w = (S(j) - 1/2) - S(i).
//
// A row's terms with the smaller edges come first, all with a minus: they are
// summed without it, and the sum turned once.
template <int N, class V>
__device__ __forceinline__ void trsk_cell(const V (&G)[6], const V (&qs)[6], const float (&R)[6],
                                          unsigned tneg, V (&Z)[6]) {
  V S[N], a[N];
  S[0] = all<V>(0.0f);
#pragma unroll
  for (int j = 1; j < N; ++j) S[j] = padd(S[j - 1], all<V>(R[j - 1]));
#pragma unroll
  for (int i = 0; i < N; ++i) a[i] = all<V>(0.0f);
#pragma unroll
  for (int j = 1; j < N; ++j) {
    const V Sh = padd(S[j], all<V>(-0.5f));
#pragma unroll
    for (int i = 0; i < j; ++i) {
      const V t = vmul(psub(Sh, S[i]), vadd(qs[i], qs[j]));
      a[i] = vfma(t, G[j], a[i]);
      a[j] = vfma(t, G[i], a[j]);
    }
    a[j] = vneg(a[j]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const V z = pmul(all<V>(0.5f), a[i]);
    Z[i] = ((tneg >> i) & 1u) ? vneg(z) : z;
  }
}

// the arithmetic of one cell from its gathered values: div F, K, the
// Bernoulli potential, the PV-flux contributions Z (cell-major zflux);
// returns the sum of the fluxes out of the cell.  kEdgePV: qt holds the PV of
// the cell's edges (formed by the edge pre-pass, APVM's upwinding included)
// instead of the PV of its triangles.
template <bool kEdgePV = false, bool kZ = true, class V = float>
__device__ __forceinline__ V cell_terms(int i, uint32_t meta, const float (&R)[6],
                                        const float2 (&kd)[6], const V (&ue)[6],
                                        const V (&hn)[6], const V (&qt)[6], V hi, float bt,
                                        float inva, V *__restrict__ bern, V *__restrict__ zflux,
                                        float grav, float h_ref,
                                        const float *__restrict__ kcv = nullptr,
                                        typename ValueOf<V>::type *__restrict__ coefdiv =
                                            nullptr,
                                        const typename ValueOf<V>::type *dv = nullptr) {
  const int n = static_cast<int>(meta & 7u);
  const unsigned tneg = meta >> 8;
  const V half = all<V>(0.5f), href = all<V>(h_ref);
  V G[6], qs[6];
  V div = all<V>(0.0f), ke = all<V>(0.0f), du = all<V>(0.0f);
  const V qlast = n == 6 ? qt[5] : (n == 5 ? qt[4] : (n == 4 ? qt[3] : qt[2]));
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    // F_e = u_e h_e, h_e the two-cell average (scalar_hx2ed)
    const V F = vmul(ue[j], vfma(half, padd(hi, hn[j]), href));
    const V d = all<V>(kd[j].y);
    G[j] = vmul(F, d);
    // q_e: edge j lies between triangles j-1 and j (scalar_tr2ed)
    qs[j] = kEdgePV ? qt[j] : pmul(half, padd(j == 0 ? qlast : qt[j - 1], qt[j]));
    div = vadd(div, G[j]);
    ke = vfma(all<V>(kd[j].x), vmul(ue[j], ue[j]), ke);
    du = vfma(dv ? dv[j] : ue[j], d, du);
  }
  // with diffusion on: K times the divergence of u (or of dv)
  if (coefdiv) coefdiv[i] = vmul(all<V>(kcv[i]), vmul(du, all<V>(inva)));
  bern[i] = vfma(all<V>(grav), padd(hi, all<V>(bt)), ke);
  // kZ false (dtred): the edges form their PV flux from the triangles
  if (kZ) {
    V Z[6];
    if (n == 6)
      trsk_cell<6>(G, qs, R, tneg, Z);
    else if (n == 5)
      trsk_cell<5>(G, qs, R, tneg, Z);
    else if (n == 4)
      trsk_cell<4>(G, qs, R, tneg, Z);
    else
      trsk_cell<3>(G, qs, R, tneg, Z);
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (j < n) zflux[6 * i + j] = Z[j];
  }
  return div;
}

// cell_terms and the mass RK stage
template <bool kEdgePV = false, bool kZ = true>
__device__ __forceinline__ void cell_math(int i, uint32_t meta, const float (&R)[6],
                                          const float2 (&kd)[6], const float (&ue)[6],
                                          const float (&hn)[6], const float (&qt)[6], float hi,
                                          float bt, float inva, float ynv, float accv,
                                          float *__restrict__ bern, float *__restrict__ zflux,
                                          float *__restrict__ acc, float *__restrict__ yout,
                                          float *__restrict__ tend, int stage, float dt,
                                          float grav, float h_ref,
                                          const float *__restrict__ kcv = nullptr,
                                          float *__restrict__ coefdiv = nullptr,
                                         const float *dv = nullptr) {
  const float div = cell_terms<kEdgePV, kZ>(i, meta, R, kd, ue, hn, qt, hi, bt, inva, bern,
                                                zflux, grav, h_ref, kcv, coefdiv, dv);
  const float masseq = __fmul_rn(-div, inva);
  if (stage < 0) {
    tend[i] = masseq;
  } else {
    float a = accv;
    yout[i] = rk_stage32(stage, masseq, ynv, &a, dt);
    if (stage < 3) acc[i] = a;
  }
}

// div F, K, Bernoulli potential, PV-flux contributions Z (cell-major
// zflux[cell][6]) and the mass RK stage of cell i, from its decoded slot
// records: edge, neighbour, triangle, kite fraction R and {KE weight,
// ttgout*d} of each slot (unused pentagon slots repeat slot 0 with zero
// weights), gathering its neighbours' values.  The cell's own values come in
// as arguments: h (deviation) hi, b bt, 1/(A a) inva, y_n ynv and the RK
// accumulator accv (read for stages 1-3).  lap: coefdiv holds its divergence
// in place of u's.
template <bool kEdgePV, bool kZ>
__device__ __forceinline__ void cell_core(int i, uint32_t meta,
                                          const int (&ed)[6], const int (&nb)[6],
                                          const int (&tr)[6], const float (&R)[6],
                                          const float2 (&kd)[6], float hi, float bt, float inva,
                                          float ynv, float accv, const float *__restrict__ hd,
                                          const float *__restrict__ u,
                                          const float *__restrict__ q_tr,
                                          float *__restrict__ bern, float *__restrict__ zflux,
                                          float *__restrict__ acc, float *__restrict__ yout,
                                          float *__restrict__ tend, int stage, float dt,
                                          float grav, float h_ref, const float *__restrict__ kcv = nullptr,
                                          float *__restrict__ coefdiv = nullptr,
                                          const float *__restrict__ lap = nullptr) {
  float ue[6], hn[6], qt[6], dv[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    ue[j] = u[ed[j]];
    hn[j] = hd[nb[j]];
    if (lap) dv[j] = lap[ed[j]];
    // kEdgePV: q_tr is the edges' PV, indexed by the slot's edge
    qt[j] = q_tr[kEdgePV ? ed[j] : tr[j]];
  }
  cell_math<kEdgePV, kZ>(i, meta, R, kd, ue, hn, qt, hi, bt, inva, ynv, accv, bern, zflux,
                             acc, yout, tend, stage, dt, grav, h_ref, kcv, coefdiv,
                         lap ? dv : nullptr);
}

// the cell's own values from global memory
__device__ __forceinline__ void cell_own(const DevMesh &M, int i,
                                         const float *__restrict__ hd,
                                         const float *__restrict__ yn,
                                         const float *__restrict__ acc, int stage, float &hi,
                                         float &bt, float &inva, float &ynv, float &accv) {
  hi = hd[i];
  bt = __ldg(&M.c_bt32[i]);
  inva = __ldg(&M.c_inva32[i]);
  ynv = stage >= 0 ? yn[i] : 0.0f;
  accv = stage >= 1 ? acc[i] : 0.0f;
}

template <bool kEdgePV, bool kZ, class Wait>
__device__ __forceinline__ void cell_body(const DevMesh &M, int i,
                                          const float *__restrict__ hd,
                                          const float *__restrict__ u,
                                          const float *__restrict__ q_tr,
                                          float *__restrict__ bern, float *__restrict__ zflux,
                                          const float *__restrict__ yn, float *__restrict__ acc,
                                          float *__restrict__ yout, float *__restrict__ tend,
                                          int stage, float dt, float grav, float h_ref,
                                          const float *__restrict__ kcv = nullptr,
                                          float *__restrict__ coefdiv = nullptr,
                                          const float *__restrict__ lap = nullptr) {
  const int nv = M.nv;
  const uint32_t meta = __ldg(&M.c_meta[i]);
  int ed[6], nb[6], tr[6];
  float R[6];
  float2 kd[6];
  // all slot records first, so that every load is in flight before the
  // gathers
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const int4 pk = __ldg(&M.c_pk[j * nv + i]);
    kd[j] = __ldg(&M.c_kd[j * nv + i]);
    ed[j] = pk.x;
    nb[j] = pk.y;
    tr[j] = pk.z;
    R[j] = __int_as_float(pk.w);
  }
  IMODEL_WAIT(Wait, hd, u, q_tr, bern, zflux, yn, acc, yout, tend, coefdiv, lap);
  float hi, bt, inva, ynv, accv;
  cell_own(M, i, hd, yn, acc, stage, hi, bt, inva, ynv, accv);
  cell_core<kEdgePV, kZ>(i, meta, ed, nb, tr, R, kd, hi, bt, inva, ynv, accv, hd, u,
                                 q_tr, bern, zflux, acc, yout, tend, stage, dt, grav, h_ref, kcv,
                                 coefdiv, lap);
}

// -grad B - (Z_c1 + Z_c2) / l_e of an edge
template <class V>
__device__ __forceinline__ V edge_terms(V b1, V b2, V z1, V z2, float g, float erad) {
  const V grad = vmul(psub(b2, b1), all<V>(-g));
  return vfma(padd(z1, z2), all<V>(__fmul_rn(-g, erad)), grad);
}

// grad_ed(K div x) - grad_ed_tg(K_tr zeta(x)) of an edge between the cells
// c1, c2
__device__ __forceinline__ float edge_lap(const DevMesh &M, int e, int c1, int c2, float g,
                                          const float *__restrict__ coefdiv,
                                          const float *__restrict__ coefvort) {
  const int t1 = __ldg(&M.e_sh[e]), t2 = __ldg(&M.e_sh[M.ne + e]);
  const float gt = __fmul_rn(coefvort[t2] - coefvort[t1], __ldg(&M.e_gtg32[e]));
  return fmaf(coefdiv[c2] - coefdiv[c1], g, -gt);
}

// the diffusion terms that the edge kernel adds: + lap when given, then sgn
// (1 or -1) times edge_lap of coefdiv and coefvort when given
struct EdgeDif {
  const float *lap = nullptr, *coefdiv = nullptr, *coefvort = nullptr;
  float sgn = 0.0f;
};

// -grad B - (Z_c1 + Z_c2) / l_e and the momentum RK stage of edge e
__device__ __forceinline__ void edge_body(const DevMesh &M, int e, uint2 w,
                                          const float *__restrict__ bern,
                                          const float *__restrict__ zflux,
                                          const float *__restrict__ yn, float *__restrict__ acc,
                                          float *__restrict__ yout, float *__restrict__ tend,
                                          int stage, float dt, int mom_on, float erad,
                                          const float *__restrict__ corr, const EdgeDif &D) {
  const int c1 = static_cast<int>(w.x & 0x0FFFFFFFu), c2 = static_cast<int>(w.y & 0x0FFFFFFFu);
  const int s1 = static_cast<int>(w.x >> 28), s2 = static_cast<int>(w.y >> 28);
  const float g = __ldg(&M.e_grad32[e]);  // 1 / (l_e a)
  float momeq = edge_terms(bern[c1], bern[c2], zflux[6 * c1 + s1], zflux[6 * c2 + s2], g, erad);
  // learned correction of the PV flux (frozen over the RK step)
  if (corr) momeq += corr[e];
  // diffusion, then hyperdiffusion
  if (D.lap) momeq += D.lap[e];
  if (D.coefdiv) momeq = fmaf(D.sgn, edge_lap(M, e, c1, c2, g, D.coefdiv, D.coefvort), momeq);
  if (!mom_on) momeq = 0.0f;
  if (stage < 0)
    tend[e] = momeq;
  else
    yout[e] = rk_stage32(stage, momeq, yn[e], acc + e, dt);
}

}  // namespace imodel
