// The phases of a tile's RK stage in shared memory (internal header), shared
// by the fused stage of single runs (swm_stage32.cu) and the ensemble kernel
// (swm_ens.cu).  Tiles and their blocks: swm_layout.h; the arithmetic:
// swm_k32_body.cuh, as in the separate kernels and with the same bits.
#pragma once
#include <type_traits>

#include "swm_k32_body.cuh"
#include "tc05.cuh"

namespace imodel {

// a bulk copy of `bytes` bytes (a multiple of 16, both addresses aligned to
// 16) whose arrival mbar counts
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *mbar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   tc05::smem_u32(mbar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(tc05::smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(tc05::smem_u32(mbar))
      : "memory");
}

// a tile's head (TileHead)
struct Tile {
  int c0, nc, nz, nh, e0, ne, nu, nt;
  int block, ux, slot, triA, triB, triC, edge, meta, bt, inva, bytes;
  __device__ __forceinline__ Tile(const int4 *head) {
    const int4 A = __ldg(head), B = __ldg(head + 1), C = __ldg(head + 2), D = __ldg(head + 3),
               E = __ldg(head + 4);
    c0 = A.x, nc = A.y, nz = A.z, nh = A.w;
    e0 = B.x, ne = B.y, nu = B.z, nt = B.w;
    block = C.x, ux = C.y, slot = C.z, triA = C.w;
    triB = D.x, triC = D.y, edge = D.z, meta = D.w;
    bt = E.x, inva = E.y, bytes = E.z;
  }
};

// one run's fields: stage input, y_n, accumulators, stage output (stage < 0:
// the tendencies); of two members, the first's, the second's mh and mu further
struct TileFields {
  const float *hd, *u, *yn_h, *yn_u;
  float *acc_h, *acc_u, *h_out, *u_out, *tend_h, *tend_u;
  size_t mh = 0, mu = 0;
};
// element i; the int index keeps it to one wide multiply-add an address
template <class V>
__device__ __forceinline__ V tile_load(const float *p, int i, size_t) {
  return p[i];
}
template <>
__device__ __forceinline__ Pair tile_load<Pair>(const float *p, int i, size_t m) {
  return Pair{p[i], (p + m)[i]};
}
__device__ __forceinline__ void tile_store(float *p, int i, size_t, float v) { p[i] = v; }
__device__ __forceinline__ void tile_store(float *p, int i, size_t m, Pair v) {
  p[i] = v.x;
  (p + m)[i] = v.y;
}

// the block's shared arrays: depths, velocities, PV, potential, flux terms
template <class V>
struct TileSharedOf {
  unsigned char *block;  // the tile's block
  V *sh, *su, *sq, *sb, *sz;
};
using TileShared = TileSharedOf<float>;

// What a thread of nthr reads in order, all of it in flight at once: the own
// depth and velocities, y_n and the accumulators of the update.  kE rounds
// cover a tile's own edges (three a cell); loops take what is left.
template <int nthr, class V = float>
struct TileOwn {
  static constexpr int kE = 3;
  V uo[kE], ynu[kE], acu[kE], ho, ynh, ach;
  // kEdges false: without y_n and the accumulators of the edges (load_edges)
  template <bool kEdges = true>
  __device__ __forceinline__ void load(const Tile &T, const TileFields &F, int stage) {
    const int tid = threadIdx.x;
    ho = all<V>(0.0f), ynh = all<V>(0.0f), ach = all<V>(0.0f);
#pragma unroll
    for (int r = 0; r < kE; ++r) {
      const int k = tid + r * nthr;
      uo[r] = ynu[r] = acu[r] = all<V>(0.0f);
      if (k < T.ne) {
        uo[r] = tile_load<V>(F.u, T.e0 + k, F.mu);
        if (kEdges && stage >= 0) ynu[r] = tile_load<V>(F.yn_u, T.e0 + k, F.mu);
        if (kEdges && stage >= 1) acu[r] = tile_load<V>(F.acc_u, T.e0 + k, F.mu);
      }
    }
    if (tid < T.nc) {
      ho = tile_load<V>(F.hd, T.c0 + tid, F.mh);
      if (stage >= 0) ynh = tile_load<V>(F.yn_h, T.c0 + tid, F.mh);
      if (stage >= 1) ach = tile_load<V>(F.acc_h, T.c0 + tid, F.mh);
    }
  }
  __device__ __forceinline__ void load_edges(const Tile &T, const TileFields &F, int stage) {
#pragma unroll
    for (int r = 0; r < kE; ++r) {
      const int k = threadIdx.x + r * nthr;
      if (k < T.ne) {
        ynu[r] = tile_load<V>(F.yn_u, T.e0 + k, F.mu);
        if (stage >= 1) acu[r] = tile_load<V>(F.acc_u, T.e0 + k, F.mu);
      }
    }
  }
  // the rim's depths and velocities (the block's index lists have arrived):
  // fewer than two rounds of velocities, one of depths; loops take the rest
  __device__ __forceinline__ void rim_load(const Tile &T, const TileFields &F,
                                           const TileSharedOf<V> &S, V (&v)[3]) {
    const int32_t *hx = reinterpret_cast<const int32_t *>(S.block);
    const int32_t *ux = reinterpret_cast<const int32_t *>(S.block + T.ux);
    const int k0 = threadIdx.x, k1 = k0 + nthr, nux = T.nu - T.ne, nhx = T.nh - T.nc;
    if (k0 < nux) v[0] = tile_load<V>(F.u, ux[k0], F.mu);
    if (k1 < nux) v[1] = tile_load<V>(F.u, ux[k1], F.mu);
    if (k0 < nhx) v[2] = tile_load<V>(F.hd, hx[k0], F.mh);
  }
  __device__ __forceinline__ void rim_store(const Tile &T, const TileFields &F,
                                            const TileSharedOf<V> &S, const V (&v)[3]) {
    const int32_t *hx = reinterpret_cast<const int32_t *>(S.block);
    const int32_t *ux = reinterpret_cast<const int32_t *>(S.block + T.ux);
    const int k0 = threadIdx.x, k1 = k0 + nthr, nux = T.nu - T.ne, nhx = T.nh - T.nc;
    if (k0 < nux) S.su[T.ne + k0] = v[0];
    if (k1 < nux) S.su[T.ne + k1] = v[1];
    if (k0 < nhx) S.sh[T.nc + k0] = v[2];
    for (int k = k1 + nthr; k < nux; k += nthr) S.su[T.ne + k] = tile_load<V>(F.u, ux[k], F.mu);
    for (int k = k1; k < nhx; k += nthr) S.sh[T.nc + k] = tile_load<V>(F.hd, hx[k], F.mh);
  }
  __device__ __forceinline__ void rim(const Tile &T, const TileFields &F,
                                      const TileSharedOf<V> &S) {
    V v[3];
    rim_load(T, F, S, v);
    rim_store(T, F, S, v);
  }
  __device__ __forceinline__ void store(const Tile &T, const TileFields &F,
                                        const TileSharedOf<V> &S) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int r = 0; r < kE; ++r)
      if (tid + r * nthr < T.ne) S.su[tid + r * nthr] = uo[r];
    for (int k = tid + kE * nthr; k < T.ne; k += nthr)
      S.su[k] = tile_load<V>(F.u, T.e0 + k, F.mu);
    if (tid < T.nc) S.sh[tid] = ho;
  }
};

// PV at the tile's triangles
template <int nthr, class V>
__device__ __forceinline__ void tile_triangles(const Tile &T, const TileSharedOf<V> &S,
                                               float h_ref, int pv_on, int *flags) {
  const float4 *ta = reinterpret_cast<const float4 *>(S.block + T.triA);
  const uint4 *tb = reinterpret_cast<const uint4 *>(S.block + T.triB);
  const uint32_t *tc = reinterpret_cast<const uint32_t *>(S.block + T.triC);
  for (int k = threadIdx.x; k < T.nt; k += nthr) {
    const float4 a = ta[k];
    const uint4 b = tb[k];
    const uint32_t iv = tc[k];
    const int ed[3] = {static_cast<int>(b.w & 1023u), static_cast<int>(b.w >> 10 & 1023u),
                       static_cast<int>(b.w >> 20)};
    const int cv[3] = {static_cast<int>(iv & 1023u), static_cast<int>(iv >> 10 & 1023u),
                       static_cast<int>(iv >> 20)};
    const float circ[3] = {a.x, a.y, a.z};
    const float kite[3] = {__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z)};
    tri_core<NoWait>(k, ed, cv, circ, kite, a.w, S.sh, S.su, S.sq, h_ref, pv_on, flags);
  }
}

// Bernoulli potential and PV-flux terms of the tile's cells; the own cells'
// depth.  For an own cell, cell(slot words, ue, kd, meta, bt, inva, new depth)
// may do more with what was gathered.
struct NoCell {
  template <class... P>
  __device__ __forceinline__ void operator()(const P &...) const {}
};
template <int nthr, class V, class Cell = NoCell>
__device__ __forceinline__ void tile_cells(const Tile &T, const TileSharedOf<V> &S,
                                           const TileFields &F, const TileOwn<nthr, V> &own,
                                           int stage, float dt, float grav, float h_ref,
                                           Cell cell = Cell{}) {
  const int tid = threadIdx.x;
  if (tid >= T.nz) return;
  const uint4 *slot = reinterpret_cast<const uint4 *>(S.block + T.slot) + tid;
  float R[6];
  V ue[6], hn[6], qt[6];
  float2 kd[6];
  uint32_t word[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const uint4 s = slot[j * T.nz];
    word[j] = s.x;
    ue[j] = S.su[s.x & 1023u];
    hn[j] = S.sh[s.x >> 10 & 1023u];
    qt[j] = S.sq[s.x >> 20];
    R[j] = __uint_as_float(s.y);
    kd[j] = make_float2(__uint_as_float(s.z), __uint_as_float(s.w));
  }
  const uint32_t meta = reinterpret_cast<const uint32_t *>(S.block + T.meta)[tid];
  const float bt = reinterpret_cast<const float *>(S.block + T.bt)[tid];
  const bool mine = tid < T.nc;
  const float inva = mine ? reinterpret_cast<const float *>(S.block + T.inva)[tid] : 0.0f;
  const V div = cell_terms(tid, meta, R, kd, ue, hn, qt, S.sh[tid], bt, inva, S.sb, S.sz, grav,
                           h_ref);
  if (!mine) return;
  const V masseq = vmul(div, all<V>(-inva));
  if (stage < 0) {
    tile_store(F.tend_h, T.c0 + tid, F.mh, masseq);
    cell(word, ue, kd, meta, bt, inva, 0.0f);
  } else {
    V a = own.ach;
    const V hnew = rk_stage32(stage, masseq, own.ynh, &a, dt);
    tile_store(F.h_out, T.c0 + tid, F.mh, hnew);
    if (stage < 3) tile_store(F.acc_h, T.c0 + tid, F.mh, a);
    cell(word, ue, kd, meta, bt, inva, hnew);
  }
}

// the own edges' velocity; force(k, cell 1, cell 2, 1 / (l erad)) is added to
// the momentum tendency of own edge k (cells by local number)
struct NoForce {
  __device__ __forceinline__ float operator()(int, int, int, float) const { return 0.0f; }
};
template <int nthr, class V, class Force = NoForce>
__device__ __forceinline__ void tile_edges(const Tile &T, const TileSharedOf<V> &S,
                                           const TileFields &F, const TileOwn<nthr, V> &own,
                                           int stage, float dt, float erad, int mom_on,
                                           Force force = Force{}) {
  const int tid = threadIdx.x;
  const uint2 *edge = reinterpret_cast<const uint2 *>(S.block + T.edge);
  auto tendency = [&](int k) -> V {
    const uint2 w = edge[k];
    const int c1 = w.x & 1023u, c2 = w.x >> 13 & 1023u;
    const float g = __uint_as_float(w.y);
    V m = edge_terms(S.sb[c1], S.sb[c2], S.sz[6 * c1 + (w.x >> 10 & 7u)],
                     S.sz[6 * c2 + (w.x >> 23)], g, erad);
    if constexpr (!std::is_same<Force, NoForce>::value) m += force(k, c1, c2, g);
    return mom_on ? m : all<V>(0.0f);
  };
  auto update = [&](int k, V m, V yn, V ac) {
    const int e = T.e0 + k;
    if (stage < 0) {
      tile_store(F.tend_u, e, F.mu, m);
    } else {
      tile_store(F.u_out, e, F.mu, rk_stage32(stage, m, yn, &ac, dt));
      if (stage < 3) tile_store(F.acc_u, e, F.mu, ac);
    }
  };
  // all reads of the rounds before their writes, which could alias them for
  // all the compiler knows
  constexpr int kE = TileOwn<nthr, V>::kE;
  V m[kE];
#pragma unroll
  for (int r = 0; r < kE; ++r)
    m[r] = tid + r * nthr < T.ne ? tendency(tid + r * nthr) : all<V>(0.0f);
#pragma unroll
  for (int r = 0; r < kE; ++r)
    if (tid + r * nthr < T.ne) update(tid + r * nthr, m[r], own.ynu[r], own.acu[r]);
  for (int k = tid + kE * nthr; k < T.ne; k += nthr)
    update(k, tendency(k), stage >= 0 ? tile_load<V>(F.yn_u, T.e0 + k, F.mu) : all<V>(0.0f),
           stage >= 1 ? tile_load<V>(F.acc_u, T.e0 + k, F.mu) : all<V>(0.0f));
}

}  // namespace imodel
