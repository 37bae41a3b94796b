// One RK stage of the FP32 cell-centred step in one kernel (trsk10).
//
// A block steps one tile of the layout (swm_layout.h): it gathers the tile's
// depths and velocities into shared memory, forms the PV of its triangles,
// then the Bernoulli potential and PV-flux terms of its cells, then the new
// velocities of its edges and depths of its cells.  PV, potential and flux
// terms of the tile's rim are formed by both tiles that need them, so no
// intermediate field goes through memory and no second launch follows.  The
// arithmetic is that of the three kernels of variant 1 (swm_k32_body.cuh),
// with the same bits.
//
// What bounds it: at level 9 HBM (about 256 B of records and 80 B of state a
// cell and stage, 6.3 TB/s measured, 0.94 of a copy's rate), where the three
// kernels move 440 B; below level 8 the latency of a block's own chain (copy,
// gather, three phases), so a block issues all loads of its thread at once
// and the copies before the wait.  Per step against the three kernels: level
// 9 738 -> 553 us, 8 189 -> 154, 7 43.7 -> 37.1, 6 24.8 -> 16.5, 5 20.9 ->
// 12.4; with the early start on every grid, eight steps a graph and short polls
// 537, 149, 33.7, 14.2, 10.5.  Loading the records into registers phase by phase and the
// state in loops instead took 982 us at level 9.
#include "imodel_swm.h"
#include "swm_layout.h"
#include "swm_moist32.cuh"
#include "swm_tile.cuh"

namespace imodel {
namespace {

// The tile's block comes in by two bulk copies that the wait for the kernel
// before does not hold back: its index lists, for the gathers, and the
// records.  Dynamic shared memory: the block, then depths, velocities, PV,
// potential; the flux terms take the place of the triangles' records, which
// are read by then.
template <int kStage, int kThr>
__global__ void __launch_bounds__(kThr, kThr == 256 ? 3 : 4)
    k_stage32(TileDev D, const float *__restrict__ hd, const float *__restrict__ u,
              const float *__restrict__ yn_h, float *__restrict__ acc_h,
              float *__restrict__ h_out, const float *__restrict__ yn_u,
              float *__restrict__ acc_u, float *__restrict__ u_out, float *__restrict__ tend_h,
              float *__restrict__ tend_u, float dt, float grav, float erad,
              float h_ref, int pv_on, int mom_on, int *flags) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint64_t mbar[2];
  const Tile T(D.head + 5 * blockIdx.x);
  if (threadIdx.x == 0) {
    const unsigned char *src = reinterpret_cast<const unsigned char *>(D.data + T.block);
    tc05::mbar_init(&mbar[0], 1);
    tc05::mbar_init(&mbar[1], 1);
    if (T.slot > 0) bulk_load(smem, src, T.slot, &mbar[0]);
    bulk_load(smem + T.slot, src + T.slot, T.bytes - T.slot, &mbar[1]);
  }
  TileShared S;
  S.block = smem;
  S.sh = reinterpret_cast<float *>(smem + D.max_bytes);
  S.su = S.sh + D.max_h;
  S.sq = S.su + D.max_u;
  S.sb = S.sq + D.max_t;
  S.sz = reinterpret_cast<float *>(smem + T.triA);
  after_prior<true, true>(hd, u, yn_h, acc_h, h_out, yn_u, acc_u, u_out, tend_h, tend_u);
  const TileFields F{hd, u, yn_h, yn_u, acc_h, acc_u, h_out, u_out, tend_h, tend_u};
  TileOwn<kThr> own;
  own.load(T, F, kStage);
  __syncthreads();  // the barriers are initialised
  // (without its lists the block still waits for its records)
  if (T.slot > 0 && tc05::mbar_wait<2, true>(&mbar[0], 0, flags, 32)) own.rim(T, F, S);
  own.store(T, F, S);
  if (!tc05::mbar_wait<2, true>(&mbar[1], 0, flags, 32)) return;
  __syncthreads();
  tile_triangles<kThr>(T, S, h_ref, pv_on, flags);
  __syncthreads();
  tile_cells(T, S, F, own, kStage, dt, grav, h_ref);
  __syncthreads();
  tile_edges(T, S, F, own, kStage, dt, erad, mom_on);
}

// ---- the moist stage ---------------------------------------------------------
// The same stage with the moist model's terms (moist_swm.f90:1151-1353; the
// separate kernels are in swm_moist.cu): the tracers' values come into shared
// memory beside the depths, an own cell adds up their fluxes over the slots it
// has gathered and forms the water sources, an own edge the thermal momentum
// source.  After the last stage the own cells also form qv, qc, qr, which no
// other cell reads.  In place of the tendency written and read back, two more
// kernels that fetch indices, depths and velocities again and a third at the
// end of the step: level 8 376 -> 280 us a step, and 253 with the registers
// held to three blocks on an SM (a few bytes spilled).
template <int kStage, int kThr>
__global__ void __launch_bounds__(kThr, 3)
    k_moist_stage32(TileDev D, MoistArgs32 A, float grav, float erad, int pv_on, int mom_on) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint64_t mbar[2];
  constexpr int kTr = 5;
  const int tid = threadIdx.x;
  const Tile T(D.head + 5 * blockIdx.x);
  if (tid == 0) {
    const unsigned char *src = reinterpret_cast<const unsigned char *>(D.data + T.block);
    tc05::mbar_init(&mbar[0], 1);
    tc05::mbar_init(&mbar[1], 1);
    if (T.slot > 0) bulk_load(smem, src, T.slot, &mbar[0]);
    bulk_load(smem + T.slot, src + T.slot, T.bytes - T.slot, &mbar[1]);
  }
  TileShared S;
  S.block = smem;
  S.sh = reinterpret_cast<float *>(smem + D.max_bytes);
  S.su = S.sh + D.max_h;
  S.sq = S.su + D.max_u;
  S.sb = S.sq + D.max_t;
  S.sz = reinterpret_cast<float *>(smem + T.triA);
  float *tr = S.sb + D.cap;  // [tracers][max_h]
  const bool own_cell = tid < T.nc;
  const int c = T.c0 + tid;
  // fixed in a run
  const float q0ex = own_cell ? A.q0ex[c] : 0.0f;
  float gthb[TileOwn<kThr>::kE];
#pragma unroll
  for (int r = 0; r < TileOwn<kThr>::kE; ++r)
    gthb[r] = tid + r * kThr < T.ne ? A.gthb[T.e0 + tid + r * kThr] : 0.0f;
  after_prior<true, true>();
  const TileFields F{A.h_in,  A.u_in,  A.yn_h, A.yn_u,  A.acc_h,
                     A.acc_u, A.h_out, A.u_out, nullptr, nullptr};
  TileOwn<kThr> own;
  own.load(T, F, kStage);
  float qi[kTr], qyn[kTr], qac[kTr], qv = 0.0f, qc = 0.0f;
#pragma unroll
  for (int k = 0; k < kTr; ++k) {
    qi[k] = qyn[k] = qac[k] = 0.0f;
    if (own_cell && (A.active >> k & 1)) {
      qi[k] = A.q_in[k][c];
      qyn[k] = A.q_yn[k][c];
      if (kStage >= 1) qac[k] = A.q_acc[k][c];
    }
  }
  if (own_cell) {
    qv = A.qv[c];
    qc = A.qc[c];
  }
  __syncthreads();  // the barriers are initialised
  if (T.slot > 0 && tc05::mbar_wait<2>(&mbar[0], 0, A.flags, 32)) {
    own.rim(T, F, S);
    const int32_t *hx = reinterpret_cast<const int32_t *>(smem);
    for (int q = tid; q < T.nh - T.nc; q += kThr) {
      const int i = hx[q];
#pragma unroll
      for (int k = 0; k < kTr; ++k)
        if (A.active >> k & 1) tr[k * D.max_h + T.nc + q] = A.q_in[k][i];
    }
  }
  own.store(T, F, S);
#pragma unroll
  for (int k = 0; k < kTr; ++k)
    if (own_cell && (A.active >> k & 1)) tr[k * D.max_h + tid] = qi[k];
  if (!tc05::mbar_wait<2>(&mbar[1], 0, A.flags, 32)) return;
  __syncthreads();
  tile_triangles<kThr>(T, S, A.h_ref, pv_on, A.flags);
  __syncthreads();
  auto cell = [&](const uint32_t (&word)[6], const float (&ue)[6], const float2 (&kd)[6],
                  uint32_t meta, float bt, float inva, float hnew) {
    const int n = static_cast<int>(meta & 7u);
    float hs[4];
    sources32(A.h_ref + S.sh[tid], bt, q0ex, qv, qc, A.dt, grav, hs);
    float w[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) w[j] = j < n ? ue[j] * (kd[j].y * inva) : 0.0f;
    float out[kTr];
#pragma unroll
    for (int k = 0; k < kTr; ++k) {
      out[k] = 0.0f;
      if (!(A.active >> k & 1)) continue;
      float d = 0.0f;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const float qn = tr[k * D.max_h + (word[j] >> 10 & 1023u)];
        // "upw1": the cell's own value where the flux leaves it (w > 0)
        const float qf = A.upw1 ? (w[j] > 0.0f ? qi[k] : qn) : (qi[k] + qn) * 0.5f;
        if (j < n) d += w[j] * qf;
      }
      const float t = k < 4 ? hs[k] - d : -d;
      float a = qac[k];
      out[k] = rk_stage32(kStage, t, qyn[k], &a, A.dt);
      A.q_out[k][c] = out[k];
      if (kStage < 3) A.q_acc[k][c] = a;
    }
    if (kStage == 3) {
      // scalar_elem_divide's guard
      const float hi = A.h_ref + hnew;
      if (fabsf(hi) < 1.1920928955078125e-12f) {
        atomicOr(A.flags, 1);
      } else {
        A.qv[c] = out[1] / hi;
        A.qc[c] = out[2] / hi;
        A.qr[c] = out[3] / hi;
      }
    }
  };
  tile_cells(T, S, F, own, kStage, A.dt, grav, A.h_ref, cell);
  __syncthreads();
  auto force = [&](int k, int c1, int c2, float g) {
    // own edges past kE rounds are rare: their constant is read here
    float b = 0.0f;
#pragma unroll
    for (int r = 0; r < TileOwn<kThr>::kE; ++r) b = k == tid + r * kThr ? gthb[r] : b;
    if (k >= TileOwn<kThr>::kE * kThr) b = A.gthb[T.e0 + k];
    return thermal32(S.sh[c1], S.sh[c2], tr[c1], tr[c2], A.h_ref, g, grav, b, A.flags);
  };
  tile_edges(T, S, F, own, kStage, A.dt, erad, mom_on, force);
}

// ---- the tiles' blocks -------------------------------------------------------
// position of k in the ascending list v[n], which holds it
__device__ __forceinline__ int place(const int32_t *v, int n, int k) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (v[mid] < k)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// a[0, n) ascending, by the whole block: bitonic sort in its mirrored form
// (Batcher 1968), every exchange towards ascending order, so that the places
// from n on need not exist
__device__ __forceinline__ void sort_block(int32_t *a, int n) {
  for (int k = 2; k < 2 * n; k *= 2)
    for (int j = k / 2; j > 0; j /= 2) {
      const int mask = j == k / 2 ? k - 1 : j;
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int l = i ^ mask;
        if (l > i && l < n && a[i] > a[l]) {
          const int32_t t = a[i];
          a[i] = a[l];
          a[l] = t;
        }
      }
    }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_fill_tiles(DevMesh M, const int4 *head,
                                                    const int32_t *lists, unsigned char *data) {
  // the lists (at most 1024 entries each): ring cells and other depths, other
  // edges, triangles
  __shared__ int32_t lh[1024], lu[1024], lt[1024];
  const Tile T(head + 5 * blockIdx.x);
  const int nhx = T.nh - T.nc, nux = T.nu - T.ne, nring = T.nz - T.nc;
  const int32_t *src = lists + __ldg(&head[5 * blockIdx.x + 4].w);
  unsigned char *block = data + 16 * static_cast<size_t>(T.block);
  int32_t *hx = reinterpret_cast<int32_t *>(block);
  int32_t *ux = reinterpret_cast<int32_t *>(block + T.ux);
  for (int k = threadIdx.x; k < nhx; k += blockDim.x) lh[k] = src[k];
  for (int k = threadIdx.x; k < nux; k += blockDim.x) lu[k] = src[nhx + k];
  for (int k = threadIdx.x; k < T.nt; k += blockDim.x) lt[k] = src[nhx + nux + k];
  sort_block(lh, nring);
  sort_block(lh + nring, nhx - nring);
  sort_block(lu, nux);
  sort_block(lt, T.nt);
  for (int k = threadIdx.x; k < nhx; k += blockDim.x) hx[k] = lh[k];
  for (int k = threadIdx.x; k < nux; k += blockDim.x) ux[k] = lu[k];
  // local numbers: depths own, ring, others; edges own, others
  auto cell = [&](int c) -> uint32_t {
    if (c >= T.c0 && c < T.c0 + T.nc) return c - T.c0;
    const int r = place(lh, nring, c);
    if (r < nring && lh[r] == c) return T.nc + r;
    return T.nz + place(lh + nring, nhx - nring, c);
  };
  auto edge = [&](int e) -> uint32_t {
    return e >= T.e0 && e < T.e0 + T.ne ? e - T.e0 : T.ne + place(lu, nux, e);
  };
  uint4 *ta = reinterpret_cast<uint4 *>(block + T.triA);
  uint4 *tb = reinterpret_cast<uint4 *>(block + T.triB);
  uint32_t *tc = reinterpret_cast<uint32_t *>(block + T.triC);
  for (int k = threadIdx.x; k < T.nt; k += blockDim.x) {
    const int t = lt[k];
    const int4 a = M.t_recA[t], b = M.t_recB[t];
    const float4 c = M.t_recC[t];
    ta[k] = make_uint4(b.z, b.w, __float_as_uint(c.x), __float_as_uint(M.t_f32[t]));
    tb[k] = make_uint4(__float_as_uint(c.y), __float_as_uint(c.z), __float_as_uint(c.w),
                       edge(a.x) | edge(a.y) << 10 | edge(a.z) << 20);
    tc[k] = cell(a.w) | cell(b.x) << 10 | cell(b.y) << 20;
  }
  uint4 *slot = reinterpret_cast<uint4 *>(block + T.slot);
  uint32_t *meta = reinterpret_cast<uint32_t *>(block + T.meta);
  float *bt = reinterpret_cast<float *>(block + T.bt);
  float *inva = reinterpret_cast<float *>(block + T.inva);
  for (int z = threadIdx.x; z < T.nz; z += blockDim.x) {
    const int c = z < T.nc ? T.c0 + z : lh[z - T.nc];
    meta[z] = M.c_meta[c];
    bt[z] = M.c_bt32[c];
    if (z < T.nc) inva[z] = M.c_inva32[c];
    for (int j = 0; j < 6; ++j) {
      // {edge, neighbour, triangle, kite fraction}, {KE weight, ttgout d};
      // unused slots repeat slot 0 with zero weights
      const int4 pk = M.c_pk[j * M.nv + c];
      const float2 kd = M.c_kd[j * M.nv + c];
      slot[j * T.nz + z] = make_uint4(edge(pk.x) | cell(pk.y) << 10 | place(lt, T.nt, pk.z) << 20,
                                      pk.w, __float_as_uint(kd.x), __float_as_uint(kd.y));
    }
  }
  uint2 *ed = reinterpret_cast<uint2 *>(block + T.edge);
  for (int k = threadIdx.x; k < T.ne; k += blockDim.x) {
    const uint2 w = M.e_vs2[T.e0 + k];  // cell | slot << 28 of both cells
    ed[k] = make_uint2(cell(w.x & 0x0FFFFFFF) | (w.x >> 28) << 10 | cell(w.y & 0x0FFFFFFF) << 13 |
                           (w.y >> 28) << 23,
                       __float_as_uint(M.e_grad32[T.e0 + k]));
  }
}

size_t fused_smem(const TileDev &T) {
  return static_cast<size_t>(T.max_bytes) +
         sizeof(float) * (static_cast<size_t>(T.max_h) + T.max_u + T.max_t + T.cap);
}

}  // namespace

// One tile's time on an SM hardly depends on its size, so small grids are cut
// into as many tiles as run at once (level 5: 12.4 us a step with 64, 14.4
// with 96 and more; level 6: 22.6, 16.5, 16.9 with 64, 96, 128), large ones
// into large tiles, which form and fetch less twice (level 7: 49.3 with 96,
// 43.0, 41.2 and 37.1 with 128, 192 and 256; level 9: 796, 652, 608, 551).
int tile_cap(int nv) { return nv <= 20000 ? 64 : (nv <= 100000 ? 96 : 256); }

namespace {
// the instance for a stage (-1: tendencies) and the tiles' size
using Stage32 = decltype(&k_stage32<0, 256>);
template <int kThr>
Stage32 stage_kernel(int stage) {
  switch (stage) {
    case 0: return k_stage32<0, kThr>;
    case 1: return k_stage32<1, kThr>;
    case 2: return k_stage32<2, kThr>;
    case 3: return k_stage32<3, kThr>;
    default: return k_stage32<-1, kThr>;
  }
}
inline int threads(const TileDev &T) { return T.cap <= 96 ? 192 : 256; }
inline Stage32 stage_kernel(const TileDev &T, int stage) {
  return threads(T) == 192 ? stage_kernel<192>(stage) : stage_kernel<256>(stage);
}
}  // namespace

void launch_fill_tiles(const DevMesh &M, int ntiles, const int4 *head, const int32_t *lists,
                       uint4 *data, cudaStream_t s) {
  if (ntiles > 0)
    k_fill_tiles<<<ntiles, 256, 0, s>>>(M, head, lists, reinterpret_cast<unsigned char *>(data));
}

namespace {
using MoistStage32 = decltype(&k_moist_stage32<0, 256>);
template <int kThr>
MoistStage32 moist_kernel(int stage) {
  switch (stage) {
    case 0: return k_moist_stage32<0, kThr>;
    case 1: return k_moist_stage32<1, kThr>;
    case 2: return k_moist_stage32<2, kThr>;
    default: return k_moist_stage32<3, kThr>;
  }
}
inline MoistStage32 moist_kernel(const TileDev &T, int stage) {
  return threads(T) == 192 ? moist_kernel<192>(stage) : moist_kernel<256>(stage);
}
size_t moist_smem(const TileDev &T) {
  return fused_smem(T) + 5 * sizeof(float) * static_cast<size_t>(T.max_h);
}
constexpr int kMost = 227 * 1024 - 1024;  // dynamic shared memory of a block
}  // namespace

bool fused_moist_ok(const TileDev &T) {
  if (T.ntiles == 0 || moist_smem(T) > kMost) return false;
  for (int stage = 0; stage < 4; ++stage)
    if (cudaFuncSetAttribute(moist_kernel(T, stage), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMost) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  return true;
}

void launch_moist_stage32_fused(const DevMesh &M, const Work<float> &W, const MoistArgs32 &A,
                                cudaStream_t s) {
  const TileDev &T = W.tiles;
  launch_pdl_smem(moist_kernel(T, A.stage), T.ntiles, threads(T), moist_smem(T), s, T, A,
                  static_cast<float>(M.grav), static_cast<float>(M.erad), W.pv_on, W.mom_on);
}

bool fused_prepare(const TileDev &T) {
  if (fused_smem(T) > kMost || T.cap > threads(T)) return false;
  for (int stage = -1; stage < 4; ++stage)
    if (cudaFuncSetAttribute(stage_kernel(T, stage), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMost) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  return true;
}

void launch_stage32_fused(const DevMesh &M, const Work<float> &W, const float *h_in,
                          const float *u_in, float *h_out, float *u_out, int stage, float dt,
                          cudaStream_t s) {
  const TileDev &T = W.tiles;
  launch_pdl_smem(stage_kernel(T, stage), T.ntiles, threads(T), fused_smem(T), s, T, h_in, u_in,
                  W.yn_h, W.acc_h, h_out, W.yn_u, W.acc_u, u_out, W.tend_h, W.tend_u, dt,
                  static_cast<float>(M.grav), static_cast<float>(M.erad), W.h_ref, W.pv_on,
                  W.mom_on, W.flags);
}

}  // namespace imodel
