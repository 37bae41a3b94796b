// Batched ensembles: several grids, each with several members, advanced by
// one persistent cooperative launch (FP32, cell-centred TRSK).
//
// The kernel loops over "macro steps": the grid with the most steps steps
// every time, the others are spread evenly over the same macro steps.  An RK
// stage is one pass over work items, a tile of a grid (swm_layout.h) for one
// member or two: the block fetches the tile's records into shared memory and
// steps the members' tile there, as the fused stage of a single run does
// (swm_tile.cuh, with the same bits).  No intermediate field goes through
// memory and one grid-wide barrier ends the stage; the barrier's wait is
// bounded and reports a timeout through the error flag instead of waiting
// forever.  Each member's state is stored like a single run's.
//
// What bounds a stage is the issue of a tile's instructions and the latency
// of its phases (a stage of few items: the barrier), so two members are
// stepped together in packed arithmetic (swm_pair.cuh), which takes 0.7 of the
// instructions.  32 members on level 6 for 32 steps with 8 on level 7 for 64:
// 54 ms with a stage in three phases (triangles, cells, edges) over members
// interleaved in memory, 24.0 by tiles a member at a time, 19.2 by pairs,
// 6.6e9 member-cell-steps a second.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "imodel_swm.h"
#include "swm_common.cuh"
#include "swm_layout.h"
#include "swm_tile.cuh"

namespace imodel {
namespace {

constexpr int kMaxGrids = 8;

// Threads of a block, and the most cells of its tiles.  By pairs the smaller
// blocks keep more of them at different phases: 32 members on level 6 with 8 on
// level 7, 32 and 64 steps, 21.3 ms with 256 threads (two blocks an SM), 20.7
// with 192 (three), 19.4 with 128 (five).
template <class V>
constexpr int kEnsThreads = 256;
template <>
constexpr int kEnsThreads<Pair> = 128;

struct GridDev {
  TileDev tiles;
  int nv, ne;
  int members, group, ngroups;  // members per work item (1 or 2), items per tile
  float h_ref, grav, erad;
  int nsteps;  // steps this launch
  float dt;
  // [members][nv] and [members][ne]
  float *yn_h, *yn_u, *ya_h, *ya_u, *yb_h, *yb_u, *acc_h, *acc_u;
};

struct EnsArgs {
  int ngrids;
  int macro_steps;
  int pv_on, mom_on;
  int single;  // no grid has more than one member
  GridDev g[kMaxGrids];
  int smem_block, smem_h, smem_u, smem_t;  // shared memory: the largest tile's sizes
  unsigned *bar_count;
  int *flags;  // bit 0: PV division by ~0, bit 2: barrier timed out, bit 32: copy timed out
  // test hook: block stall_block (-1: none) leaves before its first
  // barrier; spin_limit bounds every barrier wait (polls of ~64 ns)
  int stall_block;
  unsigned long long spin_limit;
};

// grid-wide barrier number `epoch` (0, 1, ...) with a bounded wait
// (cooperative launch: all blocks are resident).  The counter only grows, so
// the arrival that completes the barrier is also what the others poll.  The
// fences order the block's writes before its arrival and, behind the wait,
// drop the SM's L1 lines, so plain loads after the barrier see every block's
// writes.  Returns false, with bit 2 of *flags set, if it gave up.
__device__ bool grid_barrier(const EnsArgs &A, unsigned epoch) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    const unsigned target = (epoch + 1) * gridDim.x;
    atomicAdd(A.bar_count, 1u);
    const volatile unsigned *count = A.bar_count;
    unsigned long long spins = 0;
    // wraps with the counter: fewer than 2^31 arrivals apart
    while (static_cast<int>(*count - target) < 0) {
      if (++spins > A.spin_limit) {  // 2^26: several seconds; a phase takes < 10 ms
        atomicOr(A.flags, 4);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ bool steps_now(int s, int n, int S) {
  // grid with n of S macro steps steps at s iff floor((s+1)n/S) > floor(s n/S)
  return (static_cast<long long>(s + 1) * n) / S > (static_cast<long long>(s) * n) / S;
}

// item number r of a stage (grids in `on`, tile by tile, members innermost)
struct Item {
  int k, tile, m;
  __device__ __forceinline__ Item(const EnsArgs &A, unsigned on, int r) {
    for (k = 0;; ++k) {
      if (!(on >> k & 1u)) continue;
      const int n = A.g[k].tiles.ntiles * A.g[k].ngroups;
      if (r < n) break;
      r -= n;
    }
    tile = r / A.g[k].ngroups;
    m = (r - tile * A.g[k].ngroups) * A.g[k].group;
  }
};

__device__ __forceinline__ TileFields member_fields(const GridDev &G, int st, int m) {
  const size_t oh = static_cast<size_t>(m) * G.nv, ou = static_cast<size_t>(m) * G.ne;
  TileFields F;
  F.hd = (st == 0 ? G.yn_h : (st == 2 ? G.yb_h : G.ya_h)) + oh;
  F.u = (st == 0 ? G.yn_u : (st == 2 ? G.yb_u : G.ya_u)) + ou;
  F.h_out = (st == 0 ? G.ya_h : (st == 1 ? G.yb_h : (st == 2 ? G.ya_h : G.yn_h))) + oh;
  F.u_out = (st == 0 ? G.ya_u : (st == 1 ? G.yb_u : (st == 2 ? G.ya_u : G.yn_u))) + ou;
  F.yn_h = G.yn_h + oh;
  F.yn_u = G.yn_u + ou;
  F.acc_h = G.acc_h + oh;
  F.acc_u = G.acc_u + ou;
  F.tend_h = F.tend_u = nullptr;
  // a member alone is stepped as both of a pair
  const bool two = G.group == 2 && m + 1 < G.members;
  F.mh = two ? G.nv : 0;
  F.mu = two ? G.ne : 0;
  return F;
}

// V: float, a member at a time, or Pair, two
template <class V>
__global__ void __launch_bounds__(kEnsThreads<V>, std::is_same<V, Pair>::value ? 5 : 3)
    k_ensemble(EnsArgs A) {
  constexpr int kThr = kEnsThreads<V>;
  constexpr bool kPair = std::is_same<V, Pair>::value;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint64_t mbar;
  if (static_cast<int>(blockIdx.x) == A.stall_block) return;  // test hook
  if (threadIdx.x == 0) tc05::mbar_init(&mbar, 1);
  TileSharedOf<V> S;
  S.block = smem;
  S.sh = reinterpret_cast<V *>(smem + A.smem_block);
  S.su = S.sh + A.smem_h;
  S.sq = S.su + A.smem_u;
  S.sb = S.sq + A.smem_t;
  S.sz = S.sb + kThr;
  __syncthreads();
  uint32_t parity = 0;
  unsigned epoch = 0;
  int held = -1;  // block (Tile) of the records in shared memory, of grid held_k
  int held_k = -1;
  for (int s = 0; s < A.macro_steps; ++s) {
    unsigned on = 0;
    int total = 0;
    for (int k = 0; k < A.ngrids; ++k)
      if (steps_now(s, A.g[k].nsteps, A.macro_steps)) {
        on |= 1u << k;
        total += A.g[k].tiles.ntiles * A.g[k].ngroups;
      }
    // the block's share: a tile's members follow one another, for its records;
    // single members are dealt out, for the neighbours' state in the L2 (one
    // member on level 7 with one on level 8: 458 -> 430 us a step)
    int r0 = blockIdx.x, r1 = total, dr = gridDim.x;
    if (!A.single) {
      r0 = static_cast<int>(static_cast<long long>(total) * blockIdx.x / gridDim.x);
      r1 = static_cast<int>(static_cast<long long>(total) * (blockIdx.x + 1) / gridDim.x);
      dr = 1;
    }
    for (int st = 0; st < 4; ++st) {
      for (int r = r0; r < r1; r += dr) {
        const Item I(A, on, r);
        const GridDev &G = A.g[I.k];
        const Tile T(G.tiles.head + 5 * I.tile);
        const TileFields F = member_fields(G, st, I.m);
        const bool fresh = held != T.block || held_k != I.k;
        if (fresh && threadIdx.x == 0) {
          // the last tile's records have been read (barrier below); order
          // those reads before the copy's writes
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          bulk_load(smem, G.tiles.data + T.block, T.bytes, &mbar);
        }
        held = T.block;
        held_k = I.k;
        TileOwn<kThr, V> own;
        own.template load<!kPair>(T, F, st);
        if (fresh) {
          if (!tc05::mbar_wait<2>(&mbar, parity, A.flags, 32)) return;
          parity ^= 1u;
        }
        own.rim(T, F, S);
        own.store(T, F, S);
        __syncthreads();
        tile_triangles<kThr>(T, S, G.h_ref, A.pv_on, A.flags);
        __syncthreads();
        tile_cells(T, S, F, own, st, G.dt, G.grav, G.h_ref);
        // by pairs there are no registers to hold these over the cells
        if (kPair) own.load_edges(T, F, st);
        __syncthreads();
        tile_edges(T, S, F, own, st, G.dt, G.erad, A.mom_on);
        // another tile's records may come over these; the edges read neither
        // depths nor velocities
        __syncthreads();
      }
      if (!grid_barrier(A, epoch++)) return;
    }
  }
}

// a member's fields <-> reference-ordered FP64 arrays
__global__ void k_ens_gather(int n, const int32_t *__restrict__ n2o,
                             const double *__restrict__ src, float *__restrict__ dst, double shift) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = static_cast<float>(src[n2o[i]] - shift);
}
__global__ void k_ens_scatter(int n, const int32_t *__restrict__ n2o,
                              const float *__restrict__ src, double *__restrict__ dst,
                              double shift, int *flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const double v = static_cast<double>(src[i]) + shift;
    dst[n2o[i]] = v;
    if (!isfinite(v)) atomicOr(flags, 2);
  }
}

struct GridHost {
  int nv = 0, ne = 0, nt = 0, members = 0;
  bool href_fixed = false;
  double h_ref = 0.0;
  std::vector<double> areag;  // reference order
  int32_t *cell_n2o = nullptr, *edge_n2o = nullptr;
  GridDev dev{};
};

struct Ens {
  std::string err;
  int device = 0;
  int testcase = 2;
  int ngrids = 0;
  GridHost g[kMaxGrids];
  std::vector<void *> allocs;
  double *stage_h = nullptr, *stage_u = nullptr;
  unsigned *bar = nullptr;  // arrivals at the grid-wide barriers
  int *flags = nullptr;
  int *h_flags = nullptr;
  cudaStream_t stream = nullptr;
  int blocks_per_sm = 0;  // 0: as many as fit
  bool pairs = false;     // members two at a time
  size_t smem = 0;
  EnsArgs args{};         // the parts that stay: sizes, members
  bool any_state = false;
  // test hook for the next launch only (imodel_swm_ensemble_test_stall)
  int test_stall_block = -1;
  unsigned long long test_spin_limit = 0;
};

int fail(Ens *E, int code, const std::string &m) {
  E->err = m;
  return code;
}

#define EK(call)                                                                   \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess)                                                         \
      return imodel::fail(E, e_ == cudaErrorMemoryAllocation ? IMODEL_SWM_ENOMEM : IMODEL_SWM_ECUDA, \
                  std::string(#call) + ": " + cudaGetErrorString(e_));             \
  } while (0)

template <class V, class A>
int up(Ens *E, const std::vector<V, A> &v, const V **dst) {
  void *p = nullptr;
  EK(cudaMalloc(&p, (v.empty() ? 1 : v.size()) * sizeof(V)));
  E->allocs.push_back(p);
  if (!v.empty()) EK(cudaMemcpy(p, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice));
  *dst = static_cast<const V *>(p);
  return IMODEL_SWM_OK;
}

// zero-filled on s, the stream that uses the buffer first (the tiles' blocks are
// written on the default stream, behind the uploads)
template <class T>
int zalloc(Ens *E, T **p, size_t n, cudaStream_t s) {
  void *q = nullptr;
  EK(cudaMalloc(&q, (n ? n : 1) * sizeof(T)));
  E->allocs.push_back(q);
  EK(cudaMemsetAsync(q, 0, (n ? n : 1) * sizeof(T), s));
  *p = static_cast<T *>(q);
  return IMODEL_SWM_OK;
}

// the tiles' blocks, from a copy of the layout's arrays that is not kept: in one
// allocation, as getting and freeing each of the twelve took longer than all
// copies
int fill_tiles(Ens *E, const Layout &L, const TileLayout &T, const int4 *head, uint4 *data) {
  size_t bytes = 0;
  auto place = [&bytes](size_t n) {  // 256-byte aligned, as cudaMalloc would
    const size_t at = bytes;
    bytes += (n + 255) & ~static_cast<size_t>(255);
    return at;
  };
  auto size = [](const auto &v) { return v.size() * sizeof(v[0]); };
  const size_t ra = place(size(L.t_recA)), rb = place(size(L.t_recB)), rc = place(size(L.t_recC)),
               f = place(size(L.t_f32)), meta = place(size(L.c_meta)),
               inva = place(size(L.c_inva32)), bt = place(sizeof(float) * L.nv),
               gr = place(size(L.e_grad32)), pk = place(size(L.c_pk)), kd = place(size(L.c_kd)),
               vs2 = place(size(L.e_vs2)), li = place(size(T.lists));
  char *p = nullptr;
  EK(cudaMalloc(&p, bytes));
  cudaError_t e = cudaMemsetAsync(p + bt, 0, sizeof(float) * L.nv, nullptr);
  auto copy = [&](size_t at, const auto &v) {
    if (e == cudaSuccess) e = cudaMemcpy(p + at, v.data(), size(v), cudaMemcpyHostToDevice);
  };
  copy(ra, L.t_recA);
  copy(rb, L.t_recB);
  copy(rc, L.t_recC);
  copy(f, L.t_f32);
  copy(meta, L.c_meta);
  copy(inva, L.c_inva32);
  copy(gr, L.e_grad32);
  copy(pk, L.c_pk);
  copy(kd, L.c_kd);
  copy(vs2, L.e_vs2);
  copy(li, T.lists);
  if (e == cudaSuccess) {
    DevMesh M;
    std::memset(&M, 0, sizeof(M));
    M.nv = L.nv;
    M.ne = L.ne;
    M.nt = L.nt;
    M.t_recA = reinterpret_cast<const int4 *>(p + ra);
    M.t_recB = reinterpret_cast<const int4 *>(p + rb);
    M.t_recC = reinterpret_cast<const float4 *>(p + rc);
    M.t_f32 = reinterpret_cast<const float *>(p + f);
    M.c_meta = reinterpret_cast<const uint32_t *>(p + meta);
    M.c_inva32 = reinterpret_cast<const float *>(p + inva);
    M.c_bt32 = reinterpret_cast<const float *>(p + bt);
    M.e_grad32 = reinterpret_cast<const float *>(p + gr);
    M.c_pk = reinterpret_cast<const int4 *>(p + pk);
    M.c_kd = reinterpret_cast<const float2 *>(p + kd);
    M.e_vs2 = reinterpret_cast<const uint2 *>(p + vs2);
    launch_fill_tiles(M, T.ntiles, head, reinterpret_cast<const int32_t *>(p + li), data, nullptr);
    e = cudaGetLastError();
  }
  const cudaError_t g = cudaFree(p);  // waits for the kernel
  EK(e);
  EK(g);
  return IMODEL_SWM_OK;
}

using EnsKernel = void (*)(EnsArgs);
EnsKernel kernel(const Ens *E) { return E->pairs ? k_ensemble<Pair> : k_ensemble<float>; }
int threads(const Ens *E) { return E->pairs ? kEnsThreads<Pair> : kEnsThreads<float>; }

int ens_create(Ens *E, const imodel_swm_mesh *meshes, int ngrids, const int32_t *members) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return fail(E, IMODEL_SWM_ENODEV, "no CUDA device");
  if (E->device < 0 || E->device >= ndev) return fail(E, IMODEL_SWM_EINVAL, "bad device ordinal");
  EK(cudaSetDevice(E->device));
  EK(cudaStreamCreateWithFlags(&E->stream, cudaStreamNonBlocking));
  E->ngrids = ngrids;
  size_t maxn = 0;
  int rc;
  int64_t cells = 0, paired = 0;
  for (int k = 0; k < ngrids; ++k) {
    const int64_t nv = std::max(0, meshes[k].nv), m = std::max(0, members[k]);
    cells += nv * m;
    paired += nv * (m + m % 2);
  }
  // Two members at a time where there are tiles enough for every block, unless
  // a third of what is stepped would be members alone.  us a step of the first
  // grid, by pairs and singly: 4 members on level 4 with 2 on level 5 45, 40;
  //  8 with 4 52, 58; 16 with 8 62, 70; 3 on level 6 with 3 on level 7
  // 232, 244; 3 on level 6 with 1 on level 7 154, 115.
  E->args.single = 1;
  for (int k = 0; k < ngrids; ++k)
    if (members[k] > 1) E->args.single = 0;
  E->pairs = cells >= 60000 && 3 * paired <= 4 * cells;
  const int cap = std::min(tile_cap(static_cast<int>(std::min<int64_t>(cells, INT32_MAX))),
                           threads(E));
  for (int k = 0; k < ngrids; ++k) {
    if (members[k] < 1) return fail(E, IMODEL_SWM_EINVAL, "every grid needs at least one member");
    Layout L;
    std::string msg = build_layout(meshes[k], nullptr, L);
    if (!msg.empty()) return fail(E, IMODEL_SWM_EINVAL, "grid " + std::to_string(k) + ": " + msg);
    const size_t M = members[k];
    if ((static_cast<size_t>(L.ne) * M) > static_cast<size_t>(0x7FFFFFFF / 8) ||
        (static_cast<size_t>(L.nv) * 6 * M) > static_cast<size_t>(0x7FFFFFFF / 2))
      return fail(E, IMODEL_SWM_EINVAL, "grid " + std::to_string(k) + ": too many members");
    GridHost &G = E->g[k];
    G.nv = L.nv;
    G.ne = L.ne;
    G.nt = L.nt;
    G.members = members[k];
    G.areag.assign(meshes[k].hx_areag, meshes[k].hx_areag + L.nv);
    maxn = std::max(maxn, static_cast<size_t>(std::max(L.nv, L.ne)));
    GridDev &W = G.dev;
    W.nv = L.nv;
    W.ne = L.ne;
    W.members = G.members;
    W.group = E->pairs ? 2 : 1;
    W.ngroups = (W.members + W.group - 1) / W.group;
    W.grav = static_cast<float>(L.grav);
    W.erad = static_cast<float>(L.erad);
    // a tile's limits shrink with its size: one of these always fits
    TileLayout T;
    bool fits = false;
    for (int c : {cap, 128, 64})
      if (!fits && c <= cap) fits = build_tiles(L, c, T);
    if (!fits) return fail(E, IMODEL_SWM_EINVAL, "grid " + std::to_string(k) + ": no tiling");
    TileDev &D = W.tiles;
    D.cap = T.cap;
    D.ntiles = T.ntiles;
    const TileHead *head = nullptr;
    uint4 *data = nullptr;
    const int32_t *cn2o = nullptr, *en2o = nullptr;
    if ((rc = up(E, T.head, &head)) || (rc = zalloc(E, &data, T.data_bytes / sizeof(uint4), nullptr)) ||
        (rc = up(E, L.cell_n2o, &cn2o)) || (rc = up(E, L.edge_n2o, &en2o)))
      return rc;
    D.head = reinterpret_cast<const int4 *>(head);
    D.data = data;
    if ((rc = fill_tiles(E, L, T, D.head, data))) return rc;
    G.cell_n2o = const_cast<int32_t *>(cn2o);
    G.edge_n2o = const_cast<int32_t *>(en2o);
    EnsArgs &A = E->args;
    A.smem_block = std::max(A.smem_block, T.max_bytes);
    A.smem_h = std::max(A.smem_h, T.max_h);
    A.smem_u = std::max(A.smem_u, T.max_u);
    A.smem_t = std::max(A.smem_t, T.max_t);
    float **bv[] = {&W.yn_h, &W.ya_h, &W.yb_h, &W.acc_h};
    for (float **b : bv)
      if ((rc = zalloc(E, b, static_cast<size_t>(L.nv) * M, E->stream))) return rc;
    float **be[] = {&W.yn_u, &W.ya_u, &W.yb_u, &W.acc_u};
    for (float **b : be)
      if ((rc = zalloc(E, b, static_cast<size_t>(L.ne) * M, E->stream))) return rc;
  }
  EnsArgs &A = E->args;
  E->smem = A.smem_block + (E->pairs ? sizeof(Pair) : sizeof(float)) *
                               (static_cast<size_t>(A.smem_h) + A.smem_u + A.smem_t +
                                7 * threads(E));
  constexpr int kMost = 227 * 1024 - 1024;
  if (E->smem > kMost) return fail(E, IMODEL_SWM_EINVAL, "a tile does not fit an SM");
  EK(cudaFuncSetAttribute(kernel(E), cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  if ((rc = zalloc(E, &E->stage_h, maxn, E->stream)) ||
      (rc = zalloc(E, &E->stage_u, maxn, E->stream)) ||
      (rc = zalloc(E, &E->bar, 1, E->stream)) || (rc = zalloc(E, &E->flags, 1, E->stream)))
    return rc;
  EK(cudaMallocHost(&E->h_flags, sizeof(int)));
  return IMODEL_SWM_OK;
}

int ens_flags(Ens *E) {
  EK(cudaMemcpyAsync(E->h_flags, E->flags, sizeof(int), cudaMemcpyDeviceToHost, E->stream));
  EK(cudaMemsetAsync(E->flags, 0, sizeof(int), E->stream));
  EK(cudaStreamSynchronize(E->stream));
  const int f = *E->h_flags;
  if (f & 4) return fail(E, IMODEL_SWM_ECUDA, "grid barrier timed out");
  if (f & 32) return fail(E, IMODEL_SWM_ECUDA, "the ensemble kernel gave up on a bounded wait");
  if (f & 1) return fail(E, IMODEL_SWM_EDIVZERO, "division by zero in PV (|h_tr| < eps/1e5)");
  if (f & 2) return fail(E, IMODEL_SWM_EBLOWUP, "state holds NaN or Inf");
  return IMODEL_SWM_OK;
}

int ens_launch(Ens *E, const double *dt, const int32_t *nsteps, int bps) {
  EnsArgs A = E->args;
  A.ngrids = E->ngrids;
  A.pv_on = E->testcase >= 2 ? 1 : 0;
  A.mom_on = E->testcase > 1 ? 1 : 0;
  int S = 0;
  for (int k = 0; k < E->ngrids; ++k) {
    if (nsteps[k] < 0 || !std::isfinite(dt[k])) return fail(E, IMODEL_SWM_EINVAL, "bad dt or nsteps");
    A.g[k] = E->g[k].dev;
    A.g[k].nsteps = nsteps[k];
    A.g[k].dt = static_cast<float>(dt[k]);
    A.g[k].h_ref = static_cast<float>(E->g[k].h_ref);
    S = std::max(S, static_cast<int>(nsteps[k]));
  }
  if (S == 0) return IMODEL_SWM_OK;
  A.macro_steps = S;
  A.bar_count = E->bar;
  A.flags = E->flags;
  A.stall_block = E->test_stall_block;
  A.spin_limit = E->test_spin_limit ? E->test_spin_limit : (1ull << 26);
  E->test_stall_block = -1;
  E->test_spin_limit = 0;
  int dev = E->device, sms = 0, coop = 0, occ = 0;
  EK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  EK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) return fail(E, IMODEL_SWM_ECUDA, "device does not support cooperative launch");
  EK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel(E), threads(E), E->smem));
  if (occ < 1) return fail(E, IMODEL_SWM_ECUDA, "ensemble kernel does not fit an SM");
  const int per_sm = (bps > 0 && bps <= occ) ? bps : occ;
  EK(cudaMemsetAsync(E->bar, 0, sizeof(unsigned), E->stream));
  void *args[] = {&A};
  EK(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel(E)), dim3(sms * per_sm),
                                 dim3(threads(E)), args, E->smem, E->stream));
  return IMODEL_SWM_OK;
}

}  // namespace
}  // namespace imodel

using imodel::Ens;

extern "C" {

int imodel_swm_ensemble_create(const imodel_swm_mesh *meshes, int32_t ngrids,
                               const int32_t *members, int32_t testcase, int32_t device,
                               void **ens) {
  if (!ens) return IMODEL_SWM_EINVAL;
  *ens = nullptr;
  Ens *E = new (std::nothrow) Ens();
  if (!E) return IMODEL_SWM_ENOMEM;
  *ens = E;
  if (!meshes || !members || ngrids < 1 || ngrids > imodel::kMaxGrids)
    return imodel::fail(E, IMODEL_SWM_EINVAL, "need 1..8 grids with member counts");
  E->device = device;
  E->testcase = testcase;
  try {
    return imodel::ens_create(E, meshes, ngrids, members);
  } catch (const std::bad_alloc &) {
    return imodel::fail(E, IMODEL_SWM_ENOMEM, "host allocation failed");
  }
}

int imodel_swm_ensemble_set_state(void *ens, int32_t grid, int32_t member, const double *h,
                                  const double *u) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E || !h || !u || grid < 0 || grid >= E->ngrids) return IMODEL_SWM_EINVAL;
  imodel::GridHost &G = E->g[grid];
  if (member < 0 || member >= G.members) return imodel::fail(E, IMODEL_SWM_EINVAL, "bad member");
  if (cudaSetDevice(E->device) != cudaSuccess) return IMODEL_SWM_ECUDA;
  if (!G.href_fixed) {
    double s = 0.0, a = 0.0;
    for (int i = 0; i < G.nv; ++i) {
      a += G.areag[i];
      s += G.areag[i] * h[i];
    }
    G.h_ref = static_cast<double>(static_cast<float>(s / a));
    G.href_fixed = true;
  }
  EK(cudaMemcpyAsync(E->stage_h, h, sizeof(double) * G.nv, cudaMemcpyHostToDevice, E->stream));
  EK(cudaMemcpyAsync(E->stage_u, u, sizeof(double) * G.ne, cudaMemcpyHostToDevice, E->stream));
  imodel::k_ens_gather<<<(G.nv + 255) / 256, 256, 0, E->stream>>>(
      G.nv, G.cell_n2o, E->stage_h, G.dev.yn_h + static_cast<size_t>(member) * G.nv, G.h_ref);
  imodel::k_ens_gather<<<(G.ne + 255) / 256, 256, 0, E->stream>>>(
      G.ne, G.edge_n2o, E->stage_u, G.dev.yn_u + static_cast<size_t>(member) * G.ne, 0.0);
  EK(cudaGetLastError());
  EK(cudaStreamSynchronize(E->stream));
  E->any_state = true;
  return IMODEL_SWM_OK;
}

int imodel_swm_ensemble_get_state(void *ens, int32_t grid, int32_t member, double *h,
                                  double *u) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E || !h || !u || grid < 0 || grid >= E->ngrids) return IMODEL_SWM_EINVAL;
  imodel::GridHost &G = E->g[grid];
  if (member < 0 || member >= G.members) return imodel::fail(E, IMODEL_SWM_EINVAL, "bad member");
  if (cudaSetDevice(E->device) != cudaSuccess) return IMODEL_SWM_ECUDA;
  imodel::k_ens_scatter<<<(G.nv + 255) / 256, 256, 0, E->stream>>>(
      G.nv, G.cell_n2o, G.dev.yn_h + static_cast<size_t>(member) * G.nv, E->stage_h, G.h_ref,
      E->flags);
  imodel::k_ens_scatter<<<(G.ne + 255) / 256, 256, 0, E->stream>>>(
      G.ne, G.edge_n2o, G.dev.yn_u + static_cast<size_t>(member) * G.ne, E->stage_u, 0.0,
      E->flags);
  EK(cudaGetLastError());
  EK(cudaMemcpyAsync(h, E->stage_h, sizeof(double) * G.nv, cudaMemcpyDeviceToHost, E->stream));
  EK(cudaMemcpyAsync(u, E->stage_u, sizeof(double) * G.ne, cudaMemcpyDeviceToHost, E->stream));
  return imodel::ens_flags(E);
}

int imodel_swm_ensemble_advance(void *ens, const double *dt, const int32_t *nsteps) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E || !dt || !nsteps) return IMODEL_SWM_EINVAL;
  if (!E->any_state) return imodel::fail(E, IMODEL_SWM_ESTATE, "no state set");
  if (cudaSetDevice(E->device) != cudaSuccess) return IMODEL_SWM_ECUDA;
  int rc = imodel::ens_launch(E, dt, nsteps, E->blocks_per_sm);
  if (rc) return rc;
  return imodel::ens_flags(E);
}

int imodel_swm_ensemble_test_stall(void *ens, int32_t block, int64_t spin_limit) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E || block < 0 || spin_limit < 1) return IMODEL_SWM_EINVAL;
  E->test_stall_block = block;
  E->test_spin_limit = static_cast<unsigned long long>(spin_limit);
  return IMODEL_SWM_OK;
}

int imodel_swm_ensemble_tune(void *ens, const double *dt, int32_t nsteps, int32_t choice[3]) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E || !dt || !choice || nsteps <= 0) return IMODEL_SWM_EINVAL;
  if (!E->any_state) return imodel::fail(E, IMODEL_SWM_ESTATE, "no state set");
  if (cudaSetDevice(E->device) != cudaSuccess) return IMODEL_SWM_ECUDA;
  // save the state of every grid, time the candidates, restore
  std::vector<void *> saved;
  std::vector<size_t> sizes;
  std::vector<float *> bufs;
  for (int k = 0; k < E->ngrids; ++k) {
    imodel::GridHost &G = E->g[k];
    bufs.push_back(G.dev.yn_h);
    sizes.push_back(sizeof(float) * G.nv * G.members);
    bufs.push_back(G.dev.yn_u);
    sizes.push_back(sizeof(float) * G.ne * G.members);
  }
  for (size_t q = 0; q < bufs.size(); ++q) {
    void *p = nullptr;
    if (cudaMalloc(&p, sizes[q]) != cudaSuccess) {
      for (void *x : saved) cudaFree(x);
      return imodel::fail(E, IMODEL_SWM_ENOMEM, "tune: no room to save the state");
    }
    saved.push_back(p);
    cudaMemcpyAsync(p, bufs[q], sizes[q], cudaMemcpyDeviceToDevice, E->stream);
  }
  std::vector<int32_t> ns(E->ngrids, nsteps);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  int bbps = E->blocks_per_sm, occ = 0;
  int rc = IMODEL_SWM_OK;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, imodel::kernel(E), imodel::threads(E),
                                                E->smem);
  for (int bps = occ; bps >= 1 && rc == IMODEL_SWM_OK; --bps) {
    cudaEventRecord(e0, E->stream);
    rc = imodel::ens_launch(E, dt, ns.data(), bps);
    cudaEventRecord(e1, E->stream);
    if (rc) break;
    rc = imodel::ens_flags(E);
    float ms = 1e30f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rc == IMODEL_SWM_OK && ms < best) {
      best = ms;
      bbps = bps;
    }
  }
  for (size_t q = 0; q < bufs.size(); ++q)
    cudaMemcpyAsync(bufs[q], saved[q], sizes[q], cudaMemcpyDeviceToDevice, E->stream);
  cudaStreamSynchronize(E->stream);
  for (void *x : saved) cudaFree(x);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  E->blocks_per_sm = bbps;
  choice[0] = imodel::threads(E);
  choice[1] = bbps;
  choice[2] = 0;
  return IMODEL_SWM_OK;
}

int imodel_swm_ensemble_destroy(void *ens) {
  Ens *E = static_cast<Ens *>(ens);
  if (!E) return IMODEL_SWM_OK;
  if (E->stream) cudaStreamSynchronize(E->stream);
  for (void *p : E->allocs) cudaFree(p);
  if (E->h_flags) cudaFreeHost(E->h_flags);
  if (E->stream) cudaStreamDestroy(E->stream);
  delete E;
  return IMODEL_SWM_OK;
}

const char *imodel_swm_ensemble_last_error(void *ens) {
  Ens *E = static_cast<Ens *>(ens);
  return E ? E->err.c_str() : "NULL handle";
}

void *imodel_swm_ensemble_stream(void *ens) {
  Ens *E = static_cast<Ens *>(ens);
  return E ? static_cast<void *>(E->stream) : nullptr;
}

}  // extern "C"
