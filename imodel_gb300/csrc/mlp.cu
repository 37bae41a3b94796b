// Per-edge MLP of the learned TRSK correction: 24 -> 64 -> 64 -> 1, GELU,
// BF16 operands with FP32 accumulation on the 5th-generation tensor cores
// (tcgen05, accumulators in TMEM), forward, backward and Adam.
//
// Parameter vector (FP32 master copy, 5825 values):
//     W1[64][24] (out-major), b1[64], W2[64][64] (out-major), b2[64], w3[64], b3
// Inputs x[n][24] are BF16 (bit patterns in uint16).
//
// Tiles of 128 rows; one thread per row.  Forward per tile (the pipelined,
// warp-specialised kernel of mlp_pipe.cuh):
//     D1 = X W1^T      (M=128, N=64, K=32: inputs padded 24 -> 32)
//     H1 = GELU(D1 + b1) -> BF16 -> shared memory
//     D2 = H1 W2^T     (M=128, N=64, K=64)
//     y  = GELU(D2 + b2) . w3 + b3   (FP32, CUDA cores)
// Backward per tile (mean squared error):
//     dZ2 = dy w3 * GELU'(Z2) -> BF16;   dH1 = dZ2 W2 (M=128, N=64, K=64)
//     dZ1 = dH1 * GELU'(Z1) -> BF16
//     one accumulating MMA per tile gives dW2, dW1, db2, db1 at once:
//     DW += AW BW^T, AW = [H1^T; X^T; ones] (128 x batch), BW = [dZ2^T; dZ1^T]
//     (128 x batch), so DW[i][o] = dW2[o][i], DW[64+i][64+o] = dW1[o][i],
//     DW[96][o] = db2[o], DW[96][64+o] = db1[o].
// dw3 and db3 are warp-shuffle sums.  Each CTA writes its partial gradient;
// a second kernel sums the partials in a fixed order (deterministic).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "imodel_mlp.h"
#include "imodel_swm.h"
#include "swm_common.cuh"
#include "tc05.cuh"

namespace imodel {
namespace {

using namespace tc05;

constexpr int NIN = 24, K1 = 32, NH = 64, TM = 128;
constexpr int OFF_W1 = 0, OFF_B1 = 1536, OFF_W2 = 1600, OFF_B2 = 5696, OFF_W3 = 5760,
              OFF_B3 = 5824;
constexpr int NPARAM = 5825;
constexpr int NPART = NPARAM + 1;  // + loss
static_assert(TM == 128, "four warps per training tile");
constexpr int ERR_WAIT = 8;

struct Weights {
  const uint16_t *w1img;   // B operand of layer 1: [64 out][32 in], K-major image
  const uint16_t *w2img;   // B operand of layer 2: [64 out][64 in]
  const uint16_t *w2timg;  // B operand of dH1:     [64 in][64 out]
  const float *p;          // FP32 master parameters
};

__device__ __forceinline__ uint16_t bf16bits(float v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
// two FP32 values -> BF16x2 (a in the low half), round to nearest even
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
// GELU in its tanh form (Hendrycks & Gimpel 2016),
//   gelu(z) = z/2 (1 + tanh(c (z + a z^3))),  c = sqrt(2/pi), a = 0.044715,
// with the tanh of the hardware's special-function unit (tanh.approx.f32).
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Evaluated as u = (c + c a z^2) z, gelu = z/2 + (z/2) tanh(u): six FP32
// operations and one tanh, the same sequence in the scalar and the packed
// (two lanes per instruction, f32x2) forms, so both give identical values.
constexpr float kGc = 0.7978845608028654f, kGca = 0.7978845608028654f * 0.044715f;
__device__ __forceinline__ float gelu(float z) {
  const float u = fmaf(z * z, kGca, kGc) * z;
  const float hz = 0.5f * z;
  return fmaf(hz, tanh_fast(u), hz);
}
__device__ __forceinline__ float gelu_tanh(float z) {
  return tanh_fast(fmaf(z * z, kGca, kGc) * z);
}
__device__ __forceinline__ float gelu_grad(float z, float th) {
  return 0.5f * (1.0f + th) +
         0.5f * z * (1.0f - th * th) * 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * z * z);
}

// ---- packed FP32 pairs (f32x2 instructions of sm_100-family GPUs) ----------
__device__ __forceinline__ uint64_t f2pk(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2upk(uint64_t r, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(r));
}
__device__ __forceinline__ uint64_t f2mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// TWICE the gelu of the pair z = (z0, z1), lane by lane:
// z + z tanh(u) = 2 gelu(z) exactly (the halving in gelu() is exact), so the
// forward kernel halves the weights that multiply it instead (W2 and w3, also
// exact) and saves one multiply per pair
__device__ __forceinline__ uint64_t gelu2x2(float z0, float z1) {
  const uint64_t z = f2pk(z0, z1);
  const uint64_t u = f2mul(f2fma(f2mul(z, z), f2pk(kGca, kGca), f2pk(kGc, kGc)), z);
  float u0, u1;
  f2upk(u, u0, u1);
  return f2fma(z, f2pk(tanh_fast(u0), tanh_fast(u1)), z);
}

// columns [c0, c0 + 32) of row `r` of a K-major 16-bit operand with `kc`
// columns, from 32 FP32 values
__device__ __forceinline__ void store_row32(uint8_t *op, int r, int c0, const float (&v)[32],
                                            int kc) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 q;
    q.x = pack2(v[8 * c + 0], v[8 * c + 1]);
    q.y = pack2(v[8 * c + 2], v[8 * c + 3]);
    q.z = pack2(v[8 * c + 4], v[8 * c + 5]);
    q.w = pack2(v[8 * c + 6], v[8 * c + 7]);
    *reinterpret_cast<uint4 *>(op + kmaj_off(r, c0 + 8 * c, kc)) = q;
  }
}

// 32 FP32 columns [col, col+32) of this thread's TMEM lane
__device__ __forceinline__ void ld32(uint32_t taddr, float (&v)[32]) {
  float t[16];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    ld16(taddr + 16 * q, t);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[16 * q + i] = t[i];
  }
  wait_ld();
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__host__ __device__ __forceinline__ uint64_t splitmix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// ---- weight images ---------------------------------------------------------
__global__ void k_make_images(const float *__restrict__ p, uint16_t *w1img, uint16_t *w2img,
                              uint16_t *w2timg) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < NH * K1) {  // layer-1 B operand, zero-padded inputs 24..31
    const int o = t / K1, i = t % K1;
    const float w = i < NIN ? p[OFF_W1 + o * NIN + i] : 0.0f;
    w1img[kmaj_off(o, i, K1) / 2] = bf16bits(w);
  }
  if (t < NH * NH) {
    const int o = t / NH, i = t % NH;
    const uint16_t w = bf16bits(p[OFF_W2 + o * NH + i]);
    w2img[kmaj_off(o, i, NH) / 2] = w;   // [out][in]
    w2timg[kmaj_off(i, o, NH) / 2] = w;  // [in][out]
  }
}

// The learned correction adds corr[e] = q_e h_e sigma_e y_e, the PV flux of
// the predicted tangential error (pipe::EdgeTask).
// y is clipped to +-kCorrMax: the trained targets (error / sigma) stay below
// 0.25 for 99.9 % of the edges, and the clip bounds what an input unlike the
// training data can inject into the momentum equation.
constexpr float kCorrMax = 0.5f;
}  // namespace
}  // namespace imodel

#include "mlp_pipe.cuh"

namespace imodel {
namespace {

// ---- fused forward + backward over a batch ---------------------------------
// dynamic shared memory: B1 4K | B2 8K | B2T 8K | A2 16K | AW 36K | BW 36K.
// A1 (the inputs), A2 and A3 (dZ2) take turns in one place, each written when the
// product of the one before has been waited for: 108 KB, so that two CTAs share
// an SM (and its 512 TMEM columns) and hide each other's waits for products
// and rows.  A batch of 65,536 rows is 512 tiles: one CTA an SM took four
// rounds of them.
// AW and BW are written down their columns, two bytes a lane: their core
// matrices are 144 bytes apart along K, so that a warp's four lie in different
// banks (at 128 bytes every store took four passes).
constexpr int TRN_K = 144, TRN_ROWS = TM / 8 * TRN_K;  // strides of AW and BW
__device__ __forceinline__ uint32_t trn_off(int r, int k) {
  return static_cast<uint32_t>((r >> 3) * TRN_ROWS + (k >> 3) * TRN_K + (r & 7) * 16 + (k & 7) * 2);
}
constexpr int TRN_W = 16 * TRN_ROWS;  // bytes of AW, of BW
constexpr int TRN_SMEM = 4096 + 8192 + 8192 + 16384 + 2 * TRN_W;
constexpr int TRN_CTAS = 2;  // per SM

// Sums over the warp of 32 values a lane: lane l returns with the l-th.  Each
// exchange halves what a lane holds, 31 shuffles where a sum of its own for
// every value takes 160; the tree, and so the rounding, is the same.
__device__ __forceinline__ float warp_sum32(float (&p)[32], int lane) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      const float keep = up ? p[i + off] : p[i], send = up ? p[i] : p[i + off];
      p[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return p[0];
}

// Thread (row, half) of a tile: 32 of the 64 columns of a batch row (a warp
// reads the TMEM lanes of its number modulo four), so that the products' waits
// and the chains of a row are covered by 16 warps an SM.  Bound by latency: the
// chain of a tile's four products and what lies between them.  A step of 65,536
// rows with its reduction: 93 us with one CTA an SM, 56
// with two CTAs, 40 with the columns' stores spread over the banks, the sums by
// halves and the reduction in floats, 30.3 with two threads a row, the next rows
// read ahead and the prologue before the wait for the kernel before, 29.7 with a
// tile's last product waited for with the next tile's first.
constexpr int TRN_THREADS = 2 * TM, HALF = NH / 2;

__global__ void __launch_bounds__(TRN_THREADS, TRN_CTAS)
    k_mlp_train(Weights W, const uint16_t *__restrict__ x, const float *__restrict__ t,
                const float *__restrict__ wts,
                int64_t n, int64_t batch, uint64_t seed, float inv_batch,
                float *__restrict__ partials, int *err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *B1 = smem, *B2 = B1 + 4096, *B2T = B2 + 8192, *A2 = B2T + 8192, *AW = A2 + 16384,
          *BW = AW + TRN_W, *A3 = A2, *A1 = A2;
  __shared__ uint64_t mbar;
  __shared__ uint32_t tslot;
  __shared__ float sb1[NH], sb2[NH], sw3[NH];
  __shared__ float sy[TM];  // a row's output: first half's sum, then all
  // per-warp sums of dw3, db3 and the loss: each warp adds only to its own
  // entries, and the warps are summed in a fixed order at the end, so the
  // partial gradients do not depend on the order in which warps finish
  __shared__ float sdw3[TM / 32][NH], sdb3[TM / 32], sloss[TM / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = tid & (TM - 1), half = tid / TM, c0 = HALF * half;
  // AW rows 88..127 stay zero except row 96 (ones, for the bias sums)
  for (int i = tid; i < TRN_W / 16; i += TRN_THREADS)
    reinterpret_cast<uint4 *>(AW)[i] = make_uint4(0, 0, 0, 0);
  if (tid < NH)
    for (int k = 0; k < TM / 32; ++k) sdw3[k][tid] = 0.0f;
  if (tid < TM / 32) {
    sdb3[tid] = 0.0f;
    sloss[tid] = 0.0f;
  }
  if (tid == 0) mbar_init(&mbar, 1);
  if (warp == 0) tmem_alloc(&tslot, 256);
  const int64_t ntiles = (batch + TM - 1) / TM;
  // a tile's row of the data set, read one tile ahead
  bool live = false;
  uint4 c[3];
  float target = 0.0f, wt = 0.0f;
  auto fetch = [&](int64_t tile) {
    const int64_t pos = tile * TM + row;  // position in the batch
    live = tile < ntiles && pos < batch;
    c[0] = c[1] = c[2] = make_uint4(0, 0, 0, 0);
    target = wt = 0.0f;
    if (!live) return;
    // seed 0: rows 0..batch-1 in order; otherwise rows drawn with replacement
    const int64_t k = seed == 0 ? pos
                                : static_cast<int64_t>(splitmix(seed ^ static_cast<uint64_t>(pos)) %
                                                       static_cast<uint64_t>(n));
    const uint4 *src = reinterpret_cast<const uint4 *>(x + k * NIN);
    c[0] = src[0];
    c[1] = src[1];
    c[2] = src[2];
    target = t[k];
    wt = wts ? wts[k] : 1.0f;  // sample weight
  };
  fetch(blockIdx.x);
  // the weights come from the kernel before
  after_prior<true>(W.p, W.w1img, W.w2img, W.w2timg, partials);
  for (int i = tid; i < 4096 / 16; i += TRN_THREADS)
    reinterpret_cast<uint4 *>(B1)[i] = reinterpret_cast<const uint4 *>(W.w1img)[i];
  for (int i = tid; i < 8192 / 16; i += TRN_THREADS) {
    reinterpret_cast<uint4 *>(B2)[i] = reinterpret_cast<const uint4 *>(W.w2img)[i];
    reinterpret_cast<uint4 *>(B2T)[i] = reinterpret_cast<const uint4 *>(W.w2timg)[i];
  }
  if (tid < NH) {
    sb1[tid] = W.p[OFF_B1 + tid];
    sb2[tid] = W.p[OFF_B2 + tid];
    sw3[tid] = W.p[OFF_W3 + tid];
  }
  const float b3 = W.p[OFF_B3];
  __syncthreads();
  if (half == 0) *reinterpret_cast<uint16_t *>(AW + trn_off(96, row)) = bf16bits(1.0f);
  fence_async_smem();
  sync_cta();
  const uint32_t tmem = tslot;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t id64 = idesc_bf16(TM, NH), id128 = idesc_bf16(TM, 128);
  uint32_t phase = 0;
  bool ok = true;
  bool first = true;
  for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
    // --- inputs: A1 (row-major); the tile before's last product may be running
    if (half == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4 *>(A1 + kmaj_off(row, 8 * q, K1)) = c[q];
      *reinterpret_cast<uint4 *>(A1 + kmaj_off(row, 24, K1)) = make_uint4(0, 0, 0, 0);
    }
    fence_async_smem();
    sync_cta();
    if (tid == 0) {
      for (int s = 0; s < K1 / 16; ++s)
        mma(tmem, smem_desc(smem_u32(A1) + 256 * s, 128, K1 * 16),
            smem_desc(smem_u32(B1) + 256 * s, 128, K1 * 16), id64, s);
      commit(&mbar);
    }
    // (this also waits for the tile before's last product)
    ok = __syncthreads_and(mbar_wait(&mbar, phase, err, ERR_WAIT)) != 0;
    phase ^= 1u;
    fence_after_sync();
    if (half == 1) {  // X^T, rows 64..87 of AW
      const uint16_t *xs = reinterpret_cast<const uint16_t *>(c);
#pragma unroll
      for (int i = 0; i < NIN; ++i)
        *reinterpret_cast<uint16_t *>(AW + trn_off(64 + i, row)) = xs[i];
    }
    const bool alive = live;
    const float aim = target, weight = wt;
    fetch(tile + gridDim.x);
    float v[HALF];
    if (ok) {  // H1 = GELU(Z1 + b1): A2 (row-major) and AW rows 0..63 (H1^T)
      ld32(tmem + lane_base + c0, v);
#pragma unroll
      for (int j = 0; j < HALF; ++j) v[j] = gelu(v[j] + sb1[c0 + j]);
      store_row32(A2, row, c0, v, NH);
#pragma unroll
      for (int j = 0; j < HALF; ++j)
        *reinterpret_cast<uint16_t *>(AW + trn_off(c0 + j, row)) = alive ? bf16bits(v[j]) : 0;
    }
    fence_async_smem();
    sync_cta();
    if (ok && tid == 0) {
      for (int s = 0; s < NH / 16; ++s)
        mma(tmem + 64, smem_desc(smem_u32(A2) + 256 * s, 128, NH * 16),
            smem_desc(smem_u32(B2) + 256 * s, 128, NH * 16), id64, s);
      commit(&mbar);
    }
    if (ok) {  // ok is uniform across the CTA
      ok = __syncthreads_and(mbar_wait(&mbar, phase, err, ERR_WAIT)) != 0;
      phase ^= 1u;
    }
    fence_after_sync();
    if (ok) {  // output, loss, dZ2
      ld32(tmem + lane_base + 64 + c0, v);
      float h2[HALF];
      float yv = b3;
#pragma unroll
      for (int j = 0; j < HALF; ++j) {
        const float z = v[j] + sb2[c0 + j], th = gelu_tanh(z), hz = 0.5f * z;
        h2[j] = fmaf(hz, th, hz);  // gelu(z)
        v[j] = gelu_grad(z, th);
      }
      // the row's sum runs through the first half's columns, then the second's
      if (half == 0) {
#pragma unroll
        for (int j = 0; j < HALF; ++j) yv = fmaf(h2[j], sw3[j], yv);
        sy[row] = yv;
      }
      __syncthreads();
      if (half == 1) {
        yv = sy[row];
#pragma unroll
        for (int j = 0; j < HALF; ++j) yv = fmaf(h2[j], sw3[c0 + j], yv);
        sy[row] = yv;
      }
      __syncthreads();
      yv = sy[row];
      const float r = alive ? yv - aim : 0.0f;
      const float dy = 2.0f * weight * r * inv_batch;
      if (half == 0) {
        const float ls = warp_sum(weight * r * r), sdy = warp_sum(dy);
        if (lane == 0) {
          sloss[warp] += ls;
          sdb3[warp] += sdy;
        }
      }
#pragma unroll
      for (int j = 0; j < HALF; ++j) {
        h2[j] *= dy;
        v[j] = dy * sw3[c0 + j] * v[j];  // dZ2
      }
      sdw3[warp & 3][c0 + lane] += warp_sum32(h2, lane);
      store_row32(A3, row, c0, v, NH);
#pragma unroll
      for (int j = 0; j < HALF; ++j)
        *reinterpret_cast<uint16_t *>(BW + trn_off(c0 + j, row)) = bf16bits(v[j]);
    }
    fence_async_smem();
    sync_cta();
    if (ok && tid == 0) {  // dH1 = dZ2 W2 into the second TMEM block
      for (int s = 0; s < NH / 16; ++s)
        mma(tmem + 64, smem_desc(smem_u32(A3) + 256 * s, 128, NH * 16),
            smem_desc(smem_u32(B2T) + 256 * s, 128, NH * 16), id64, s);
      commit(&mbar);
    }
    if (ok) {  // ok is uniform across the CTA
      ok = __syncthreads_and(mbar_wait(&mbar, phase, err, ERR_WAIT)) != 0;
      phase ^= 1u;
    }
    fence_after_sync();
    if (ok) {  // dZ1 = dH1 * GELU'(Z1): BW rows 64..127
      float z1[HALF];
      ld32(tmem + lane_base + c0, z1);
      ld32(tmem + lane_base + 64 + c0, v);
#pragma unroll
      for (int j = 0; j < HALF; ++j) {
        const float z = z1[j] + sb1[c0 + j], dz1 = v[j] * gelu_grad(z, gelu_tanh(z));
        *reinterpret_cast<uint16_t *>(BW + trn_off(64 + c0 + j, row)) = bf16bits(dz1);
      }
    }
    fence_async_smem();
    sync_cta();
    if (ok && tid == 0) {  // DW += AW BW^T over the 128 batch rows of the tile
      for (int s = 0; s < TM / 16; ++s)
        mma(tmem + 128, smem_desc(smem_u32(AW) + 2 * TRN_K * s, TRN_K, TRN_ROWS),
            smem_desc(smem_u32(BW) + 2 * TRN_K * s, TRN_K, TRN_ROWS), id128,
            (first && s == 0) ? 0u : 1u);
    }
    first = false;
  }
  if (ok && !first) {  // the last tile's last product
    if (tid == 0) commit(&mbar);
    ok = __syncthreads_and(mbar_wait(&mbar, phase, err, ERR_WAIT)) != 0;
    fence_after_sync();
  }
  // partial gradients of this CTA, each half its columns
  float *out = partials + static_cast<int64_t>(blockIdx.x) * NPART;
  if (ok && !first) {
    float dw[HALF];
    // columns 0..63 of DW: rows 0..63 -> dW2^T; row 96 -> db2
    ld32(tmem + lane_base + 128 + c0, dw);
    if (row < NH) {
#pragma unroll
      for (int o = 0; o < HALF; ++o) out[OFF_W2 + (c0 + o) * NH + row] = dw[o];
    } else if (row == 96) {
#pragma unroll
      for (int o = 0; o < HALF; ++o) out[OFF_B2 + c0 + o] = dw[o];
    }
    // columns 64..127: rows 64..87 -> dW1^T; row 96 -> db1
    ld32(tmem + lane_base + 192 + c0, dw);
    if (row >= 64 && row < 64 + NIN) {
#pragma unroll
      for (int o = 0; o < HALF; ++o) out[OFF_W1 + (c0 + o) * NIN + (row - 64)] = dw[o];
    } else if (row == 96) {
#pragma unroll
      for (int o = 0; o < HALF; ++o) out[OFF_B1 + c0 + o] = dw[o];
    }
  } else if (tid < NH) {
    for (int o = 0; o < NH; ++o) out[OFF_W2 + o * NH + tid] = 0.0f;
    out[OFF_B2 + tid] = 0.0f;
    out[OFF_B1 + tid] = 0.0f;
    if (tid < NIN)
      for (int o = 0; o < NH; ++o) out[OFF_W1 + o * NIN + tid] = 0.0f;
  }
  __syncthreads();
  if (tid < NH) out[OFF_W3 + tid] = ((sdw3[0][tid] + sdw3[1][tid]) + sdw3[2][tid]) + sdw3[3][tid];
  if (tid == 0) {
    out[OFF_B3] = ((sdb3[0] + sdb3[1]) + sdb3[2]) + sdb3[3];
    out[NPARAM] = ((sloss[0] + sloss[1]) + sloss[2]) + sloss[3];
  }
  sync_cta();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// Sum of the CTAs' partial gradients in a fixed order: a block takes 32
// parameters, its warp w every kRed-th partial from w on, and the warps' sums
// are added in order, in FP64.  A warp's own sum is kept in three floats that
// take up each other's rounding errors (TwoSum, Knuth 1969): together they hold
// the sum beyond FP64's precision, and FP64 additions, two a cycle and SM here,
// bounded the kernel (16.1 us at 304 partials, 7.5 with these).  (One thread a parameter,
// 152 values in a row, took 27.)  With ADAM the parameter's update follows at
// once, and its BF16 images with it.
constexpr int kRed = 16;
struct AdamArgs {
  float *p, *m, *v, *loss;
  uint16_t *w1img, *w2img, *w2timg;
  float lr, b1, b2, eps, c1, c2;
};
// a = a + b rounded; returns the error of it
__device__ __forceinline__ float two_sum(float &a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
  a = s;
  return e;
}
template <bool ADAM>
__global__ void __launch_bounds__(32 * kRed) k_reduce(const float *__restrict__ partials, int nblk,
                                                      float *__restrict__ grad, AdamArgs A) {
  __shared__ double part[kRed][32];
  const int lane = threadIdx.x & 31, w0 = threadIdx.x >> 5, q = blockIdx.x * 32 + lane;
  after_prior<true>(partials, grad, A.p, A.m, A.v, A.loss, A.w1img, A.w2img, A.w2timg);
  double s = 0.0;
  if (q < NPART) {
    const float *p = partials + q;
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
    constexpr int kBatch = 10;  // loads in flight
    for (int b = w0; b < nblk; b += kBatch * kRed) {
      float x[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        x[k] = b + k * kRed < nblk ? p[static_cast<int64_t>(b + k * kRed) * NPART] : 0.0f;
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const float e = two_sum(s0, x[k]);
        s2 += two_sum(s1, e);
      }
    }
    s = static_cast<double>(s0) + (static_cast<double>(s1) + static_cast<double>(s2));
    if (!isfinite(s)) {  // an infinity, or a sum beyond FP32's range
      s = 0.0;
      for (int b = w0; b < nblk; b += kRed) s += p[static_cast<int64_t>(b) * NPART];
    }
  }
  part[w0][lane] = s;
  __syncthreads();
  if (w0 != 0 || q >= NPART) return;
#pragma unroll
  for (int k = 1; k < kRed; ++k) s += part[k][lane];
  const float gi = static_cast<float>(s);
  if (!ADAM) {
    grad[q] = gi;
    return;
  }
  if (q == NPARAM) {
    *A.loss = gi;
    return;
  }
  const float mi = A.b1 * A.m[q] + (1.0f - A.b1) * gi;
  const float vi = A.b2 * A.v[q] + (1.0f - A.b2) * gi * gi;
  A.m[q] = mi;
  A.v[q] = vi;
  const float w = A.p[q] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
  A.p[q] = w;
  if (q < OFF_B1) {
    A.w1img[kmaj_off(q / NIN, q % NIN, K1) / 2] = bf16bits(w);
  } else if (q >= OFF_W2 && q < OFF_B2) {
    const int o = (q - OFF_W2) / NH, i = (q - OFF_W2) % NH;
    A.w2img[kmaj_off(o, i, NH) / 2] = bf16bits(w);
    A.w2timg[kmaj_off(i, o, NH) / 2] = bf16bits(w);
  }
}

struct Mlp {
  std::string err;
  int device = 0;
  float *p = nullptr, *m = nullptr, *v = nullptr, *g = nullptr, *partials = nullptr;
  uint16_t *img = nullptr;  // w1img | w2img | w2timg
  int *d_err = nullptr;
  int *h_err = nullptr;
  int sms = 0;
  int64_t step = 0;
  // dataset
  uint16_t *dx = nullptr;
  float *dt = nullptr;
  float *dw = nullptr;  // sample weights or NULL
  int64_t dn = 0;
  cudaStream_t stream = nullptr;
};

int fail(Mlp *P, int code, const std::string &msg) {
  P->err = msg;
  return code;
}

#define MK(call)                                                                         \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return imodel::fail(P, e_ == cudaErrorMemoryAllocation ? IMODEL_SWM_ENOMEM          \
                                                             : IMODEL_SWM_ECUDA,          \
                          std::string(#call) + ": " + cudaGetErrorString(e_));           \
  } while (0)

Weights weights(Mlp *P) {
  Weights W;
  W.w1img = P->img;
  W.w2img = P->img + NH * K1;
  W.w2timg = P->img + NH * K1 + NH * NH;
  W.p = P->p;
  return W;
}

int images(Mlp *P) {
  Weights W = weights(P);
  k_make_images<<<(NH * NH + 255) / 256, 256, 0, P->stream>>>(
      P->p, const_cast<uint16_t *>(W.w1img), const_cast<uint16_t *>(W.w2img),
      const_cast<uint16_t *>(W.w2timg));
  MK(cudaGetLastError());
  return IMODEL_SWM_OK;
}

int check_err(Mlp *P) {
  MK(cudaMemcpyAsync(P->h_err, P->d_err, sizeof(int), cudaMemcpyDeviceToHost, P->stream));
  MK(cudaMemsetAsync(P->d_err, 0, sizeof(int), P->stream));
  MK(cudaStreamSynchronize(P->stream));
  if (*P->h_err) return fail(P, IMODEL_SWM_ECUDA, "tensor-core completion wait timed out");
  return IMODEL_SWM_OK;
}

// one batch's gradient and loss sum into P->g or, with A, straight into an Adam
// step and A->loss
int run_grad(Mlp *P, const uint16_t *x, const float *t, const float *w, int64_t n, int64_t batch,
             uint64_t seed, const AdamArgs *A) {
  const int64_t ntiles = (batch + TM - 1) / TM;
  const int nblk = static_cast<int>(std::min<int64_t>(ntiles, TRN_CTAS * P->sms));
  launch_pdl_smem(k_mlp_train, nblk, TRN_THREADS, TRN_SMEM, P->stream, weights(P), x, t, w, n, batch, seed,
                  1.0f / static_cast<float>(batch), P->partials, P->d_err);
  MK(cudaGetLastError());
  constexpr int blocks = (NPART + 31) / 32;
  if (A)
    launch_pdl(k_reduce<true>, blocks, 32 * kRed, P->stream, P->partials, nblk, nullptr, *A);
  else
    launch_pdl(k_reduce<false>, blocks, 32 * kRed, P->stream, P->partials, nblk, P->g, AdamArgs{});
  MK(cudaGetLastError());
  return IMODEL_SWM_OK;
}

}  // namespace

// ---- entry points used by the shallow-water handle (swm_capi.cu) -----------
int learned_prepare(const float *params_host, LearnedDev *L, cudaStream_t s) {
  if (cudaMalloc(&L->p, NPART * sizeof(float)) != cudaSuccess) return IMODEL_SWM_ENOMEM;
  if (cudaMalloc(&L->img, (NH * K1 + 2 * NH * NH) * 2) != cudaSuccess) return IMODEL_SWM_ENOMEM;
  if (cudaMemcpyAsync(L->p, params_host, NPARAM * sizeof(float), cudaMemcpyHostToDevice, s) !=
      cudaSuccess)
    return IMODEL_SWM_ECUDA;
  k_make_images<<<(NH * NH + 255) / 256, 256, 0, s>>>(L->p, L->img, L->img + NH * K1,
                                                      L->img + NH * K1 + NH * NH);
  if (cudaGetLastError() != cudaSuccess) return IMODEL_SWM_ECUDA;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&L->sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaFuncSetAttribute(pipe::k_mlp_pipe<pipe::EdgeTask, 2>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, pipe::SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(pipe::k_mlp_pipe<pipe::EdgeTask, 3>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, pipe::SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(pipe::k_mlp_pipe<pipe::EdgeTask, 4>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, pipe::SMEM) != cudaSuccess)
    return IMODEL_SWM_ECUDA;
  return IMODEL_SWM_OK;
}

void learned_launch(const DevMesh &M, const LearnedDev &L, const float *hd, const float *u,
                    const float *q_tr, float h_ref, int gather_groups, int *err, cudaStream_t s) {
  Weights W;
  W.w1img = L.img;
  W.w2img = L.img + NH * K1;
  W.w2timg = L.img + NH * K1 + NH * NH;
  W.p = L.p;
  const int64_t ne = M.ne;
  const int64_t ntiles = (ne + TM - 1) / TM;
  const int nblk = static_cast<int>(std::min<int64_t>(ntiles, L.sms > 0 ? L.sms : 1));
  pipe::EdgeTask task{L.blocks, u, q_tr, hd, h_ref, L.corr};
  if (gather_groups == 2)
    pipe::k_mlp_pipe<pipe::EdgeTask, 2><<<nblk, pipe::THREADS, pipe::SMEM, s>>>(W, ne, task, err);
  else if (gather_groups == 3)
    pipe::k_mlp_pipe<pipe::EdgeTask, 3><<<nblk, pipe::THREADS, pipe::SMEM, s>>>(W, ne, task, err);
  else
    pipe::k_mlp_pipe<pipe::EdgeTask, 4><<<nblk, pipe::THREADS, pipe::SMEM, s>>>(W, ne, task, err);
}

}  // namespace imodel

using imodel::Mlp;

extern "C" {

int imodel_mlp_create(int32_t device, void **mlp) {
  if (!mlp) return IMODEL_SWM_EINVAL;
  Mlp *P = new (std::nothrow) Mlp();
  *mlp = P;
  if (!P) return IMODEL_SWM_ENOMEM;
  P->device = device;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return imodel::fail(P, IMODEL_SWM_ENODEV, "no CUDA device");
  MK(cudaSetDevice(device));
  MK(cudaStreamCreateWithFlags(&P->stream, cudaStreamNonBlocking));
  MK(cudaDeviceGetAttribute(&P->sms, cudaDevAttrMultiProcessorCount, device));
  MK(cudaFuncSetAttribute(imodel::k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          imodel::TRN_SMEM));
  MK(cudaFuncSetAttribute(imodel::pipe::k_mlp_pipe<imodel::pipe::RowsTask, 2>,
                          cudaFuncAttributeMaxDynamicSharedMemorySize, imodel::pipe::SMEM));
  MK(cudaMalloc(&P->p, imodel::NPART * sizeof(float)));
  MK(cudaMalloc(&P->m, imodel::NPART * sizeof(float)));
  MK(cudaMalloc(&P->v, imodel::NPART * sizeof(float)));
  MK(cudaMalloc(&P->g, imodel::NPART * sizeof(float)));
  MK(cudaMalloc(&P->partials, static_cast<size_t>(imodel::TRN_CTAS * P->sms) * imodel::NPART *
                                  sizeof(float)));
  MK(cudaMalloc(&P->img, (imodel::NH * imodel::K1 + 2 * imodel::NH * imodel::NH) * 2));
  MK(cudaMalloc(&P->d_err, sizeof(int)));
  MK(cudaMemsetAsync(P->p, 0, imodel::NPART * sizeof(float), P->stream));
  MK(cudaMemsetAsync(P->m, 0, imodel::NPART * sizeof(float), P->stream));
  MK(cudaMemsetAsync(P->v, 0, imodel::NPART * sizeof(float), P->stream));
  MK(cudaMemsetAsync(P->d_err, 0, sizeof(int), P->stream));
  MK(cudaMallocHost(&P->h_err, sizeof(int)));
  return IMODEL_SWM_OK;
}

int imodel_mlp_set_params(void *mlp, const float *params, int32_t n) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || !params || n != imodel::NPARAM) return IMODEL_SWM_EINVAL;
  MK(cudaSetDevice(P->device));
  MK(cudaMemcpyAsync(P->p, params, n * sizeof(float), cudaMemcpyHostToDevice, P->stream));
  MK(cudaMemsetAsync(P->m, 0, n * sizeof(float), P->stream));
  MK(cudaMemsetAsync(P->v, 0, n * sizeof(float), P->stream));
  P->step = 0;
  int rc = imodel::images(P);
  if (rc) return rc;
  MK(cudaStreamSynchronize(P->stream));
  return IMODEL_SWM_OK;
}

int imodel_mlp_get_params(void *mlp, float *params, int32_t n) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || !params || n != imodel::NPARAM) return IMODEL_SWM_EINVAL;
  MK(cudaSetDevice(P->device));
  MK(cudaMemcpyAsync(params, P->p, n * sizeof(float), cudaMemcpyDeviceToHost, P->stream));
  MK(cudaStreamSynchronize(P->stream));
  return IMODEL_SWM_OK;
}

int imodel_mlp_forward(void *mlp, const uint16_t *x, int64_t n, float *y) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || !x || !y || n <= 0) return IMODEL_SWM_EINVAL;
  MK(cudaSetDevice(P->device));
  uint16_t *dx = nullptr;
  float *dy = nullptr;
  MK(cudaMalloc(&dx, static_cast<size_t>(n) * imodel::NIN * 2));
  cudaError_t e = cudaMalloc(&dy, static_cast<size_t>(n) * sizeof(float));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dx, x, static_cast<size_t>(n) * imodel::NIN * 2, cudaMemcpyHostToDevice,
                        P->stream);
  if (e == cudaSuccess) {
    const int64_t ntiles = (n + imodel::TM - 1) / imodel::TM;
    const int nblk = static_cast<int>(std::min<int64_t>(ntiles, P->sms));
    // rows need no gathers: two gather groups, four epilogue groups
    imodel::pipe::k_mlp_pipe<imodel::pipe::RowsTask, 2>
        <<<nblk, imodel::pipe::THREADS, imodel::pipe::SMEM, P->stream>>>(
            imodel::weights(P), n, imodel::pipe::RowsTask{dx, dy}, P->d_err);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(y, dy, static_cast<size_t>(n) * sizeof(float), cudaMemcpyDeviceToHost,
                        P->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(P->stream);
  cudaFree(dx);
  cudaFree(dy);
  if (e != cudaSuccess) return imodel::fail(P, IMODEL_SWM_ECUDA, cudaGetErrorString(e));
  return imodel::check_err(P);
}

int imodel_mlp_grad(void *mlp, const uint16_t *x, const float *t, const float *w, int64_t n,
                    uint64_t seed,
                    int64_t batch, float *grad, double *loss) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || !x || !t || !grad || n <= 0 || batch <= 0) return IMODEL_SWM_EINVAL;
  MK(cudaSetDevice(P->device));
  uint16_t *dx = nullptr;
  float *dt = nullptr;
  MK(cudaMalloc(&dx, static_cast<size_t>(n) * imodel::NIN * 2));
  MK(cudaMalloc(&dt, static_cast<size_t>(n) * sizeof(float)));
  float *dwt = nullptr;
  if (w) MK(cudaMalloc(&dwt, static_cast<size_t>(n) * sizeof(float)));
  if (w)
    MK(cudaMemcpyAsync(dwt, w, static_cast<size_t>(n) * sizeof(float), cudaMemcpyHostToDevice,
                       P->stream));
  MK(cudaMemcpyAsync(dx, x, static_cast<size_t>(n) * imodel::NIN * 2, cudaMemcpyHostToDevice,
                     P->stream));
  MK(cudaMemcpyAsync(dt, t, static_cast<size_t>(n) * sizeof(float), cudaMemcpyHostToDevice,
                     P->stream));
  int rc = imodel::run_grad(P, dx, dt, dwt, n, batch, seed, nullptr);
  std::vector<float> g(imodel::NPART);
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(g.data(), P->g, imodel::NPART * sizeof(float),
                                    cudaMemcpyDeviceToHost, P->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(P->stream);
    if (e != cudaSuccess) rc = imodel::fail(P, IMODEL_SWM_ECUDA, cudaGetErrorString(e));
  }
  cudaFree(dx);
  cudaFree(dt);
  if (dwt) cudaFree(dwt);
  if (rc) return rc;
  rc = imodel::check_err(P);
  if (rc) return rc;
  std::memcpy(grad, g.data(), imodel::NPARAM * sizeof(float));
  if (loss) *loss = static_cast<double>(g[imodel::NPARAM]) / static_cast<double>(batch);
  return IMODEL_SWM_OK;
}

int imodel_mlp_load_dataset(void *mlp, const uint16_t *x, const float *t, const float *w,
                            int64_t n) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || !x || !t || n <= 0) return IMODEL_SWM_EINVAL;
  MK(cudaSetDevice(P->device));
  if (P->dx) cudaFree(P->dx);
  if (P->dt) cudaFree(P->dt);
  if (P->dw) cudaFree(P->dw);
  P->dw = nullptr;
  P->dx = nullptr;
  P->dt = nullptr;
  P->dn = 0;
  MK(cudaMalloc(&P->dx, static_cast<size_t>(n) * imodel::NIN * 2));
  MK(cudaMalloc(&P->dt, static_cast<size_t>(n) * sizeof(float)));
  if (w) {
    MK(cudaMalloc(&P->dw, static_cast<size_t>(n) * sizeof(float)));
    MK(cudaMemcpyAsync(P->dw, w, static_cast<size_t>(n) * sizeof(float), cudaMemcpyHostToDevice,
                       P->stream));
  }
  MK(cudaMemcpyAsync(P->dx, x, static_cast<size_t>(n) * imodel::NIN * 2, cudaMemcpyHostToDevice,
                     P->stream));
  MK(cudaMemcpyAsync(P->dt, t, static_cast<size_t>(n) * sizeof(float), cudaMemcpyHostToDevice,
                     P->stream));
  MK(cudaStreamSynchronize(P->stream));
  P->dn = n;
  return IMODEL_SWM_OK;
}

int imodel_mlp_train(void *mlp, int64_t steps, int64_t batch, float lr, uint64_t seed,
                     float *losses) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P || steps <= 0 || batch <= 0) return IMODEL_SWM_EINVAL;
  if (!P->dn) return imodel::fail(P, IMODEL_SWM_ESTATE, "no dataset loaded");
  MK(cudaSetDevice(P->device));
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::vector<float> lossbuf(static_cast<size_t>(steps), 0.0f);
  float *dloss = nullptr;
  MK(cudaMalloc(&dloss, static_cast<size_t>(steps) * sizeof(float)));
  int rc = IMODEL_SWM_OK;
  for (int64_t s = 0; s < steps && !rc; ++s) {
    const uint64_t draw = imodel::splitmix(seed + static_cast<uint64_t>(P->step));
    P->step += 1;
    const imodel::Weights W = imodel::weights(P);
    imodel::AdamArgs A;
    A.p = P->p;
    A.m = P->m;
    A.v = P->v;
    A.loss = dloss + s;
    A.w1img = const_cast<uint16_t *>(W.w1img);
    A.w2img = const_cast<uint16_t *>(W.w2img);
    A.w2timg = const_cast<uint16_t *>(W.w2timg);
    A.lr = lr;
    A.b1 = b1;
    A.b2 = b2;
    A.eps = eps;
    A.c1 = 1.0f - std::pow(b1, static_cast<float>(P->step));
    A.c2 = 1.0f - std::pow(b2, static_cast<float>(P->step));
    rc = imodel::run_grad(P, P->dx, P->dt, P->dw, P->dn, batch, draw, &A);
    if (rc) P->step -= 1;
  }
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(lossbuf.data(), dloss, static_cast<size_t>(steps) * sizeof(float),
                                    cudaMemcpyDeviceToHost, P->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(P->stream);
    if (e != cudaSuccess) rc = imodel::fail(P, IMODEL_SWM_ECUDA, cudaGetErrorString(e));
  }
  cudaFree(dloss);
  if (rc) return rc;
  rc = imodel::check_err(P);
  if (rc) return rc;
  if (losses)
    for (int64_t s = 0; s < steps; ++s) losses[s] = lossbuf[s] / static_cast<float>(batch);
  return IMODEL_SWM_OK;
}

int imodel_mlp_destroy(void *mlp) {
  Mlp *P = static_cast<Mlp *>(mlp);
  if (!P) return IMODEL_SWM_OK;
  if (P->stream) cudaStreamSynchronize(P->stream);
  for (void *q : {static_cast<void *>(P->p), static_cast<void *>(P->m), static_cast<void *>(P->v),
                  static_cast<void *>(P->g), static_cast<void *>(P->partials),
                  static_cast<void *>(P->img), static_cast<void *>(P->d_err),
                  static_cast<void *>(P->dx), static_cast<void *>(P->dt),
                  static_cast<void *>(P->dw)})
    if (q) cudaFree(q);
  if (P->h_err) cudaFreeHost(P->h_err);
  if (P->stream) cudaStreamDestroy(P->stream);
  delete P;
  return IMODEL_SWM_OK;
}

const char *imodel_mlp_last_error(void *mlp) {
  Mlp *P = static_cast<Mlp *>(mlp);
  return P ? P->err.c_str() : "NULL handle";
}

}  // extern "C"
