// Learned Picard start: a mesh-graph network on the triangle b-grid, BF16 on the tcgen05 tensor
// cores with FP32 accumulation in tensor memory.
//
// This file holds the tensor-core GEMM tile and the C entry point that exercises it alone
// (ufe_umma_gemm_bf16); the network's kernels build on the same tile.
#include <algorithm>
#include <vector>

#include "ufe_internal.cuh"
#include "ufe_umma.cuh"

namespace {

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
  return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// Y[M x N] = X[M x K] * W[N x K]^T, X and W BF16 row-major, Y FP32; one CTA per 128 rows.
template <int N>
__global__ void __launch_bounds__(128) k_gemm_tile_test(int M, int K, const __nv_bfloat16 *__restrict__ X,
                                                        const __nv_bfloat16 *__restrict__ W, float *__restrict__ Y,
                                                        int *err) {
  extern __shared__ uint8_t smraw[];
  __shared__ uint64_t mbar;
  __shared__ uint32_t tslot;
  uint8_t *sm = align1024(smraw);
  const int kblocks = K / 64;
  uint8_t *sA = sm;
  uint8_t *sB = sm + kblocks * 128 * 128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = blockIdx.x * 128;
  // A: thread tid stages row tid, 16-byte chunks into their swizzled positions
  for (int kb = 0; kb < kblocks; ++kb)
    for (int c = 0; c < 8; ++c) {
      const uint4 v = *reinterpret_cast<const uint4 *>(X + (int64_t)(row0 + tid) * K + kb * 64 + c * 8);
      *reinterpret_cast<uint4 *>(sA + kb * 128 * 128 + umma::sw128_chunk(tid, c)) = v;
    }
  for (int idx = tid; idx < N * kblocks * 8; idx += 128) {
    const int r = idx / (kblocks * 8), rem = idx - r * kblocks * 8, kb = rem >> 3, c = rem & 7;
    const uint4 v = *reinterpret_cast<const uint4 *>(W + (int64_t)r * K + kb * 64 + c * 8);
    *reinterpret_cast<uint4 *>(sB + kb * N * 128 + umma::sw128_chunk(r, c)) = v;
  }
  if (warp == 0) umma::tmem_alloc(&tslot, N);
  if (tid == 0) {
    umma::mbar_init(umma::smem_u32(&mbar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_smem_async();
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  const uint32_t tmem = tslot;
  if (tid == 0) {
    umma::mma_tile<N>(tmem, umma::smem_u32(sA), umma::smem_u32(sB), kblocks, false);
    umma::commit(umma::smem_u32(&mbar));
  }
  bool ok = umma::mbar_wait(umma::smem_u32(&mbar), 0);
  ok = __syncthreads_and(ok);
  umma::fence_after();
  if (ok) {
    for (int c0 = 0; c0 < N; c0 += 16) {
      float v[16];
      umma::tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + c0, v);
      float *y = Y + (int64_t)(row0 + 32 * warp + lane) * N + c0;
#pragma unroll
      for (int i = 0; i < 16; ++i) y[i] = v[i];
    }
  } else {
    if (tid == 0) atomicExch(err, 1);
    umma::mbar_wait(umma::smem_u32(&mbar), 0);   // bounded: let the MMAs drain before freeing TMEM
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  if (warp == 0) umma::tmem_dealloc(tmem, N);
}

// ================================================================================================
// The network.  Nodes are triangles; each has up to three neighbours (TriC).  Width C = 64.
//   h0      = relu(We x + be)                                  (x: FIN = 16 features, zero-padded)
//   layer l: a = mean_{j in N(i)} h_j;  t = relu(W1 [h, a] + b1);  h <- h + W2 t + b2   (4 layers)
//   y       = Wd h + bd        (kGnnOut = 3 outputs: u, v scaled, and the log-viscosity)
// BF16 operands, FP32 accumulation (TMEM) and FP32 activations in global memory.
constexpr int kC = 64;
constexpr int kFin = 16;
constexpr int kLayers = 4;
constexpr int kNb = 3;

// parameter offsets (floats) in the flat FP32 parameter vector
constexpr int kOffWe = 0;                                   // [64 x 16]
constexpr int kOffBe = kOffWe + kC * kFin;                  // [64]
constexpr int kOffL0 = kOffBe + kC;
constexpr int kLayerSize = kC * 2 * kC + kC + kC * kC + kC; // W1 [64x128], b1, W2 [64x64], b2
constexpr int kOffWd = kOffL0 + kLayers * kLayerSize;       // [kGnnOut x 64]
constexpr int kOffBd = kOffWd + kGnnOut * kC;               // [kGnnOut]
constexpr int kParams = kOffBd + kGnnOut;
__host__ __device__ constexpr int off_W1(int l) { return kOffL0 + l * kLayerSize; }
__host__ __device__ constexpr int off_b1(int l) { return off_W1(l) + kC * 2 * kC; }
__host__ __device__ constexpr int off_W2(int l) { return off_b1(l) + kC; }
__host__ __device__ constexpr int off_b2(int l) { return off_W2(l) + kC * kC; }

// BF16 weight copies in the layouts the tile reads (B operand: [N rows x K], row-major)
constexpr int kBfWe = 0;                                    // [64 x 64]  (We, inputs padded to 64)
constexpr int kBfL0 = kBfWe + kC * kC;
constexpr int kBfLayer = kC * 2 * kC + kC * kC + kC * kC + 2 * kC * kC;   // W1, W2, W2T, W1T
__host__ __device__ constexpr int bf_W1(int l) { return kBfL0 + l * kBfLayer; }       // [64 x 128]
__host__ __device__ constexpr int bf_W2(int l) { return bf_W1(l) + kC * 2 * kC; }     // [64 x 64]
__host__ __device__ constexpr int bf_W2T(int l) { return bf_W2(l) + kC * kC; }        // [64 x 64]
__host__ __device__ constexpr int bf_W1T(int l) { return bf_W2T(l) + kC * kC; }       // [128 x 64]
constexpr int kBfTotal = kBfL0 + kLayers * kBfLayer;

__device__ __forceinline__ uint16_t bf16_bits(float x) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  return (uint32_t)bf16_bits(a) | ((uint32_t)bf16_bits(b) << 16);
}
// eight floats -> one 16-byte chunk of BF16
__device__ __forceinline__ uint4 pack8(const float *v) {
  return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

// Stage a [rows x 64*kblocks] BF16 matrix (global, row-major) as a B operand.
__device__ __forceinline__ void stage_weights(uint8_t *dst, const uint16_t *__restrict__ W, int rows, int kblocks) {
  for (int idx = threadIdx.x; idx < rows * kblocks * 8; idx += blockDim.x) {
    const int r = idx / (kblocks * 8), rem = idx - r * kblocks * 8, kb = rem >> 3, c = rem & 7;
    const uint4 v = *reinterpret_cast<const uint4 *>(W + (int64_t)r * 64 * kblocks + kb * 64 + c * 8);
    *reinterpret_cast<uint4 *>(dst + kb * rows * 128 + umma::sw128_chunk(r, c)) = v;
  }
}
struct Sync {
  uint64_t mbar;
  uint32_t tslot;
};

// CTA-wide: make staged shared memory visible to the tensor core and order it before the MMA
__device__ __forceinline__ void smem_to_mma() {
  __syncwarp();   // per-row conditions came before
  umma::fence_smem_async();
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
}
// thread 0 issued MMAs and committed to the barrier; every thread waits (bounded).  Returns false
// (CTA-uniform) on a timeout and records it.
__device__ __forceinline__ bool mma_done(Sync &sy, uint32_t &phase, int *err) {
  bool ok = umma::mbar_wait(umma::smem_u32(&sy.mbar), phase);
  phase ^= 1;
  ok = __syncthreads_and(ok);
  umma::fence_after();
  if (!ok && threadIdx.x == 0) atomicExch(err, 1);
  return ok;
}
__device__ __forceinline__ void sync_setup(Sync &sy, uint32_t tmem_cols) {
  if (threadIdx.x < 32) umma::tmem_alloc(&sy.tslot, tmem_cols);
  if (threadIdx.x == 0) {
    umma::mbar_init(umma::smem_u32(&sy.mbar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
}
__device__ __forceinline__ void sync_teardown(Sync &sy, uint32_t phase, uint32_t tmem_cols, bool ok) {
  if (!ok) umma::mbar_wait(umma::smem_u32(&sy.mbar), phase ^ 1);   // bounded drain of the failed phase
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  if (threadIdx.x < 32) umma::tmem_dealloc(sy.tslot, tmem_cols);
}
struct Graph {
  int64_t n;                     // nodes
  const int32_t *__restrict__ nbr;   // n x 3, -1: none
};

// decoder gradient: dWd [kGnnOut x 64] and dbd
constexpr int kDecParts = kGnnOut * kC + kGnnOut;
static_assert(kGnnOut * kC + 64 <= 256, "one thread of a CTA per entry of the decoder's gradient");

// ---- the layer kernels ---------------------------------------------------------------------------
// What bounds them is memory, not the tensor cores: a layer reads each node's row and its neighbours' rows
// (256 B each, mostly L2 hits) and writes one, 30 MB per 115k nodes and layer.  So a CTA of 256 threads stays
// resident, stages the layer's weights once and loops over 128-node tiles; rows are read and written
// coalesced (16 lanes per row, 16 bytes each, the sums of a column always in the same thread) and pass
// through swizzled shared memory on their way to and from the tensor cores; the CTAs on an SM overlap one
// another's loads and MMAs.  Measured (cold caches): a forward layer on 115k nodes 34 us, where one thread per
// row with 256-byte strides and weights staged for every tile took 118; a layer's backward pass on 60k nodes 54
// us, where six kernels (transposing stores for the weight gradients, a serial sum of their partials) took 340;
// the decoder inside the last layer, 32 us before.
//
// The backward pass of a layer is one kernel as well.  dh_out is gathered while it is loaded (the mean's
// backward), and the weight gradients D[features x outputs] += A^T B over the tile's nodes read the same
// tiles as the data gradients: a [node][64 features] tile is K-major for a product over features and
// MN-major for a product over nodes (transpose bits in the instruction descriptor), so nothing is
// transposed.  Their accumulators stay in tensor memory over all tiles of the CTA.
constexpr int kTile = 128;
constexpr int kGnnThreads = 256;
constexpr int kTileBytes = kTile * 128;   // a K block: 128 rows x 64 BF16

struct RowMap {   // coalesced view of a tile: this thread's float4 column and first row (rows rr + 16 m)
  int c4, rr;
  __device__ __forceinline__ RowMap() : c4(threadIdx.x & 15), rr(threadIdx.x >> 4) {}
};
// four floats as BF16 at (row r, columns 4 c4 ...) of a K block
__device__ __forceinline__ void stage4(uint8_t *tile, int r, int c4, float4 v) {
  *reinterpret_cast<uint2 *>(tile + umma::sw128_chunk(r, c4 >> 1) + (c4 & 1) * 8) =
      make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
}
// FP32 tile [128][64], float4 columns permuted so that reads by row and by column are free of conflicts
__device__ __forceinline__ float4 *otile(uint8_t *o, int r, int c4) {
  return reinterpret_cast<float4 *>(o + r * 256 + ((c4 ^ (r & 15)) << 4));
}
__device__ __forceinline__ float4 ld_row(const float *__restrict__ h, int64_t i, int c4) {
  return __ldg(reinterpret_cast<const float4 *>(h + i * kC) + c4);
}
__device__ __forceinline__ float4 f4_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void f4_add(float4 &a, float4 b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  a.w += b.w;
}
// sum of the neighbours' rows (FP32, neighbour order), and their number
__device__ __forceinline__ int neighbour_sum(const Graph &g, const float *__restrict__ h, int64_t i, int c4, float4 &a) {
  int j[kNb], deg = 0;
  float4 t[kNb];
#pragma unroll
  for (int q = 0; q < kNb; ++q) j[q] = __ldg(g.nbr + i * kNb + q);
#pragma unroll
  for (int q = 0; q < kNb; ++q)
    if (j[q] >= 0) t[q] = ld_row(h, j[q], c4);
#pragma unroll
  for (int q = 0; q < kNb; ++q)
    if (j[q] >= 0) {
      f4_add(a, t[q]);
      ++deg;
    }
  return deg;
}
__device__ __forceinline__ float4 neighbour_mean4(const Graph &g, const float *__restrict__ h, int64_t i, int c4) {
  float4 a = f4_zero();
  const int deg = neighbour_sum(g, h, i, c4, a);
  if (deg > 0) {
    const float inv = 1.0f / (float)deg;
    a.x *= inv;
    a.y *= inv;
    a.z *= inv;
    a.w *= inv;
  }
  return a;
}
// 32 TMEM columns from `col` of row 32 (warp % 4) + lane
__device__ __forceinline__ void tmem_row32(uint32_t tmem, int col, float *v) {
  const uint32_t base = tmem + ((uint32_t)(32 * ((threadIdx.x >> 5) & 3)) << 16) + col;
  umma::tmem_ld16(base, v);
  umma::tmem_ld16(base + 16, v + 16);
}
// the epilogue's view: this thread's row and first column
struct EpiMap {
  int r, col;
  __device__ __forceinline__ EpiMap()
      : r(32 * ((threadIdx.x >> 5) & 3) + (threadIdx.x & 31)), col(32 * (threadIdx.x >> 7)) {}
};
__device__ __forceinline__ void issue_commit(Sync &sy) { umma::commit(umma::smem_u32(&sy.mbar)); }

__global__ void __launch_bounds__(kGnnThreads, 4) k_gnn_encoder(Graph g, const float *__restrict__ x,
                                                                const uint16_t *__restrict__ wbf,
                                                                const float *__restrict__ prm, float *__restrict__ h0,
                                                                int *err) {
  extern __shared__ uint8_t smraw[];
  __shared__ Sync sy;
  __shared__ float be[kC];
  uint8_t *sm = align1024(smraw);
  uint8_t *sA = sm, *sB = sA + kTileBytes, *sO = sB + 64 * 128;
  const RowMap m;
  const EpiMap e;
  // features 16 .. 63 of the tile stay zero
  for (int i = threadIdx.x; i < kTileBytes / 16; i += kGnnThreads) reinterpret_cast<uint4 *>(sA)[i] = make_uint4(0, 0, 0, 0);
  stage_weights(sB, wbf + kBfWe, kC, 1);
  if (threadIdx.x < kC) be[threadIdx.x] = prm[kOffBe + threadIdx.x];
  sync_setup(sy, 64);
  uint32_t phase = 0;
  bool ok = true;
  for (int64_t i0 = (int64_t)blockIdx.x * kTile; i0 < g.n && ok; i0 += (int64_t)gridDim.x * kTile) {
    const int rows = (int)min((int64_t)kTile, g.n - i0);
#pragma unroll
    for (int q = 0; q < 2; ++q) {   // 4 lanes per row of 16 features
      const int t = threadIdx.x + q * kGnnThreads, r = t >> 2, c4 = t & 3;
      stage4(sA, r, c4, r < rows ? __ldg(reinterpret_cast<const float4 *>(x + (i0 + r) * kFin) + c4) : f4_zero());
    }
    smem_to_mma();
    if (threadIdx.x == 0) {
      umma::mma_tile<64>(sy.tslot, umma::smem_u32(sA), umma::smem_u32(sB), 1, false);
      issue_commit(sy);
    }
    ok = mma_done(sy, phase, err);
    if (!ok) break;
    float v[32];
    tmem_row32(sy.tslot, e.col, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = fmaxf(v[k] + be[e.col + k], 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      *otile(sO, e.r, e.col / 4 + k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      if (r < rows) reinterpret_cast<float4 *>(h0 + (i0 + r) * kC)[m.c4] = *otile(sO, r, m.c4);
    }
  }
  sync_teardown(sy, phase, 64, ok);
}

// The decoder's arguments: y = Wd h + bd of the last layer's output.  With targets (training): the loss (w: per-node
// weight divided by the batch's total weight, 0 for nodes outside the loss), dy in y's place and the
// decoder's gradient, per CTA.
struct DecoderArgs {
  float *y;
  const float *target, *w;
  double *loss_part;
  float *dpart;
};

template <bool kTrain, bool kLast>
__global__ void __launch_bounds__(kGnnThreads, 2) k_gnn_layer_fwd(Graph g, int layer, const uint16_t *__restrict__ wbf,
                                                                  const float *__restrict__ prm,
                                                                  const float *__restrict__ h_in,
                                                                  float *__restrict__ h_out, uint16_t *__restrict__ t_out,
                                                                  DecoderArgs dec, int *err) {
  extern __shared__ uint8_t smraw[];
  __shared__ Sync sy;
  __shared__ float b1[kC], b2[kC], wd[kGnnOut * kC], bd[kGnnOut], sdy[kLast && kTrain ? kTile * kGnnOut : 1];
  __shared__ double sloss[kLast && kTrain ? 4 : 1];
  uint8_t *sm = align1024(smraw);
  uint8_t *sA1 = sm;                       // 128 x 128 (2 K blocks); then the FP32 output tile
  uint8_t *sB1 = sA1 + 2 * kTileBytes;     // 64 x 128
  uint8_t *sA2 = sB1 + 2 * 64 * 128;       // 128 x 64
  uint8_t *sB2 = sA2 + kTileBytes;         // 64 x 64
  const RowMap m;
  const EpiMap e;
  stage_weights(sB1, wbf + bf_W1(layer), kC, 2);
  stage_weights(sB2, wbf + bf_W2(layer), kC, 1);
  if (threadIdx.x < kC) {
    b1[threadIdx.x] = prm[off_b1(layer) + threadIdx.x];
    b2[threadIdx.x] = prm[off_b2(layer) + threadIdx.x];
  }
  if (kLast) {
    if (threadIdx.x < kGnnOut * kC) wd[threadIdx.x] = prm[kOffWd + threadIdx.x];
    if (threadIdx.x < kGnnOut) bd[threadIdx.x] = prm[kOffBd + threadIdx.x];
  }
  sync_setup(sy, 128);
  uint32_t phase = 0;
  bool ok = true;
  double loss = 0.0;
  float dgrad = 0.f;   // kLast && kTrain: this thread's entry of the decoder's gradient
  for (int64_t i0 = (int64_t)blockIdx.x * kTile; i0 < g.n && ok; i0 += (int64_t)gridDim.x * kTile) {
    const int rows = (int)min((int64_t)kTile, g.n - i0);
    float4 own[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      own[q] = r < rows ? ld_row(h_in, i0 + r, m.c4) : f4_zero();
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      stage4(sA1, r, m.c4, own[q]);
      stage4(sA1 + kTileBytes, r, m.c4, r < rows ? neighbour_mean4(g, h_in, i0 + r, m.c4) : f4_zero());
    }
    smem_to_mma();
    if (threadIdx.x == 0) {
      umma::mma_tile<64>(sy.tslot, umma::smem_u32(sA1), umma::smem_u32(sB1), 2, false);
      issue_commit(sy);
    }
    ok = mma_done(sy, phase, err);
    if (!ok) break;
    float v[32];
    tmem_row32(sy.tslot, e.col, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = fmaxf(v[k] + b1[e.col + k], 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<uint4 *>(sA2 + umma::sw128_chunk(e.r, e.col / 8 + c)) = pack8(v + 8 * c);
    smem_to_mma();
    if (threadIdx.x == 0) {
      umma::mma_tile<64>(sy.tslot + 64, umma::smem_u32(sA2), umma::smem_u32(sB2), 1, false);
      issue_commit(sy);
    }
    if (kTrain) {   // t = relu(...) for the backward pass, from the staged tile
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = threadIdx.x + q * kGnnThreads, r = t >> 3, c = t & 7;
        if (r < rows)
          reinterpret_cast<uint4 *>(t_out + (i0 + r) * kC)[c] =
              *reinterpret_cast<const uint4 *>(sA2 + umma::sw128_chunk(r, c));
      }
    }
    ok = mma_done(sy, phase, err);
    if (!ok) break;
    tmem_row32(sy.tslot, 64 + e.col, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = v[k] + b2[e.col + k];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      *otile(sA1, e.r, e.col / 4 + k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      float4 o = *otile(sA1, r, m.c4);
      o = make_float4(own[q].x + o.x, own[q].y + o.y, own[q].z + o.z, own[q].w + o.w);
      if (kLast) *otile(sA1, r, m.c4) = o;
      else if (r < rows) reinterpret_cast<float4 *>(h_out + (i0 + r) * kC)[m.c4] = o;
    }
    __syncthreads();   // the tile is staged again, or read by rows
    if (kLast) {
      const int r = threadIdx.x;
      if (r < kTile) {
        float yo[kGnnOut], sc[kGnnOut];
#pragma unroll
        for (int c = 0; c < kGnnOut; ++c) sc[c] = 0.f;
#pragma unroll 4
        for (int k = 0; k < kC / 4; ++k) {
          const float4 hv = *otile(sA1, r, k);
#pragma unroll
          for (int c = 0; c < kGnnOut; ++c) {
            const float *wk = wd + c * kC + 4 * k;
            sc[c] += wk[0] * hv.x;
            sc[c] += wk[1] * hv.y;
            sc[c] += wk[2] * hv.z;
            sc[c] += wk[3] * hv.w;
          }
        }
#pragma unroll
        for (int c = 0; c < kGnnOut; ++c) yo[c] = bd[c] + sc[c];
        if (kTrain) {
          const float wi = r < rows ? dec.w[i0 + r] : 0.f;
#pragma unroll
          for (int c = 0; c < kGnnOut; ++c) {
            const float er = r < rows ? yo[c] - dec.target[kGnnOut * (i0 + r) + c] : 0.f;
            loss += (double)wi * ((double)er * er);
            yo[c] = 2.f * wi * er;   // dy takes y's place
            sdy[r * kGnnOut + c] = yo[c];
          }
        }
        if (r < rows)
#pragma unroll
          for (int c = 0; c < kGnnOut; ++c) dec.y[kGnnOut * (i0 + r) + c] = yo[c];
      }
      __syncthreads();   // the tile is staged again, or read for the decoder's gradient
      if (kTrain) {
        const int c = threadIdx.x >> 6, k = threadIdx.x & 63;
        if (c < kGnnOut) {
          for (int q = 0; q < rows; ++q)
            dgrad += sdy[q * kGnnOut + c] * reinterpret_cast<const float *>(otile(sA1, q, k >> 2))[k & 3];
        } else if (k < kGnnOut) {
          for (int q = 0; q < rows; ++q) dgrad += sdy[q * kGnnOut + k];
        }
        __syncthreads();
      }
    }
  }
  if (kLast && kTrain) {
    if (threadIdx.x < kDecParts) dec.dpart[(int64_t)blockIdx.x * kDecParts + threadIdx.x] = dgrad;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if ((threadIdx.x & 31) == 0 && threadIdx.x < kTile) sloss[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) dec.loss_part[blockIdx.x] = (sloss[0] + sloss[1]) + (sloss[2] + sloss[3]);
  }
  sync_teardown(sy, phase, 128, ok);
}

// ---- backward ------------------------------------------------------------------------------------
// What a layer's backward pass leaves per node: dh_acc and dA (what each neighbour receives through the mean); the
// gradient that arrives at a node is dh_acc + the sum of its neighbours' dA (the adjacency is symmetric).
struct GradIn {
  const float *dacc, *dA;   // of the layer above; or, for the last layer,
  const float *dy;          // the decoder's dy (then dacc and dA are null)
};
__device__ __forceinline__ float4 grad_gather(const Graph &g, const GradIn &in, int64_t i, int c4) {
  float4 a = ld_row(in.dacc, i, c4);
  neighbour_sum(g, in.dA, i, c4, a);
  return a;
}
__device__ __forceinline__ float4 grad_decoder(const GradIn &in, const float *wd, int64_t i, int c4) {
  float d[kGnnOut];
#pragma unroll
  for (int c = 0; c < kGnnOut; ++c) d[c] = __ldg(in.dy + kGnnOut * i + c);
  float4 a = f4_zero();
#pragma unroll
  for (int c = 0; c < kGnnOut; ++c) {
    const float4 wv = *reinterpret_cast<const float4 *>(wd + c * kC + 4 * c4);
    f4_add(a, make_float4(wv.x * d[c], wv.y * d[c], wv.z * d[c], wv.w * d[c]));
  }
  return a;
}

// Weight-gradient partials per CTA: [128 features x 64 outputs] FP32, then the 64 column sums (bias).
constexpr int kPartW = 128 * kC, kPart = kPartW + kC;

// D[128 x 64] (+)= A^T B over the tile's 128 nodes: A the MN-major view of feature blocks a_stride bytes apart
// (0: one block, twice), B of one block of 64 outputs.  One thread calls this.
__device__ __forceinline__ void mma_wgrad(uint32_t tmem_d, uint32_t a, uint32_t a_stride, uint32_t b, bool accumulate) {
  constexpr uint32_t idesc = umma::idesc_bf16_f32(128, kC) | (1u << 15) | (1u << 16);
#pragma unroll
  for (int j = 0; j < kTile / 16; ++j)
    umma::mma_bf16(tmem_d, umma::desc_sw128_mn(a + j * 2048, a_stride), umma::desc_sw128_mn(b + j * 2048, 0), idesc,
                   (accumulate || j > 0) ? 1u : 0u);
}
// this thread's half row of a weight-gradient accumulator, of the first `features` rows, to the CTA's partial
__device__ __forceinline__ void store_partial(uint32_t tmem, const EpiMap &e, int features, float *part) {
  float v[32];
  tmem_row32(tmem, e.col, v);
  if (e.r >= features) return;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    reinterpret_cast<float4 *>(part + e.r * kC + e.col)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}
// column sums of the coalesced view (four columns per thread, 16 threads per column) in a fixed order
__device__ __forceinline__ void store_column_sums(uint8_t *scratch, const RowMap &m, float4 s, float *out) {
  float4 *red = reinterpret_cast<float4 *>(scratch);
  __syncthreads();
  red[m.rr * 16 + m.c4] = s;
  __syncthreads();
  if (threadIdx.x < 16) {
    float4 a = red[threadIdx.x];
    for (int q = 1; q < 16; ++q) f4_add(a, red[q * 16 + threadIdx.x]);
    reinterpret_cast<float4 *>(out)[threadIdx.x] = a;
  }
}

// dt = dh_out W2 (masked by t > 0) = ds; dz = ds W1 -> dh_acc = dh_out + dz[:64], dA = dz[64:] / deg; and the
// partials of dW2 = dh_out^T t, db2, dW1 = ds^T [h, mean], db1.
__global__ void __launch_bounds__(kGnnThreads, 2) k_gnn_layer_bwd(Graph g, int layer, const uint16_t *__restrict__ wbf,
                                                                  const float *__restrict__ prm, GradIn in,
                                                                  const uint16_t *__restrict__ t_in,
                                                                  const float *__restrict__ h_in,
                                                                  float *__restrict__ dacc, float *__restrict__ dA,
                                                                  float *__restrict__ part1, float *__restrict__ part2,
                                                                  int *err) {
  extern __shared__ uint8_t smraw[];
  __shared__ Sync sy;
  __shared__ __align__(16) float wd[kGnnOut * kC];
  uint8_t *sm = align1024(smraw);
  uint8_t *sD = sm;                      // dh_out
  uint8_t *sT = sD + kTileBytes;         // t; with sD the FP32 output tile later
  uint8_t *sH = sT + kTileBytes;         // h, then the mean
  uint8_t *sS = sH + 2 * kTileBytes;     // ds
  uint8_t *sB = sS + kTileBytes;         // 64 x 64: W2^T
  uint8_t *sB2 = sB + 64 * 128;          // 128 x 64: W1^T
  const RowMap m;
  const EpiMap e;
  const int lane = threadIdx.x & 31;
  stage_weights(sB, wbf + bf_W2T(layer), kC, 1);
  stage_weights(sB2, wbf + bf_W1T(layer), 2 * kC, 1);
  if (threadIdx.x < kGnnOut * kC) wd[threadIdx.x] = prm[kOffWd + threadIdx.x];
  sync_setup(sy, 256);
  const uint32_t tD = sy.tslot, tW2 = tD + 128, tW1 = tD + 192;
  uint32_t phase = 0;
  bool ok = true, first = true;
  float4 bias2 = f4_zero();
  float bias1 = 0.f;   // column e.col + lane, summed over this warp's rows
  for (int64_t i0 = (int64_t)blockIdx.x * kTile; i0 < g.n && ok; i0 += (int64_t)gridDim.x * kTile) {
    const int rows = (int)min((int64_t)kTile, g.n - i0);
    float4 own[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      own[q] = f4_zero();
      if (r < rows) own[q] = in.dy ? grad_decoder(in, wd, i0 + r, m.c4) : grad_gather(g, in, i0 + r, m.c4);
      stage4(sD, r, m.c4, own[q]);
      f4_add(bias2, own[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int t = threadIdx.x + q * kGnnThreads, r = t >> 3, c = t & 7;
      *reinterpret_cast<uint4 *>(sT + umma::sw128_chunk(r, c)) =
          r < rows ? __ldg(reinterpret_cast<const uint4 *>(t_in + (i0 + r) * kC) + c) : make_uint4(0, 0, 0, 0);
    }
    smem_to_mma();
    if (threadIdx.x == 0) {
      umma::mma_tile<64>(tD, umma::smem_u32(sD), umma::smem_u32(sB), 1, false);
      mma_wgrad(tW2, umma::smem_u32(sT), 0, umma::smem_u32(sD), !first);
      issue_commit(sy);
    }
    // the layer's input and its mean, while the first products run
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      stage4(sH, r, m.c4, r < rows ? ld_row(h_in, i0 + r, m.c4) : f4_zero());
      stage4(sH + kTileBytes, r, m.c4, r < rows ? neighbour_mean4(g, h_in, i0 + r, m.c4) : f4_zero());
    }
    ok = mma_done(sy, phase, err);
    if (!ok) break;
    float v[32];
    tmem_row32(tD, e.col, v);
#pragma unroll
    for (int c = 0; c < 4; ++c) {   // t > 0: a positive BF16's bits lie in 1 .. 0x7f80 (t is never NaN)
      const uint4 tv = *reinterpret_cast<const uint4 *>(sT + umma::sw128_chunk(e.r, e.col / 8 + c));
      const uint32_t tw[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float t = __uint_as_float(k & 1 ? tw[k >> 1] & 0xffff0000u : tw[k >> 1] << 16);
        v[8 * c + k] = t > 0.f ? v[8 * c + k] : 0.f;
      }
      *reinterpret_cast<uint4 *>(sS + umma::sw128_chunk(e.r, e.col / 8 + c)) = pack8(v + 8 * c);
    }
    smem_to_mma();
    if (threadIdx.x == 0) {
      umma::mma_tile<128>(tD, umma::smem_u32(sS), umma::smem_u32(sB2), 1, false);
      mma_wgrad(tW1, umma::smem_u32(sH), kTileBytes, umma::smem_u32(sS), !first);
      issue_commit(sy);
    }
    // db1: the columns of v over the warp's 32 rows, each lane ends with one column (31 additions)
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      const bool up = lane & w;
#pragma unroll
      for (int k = 0; k < w; ++k) {
        const float keep = up ? v[k + w] : v[k], send = up ? v[k] : v[k + w];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, w);
      }
    }
    bias1 += v[0];
    ok = mma_done(sy, phase, err);
    if (!ok) break;
    first = false;
#pragma unroll
    for (int half = 0; half < 2; ++half) {   // dz[:64], then dz[64:], through the FP32 tile (over sD, sT)
      if (half) __syncthreads();             // the first half has been read, and the warps are whole again
      tmem_row32(tD, 64 * half + e.col, v);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        *otile(sD, e.r, e.col / 4 + k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      umma::fence_before();
      __syncthreads();
      umma::fence_after();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int r = m.rr + 16 * q;
        float4 o = *otile(sD, r, m.c4);
        if (r < rows && half == 0) {
          o = make_float4(own[q].x + o.x, own[q].y + o.y, own[q].z + o.z, own[q].w + o.w);
          reinterpret_cast<float4 *>(dacc + (i0 + r) * kC)[m.c4] = o;
        } else if (r < rows) {
          int deg = 0;
#pragma unroll
          for (int j = 0; j < kNb; ++j) deg += __ldg(g.nbr + (i0 + r) * kNb + j) >= 0;
          const float inv = deg > 0 ? 1.0f / (float)deg : 0.f;
          reinterpret_cast<float4 *>(dA + (i0 + r) * kC)[m.c4] = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
        }
      }
    }
    __syncthreads();   // the FP32 tile is staged again
  }
  float *p1 = part1 + (int64_t)blockIdx.x * kPart, *p2 = part2 + (int64_t)blockIdx.x * kPart;
  if (ok) {   // every CTA has at least one tile
    store_partial(tW1, e, 2 * kC, p1);
    store_partial(tW2, e, kC, p2);
  }
  store_column_sums(sD, m, bias2, p2 + kPartW);
  float *red = reinterpret_cast<float *>(sS);
  red[threadIdx.x] = bias1;
  __syncthreads();
  if (threadIdx.x < kC) {   // warps 0-3 hold columns 0-31, warps 4-7 columns 32-63
    const float *q = red + (threadIdx.x >> 5) * 128 + (threadIdx.x & 31);
    p1[kPartW + threadIdx.x] = ((q[0] + q[32]) + q[64]) + q[96];
  }
  sync_teardown(sy, phase, 256, ok);
}

// encoder backward: ds = (the gradient at h0) * (h0 > 0); partials of dWe = ds^T x and dbe
__global__ void __launch_bounds__(kGnnThreads, 3) k_gnn_encoder_bwd(Graph g, const float *__restrict__ x, GradIn in,
                                                                    const float *__restrict__ h0,
                                                                    float *__restrict__ part, int *err) {
  extern __shared__ uint8_t smraw[];
  __shared__ Sync sy;
  uint8_t *sm = align1024(smraw);
  uint8_t *sD = sm, *sX = sD + kTileBytes;
  const RowMap m;
  const EpiMap e;
  for (int i = threadIdx.x; i < kTileBytes / 16; i += kGnnThreads) reinterpret_cast<uint4 *>(sX)[i] = make_uint4(0, 0, 0, 0);
  sync_setup(sy, 64);
  uint32_t phase = 0;
  bool ok = true, first = true;
  float4 bias = f4_zero();
  for (int64_t i0 = (int64_t)blockIdx.x * kTile; i0 < g.n && ok; i0 += (int64_t)gridDim.x * kTile) {
    const int rows = (int)min((int64_t)kTile, g.n - i0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = m.rr + 16 * q;
      float4 d = f4_zero();
      if (r < rows) {
        d = grad_gather(g, in, i0 + r, m.c4);
        const float4 h = ld_row(h0, i0 + r, m.c4);
        if (!(h.x > 0.f)) d.x = 0.f;
        if (!(h.y > 0.f)) d.y = 0.f;
        if (!(h.z > 0.f)) d.z = 0.f;
        if (!(h.w > 0.f)) d.w = 0.f;
      }
      stage4(sD, r, m.c4, d);
      f4_add(bias, d);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int t = threadIdx.x + q * kGnnThreads, r = t >> 2, c4 = t & 3;
      stage4(sX, r, c4, r < rows ? __ldg(reinterpret_cast<const float4 *>(x + (i0 + r) * kFin) + c4) : f4_zero());
    }
    smem_to_mma();
    if (threadIdx.x == 0) {
      mma_wgrad(sy.tslot, umma::smem_u32(sX), 0, umma::smem_u32(sD), !first);
      issue_commit(sy);
    }
    ok = mma_done(sy, phase, err);
    first = false;
  }
  float *p = part + (int64_t)blockIdx.x * kPart;
  if (ok) store_partial(sy.tslot, e, kFin, p);
  store_column_sums(sD, m, bias, p + kPartW);
  sync_teardown(sy, phase, 64, ok);
}

// Sum all CTAs' partials into the gradient vector, in a fixed order: each block takes 32 consecutive entries of one
// of the nine [128 x 64] + 64 partial sets (0: encoder, 1 + 2l: W1 and b1, 2 + 2l: W2 and b2 of layer l) or of
// the decoder's, its eight warps every eighth CTA, and adds the warps' sums in order.
constexpr int kPartSets = 1 + 2 * kLayers;
constexpr int kReduceBlocks = kPartSets * (kPart / 32) + (kDecParts + 31) / 32;
__global__ void __launch_bounds__(256) k_gnn_reduce(int nparts, int ndec, const float *__restrict__ part,
                                                    const float *__restrict__ dpart, float *__restrict__ grad) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int set = blockIdx.x / (kPart / 32);
  float s = 0.f;
  int off = -1;
  if (set < kPartSets) {
    const int en = (blockIdx.x % (kPart / 32)) * 32 + lane;
    const int fin = set == 0 ? kFin : (set & 1) ? 2 * kC : kC, layer = (set - 1) >> 1;
    const int w0 = set == 0 ? kOffWe : (set & 1) ? off_W1(layer) : off_W2(layer);
    const int b0 = set == 0 ? kOffBe : (set & 1) ? off_b1(layer) : off_b2(layer);
    const int f = en / kC, o = en % kC;   // en < kPartW: row f, column o
    off = en >= kPartW ? b0 + en - kPartW : f < fin ? w0 + o * fin + f : -1;
    const float *p = part + (int64_t)set * nparts * kPart + en;
    if (off >= 0)
      for (int c = warp; c < nparts; c += 8) s += __ldg(p + (int64_t)c * kPart);
  } else {
    const int en = (blockIdx.x - kPartSets * (kPart / 32)) * 32 + lane;
    off = en < kGnnOut * kC ? kOffWd + en : en < kDecParts ? kOffBd + en - kGnnOut * kC : -1;
    if (off >= 0)
      for (int c = warp; c < ndec; c += 8) s += __ldg(dpart + (int64_t)c * kDecParts + en);
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && off >= 0) {
    for (int q = 1; q < 8; ++q) s += red[q][lane];
    grad[off] = s;
  }
}

// Adam (FP32) on the flat parameter vector
__global__ void k_gnn_adam(int n, float *__restrict__ p, const float *__restrict__ gr, float *__restrict__ m,
                           float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float g = gr[t];
  const float mt = b1 * m[t] + (1.f - b1) * g;
  const float vt = b2 * v[t] + (1.f - b2) * g * g;
  m[t] = mt;
  v[t] = vt;
  p[t] -= lr * (mt / c1) / (sqrtf(vt / c2) + eps);
}

// BF16 tile copies of the weights
__global__ void k_gnn_pack(const float *__restrict__ prm, uint16_t *__restrict__ wbf) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < kC * kC) {   // We padded to 64 inputs
    const int o = t / kC, f = t % kC;
    wbf[kBfWe + t] = bf16_bits(f < kFin ? prm[kOffWe + o * kFin + f] : 0.f);
  }
  for (int l = 0; l < kLayers; ++l) {
    if (t < kC * 2 * kC) {
      const int o = t / (2 * kC), f = t % (2 * kC);
      const float w1 = prm[off_W1(l) + o * 2 * kC + f];
      wbf[bf_W1(l) + t] = bf16_bits(w1);
      wbf[bf_W1T(l) + f * kC + o] = bf16_bits(w1);
    }
    if (t < kC * kC) {
      const int o = t / kC, f = t % kC;
      const float w2 = prm[off_W2(l) + t];
      wbf[bf_W2(l) + t] = bf16_bits(w2);
      wbf[bf_W2T(l) + f * kC + o] = bf16_bits(w2);
    }
  }
}

template <int N>
void launch_gemm_tile_test(cudaStream_t s, int M, int K, const __nv_bfloat16 *X, const __nv_bfloat16 *W, float *Y,
                           int *err) {
  const int kblocks = K / 64;
  const size_t smem = (size_t)kblocks * (128 + N) * 128 + 1024;
  UFE_CUDA(cudaFuncSetAttribute(k_gemm_tile_test<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_gemm_tile_test<N><<<M / 128, 128, smem, s>>>(M, K, X, W, Y, err);
  UFE_CUDA(cudaGetLastError());
}

}  // namespace

extern "C" int32_t ufe_umma_gemm_bf16(ufe_ctx *ctx, int32_t M, int32_t N, int32_t K, const uint16_t *X,
                                      const uint16_t *W, float *Y) {
  return guarded(ctx, [&]() -> int32_t {
    UFE_REQUIRE(M > 0 && M % 128 == 0 && (N == 64 || N == 128) && K > 0 && K % 64 == 0 && K <= 256,
                UFE_ERR_INVALID, "umma gemm: need M % 128 == 0, N in {64, 128}, K % 64 == 0, K <= 256");
    UFE_REQUIRE(X && W && Y, UFE_ERR_INVALID, "umma gemm: NULL argument");
    UFE_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const size_t nx = (size_t)M * K, nw = (size_t)N * K, ny = (size_t)M * N;
    uint8_t *buf = (uint8_t *)dev_alloc(nx * 2 + nw * 2 + ny * 4 + 256);
    __nv_bfloat16 *dX = (__nv_bfloat16 *)buf;
    __nv_bfloat16 *dW = dX + nx;
    float *dY = (float *)(buf + ((nx * 2 + nw * 2 + 15) & ~size_t(15)));
    int *err = (int *)(dY + ny);
    int herr = 0;
    try {
      UFE_CUDA(cudaMemcpyAsync(dX, X, nx * 2, cudaMemcpyHostToDevice, s));
      UFE_CUDA(cudaMemcpyAsync(dW, W, nw * 2, cudaMemcpyHostToDevice, s));
      UFE_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
      if (N == 64)
        launch_gemm_tile_test<64>(s, M, K, dX, dW, dY, err);
      else
        launch_gemm_tile_test<128>(s, M, K, dX, dW, dY, err);
      UFE_CUDA(cudaMemcpyAsync(Y, dY, ny * 4, cudaMemcpyDeviceToHost, s));
      UFE_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
      UFE_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
      dev_free(buf);
      throw;
    }
    dev_free(buf);
    UFE_REQUIRE(herr == 0, UFE_ERR_DEVICE, "umma gemm: tensor-core completion timed out");
    return UFE_OK;
  });
}

// ================================================================================================
// Host side
struct GnnMember {
  int64_t n = 0;
  int32_t *nbr = nullptr;
  float *x = nullptr, *y = nullptr, *w = nullptr;   // features, targets, loss weights (sum 1)
};

struct ufe_gnn {
  ufe_ctx *ctx = nullptr;            // device, stream and error text (must outlive the network)
  int device = 0;
  float *prm = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  uint16_t *wbf = nullptr;
  int *err = nullptr;
  int64_t adam_t = 0;
  int64_t cap = 0;                   // node capacity of the work buffers
  float *h[kLayers + 1] = {};
  uint16_t *t[kLayers] = {};
  float *dacc[2] = {}, *dA[2] = {}, *ybuf = nullptr;   // dacc, dA: of the layer above and of this one, in turn
  float *part = nullptr, *dpart = nullptr;             // gradient partials per CTA
  int part_ctas = 0;                                   // that part holds (0.3 MB each)
  double *loss_part = nullptr;
  double *loss_host = nullptr;       // pinned
  // scratch for explicit graphs and mesh features
  int32_t *gnbr = nullptr;
  float *gx = nullptr, *gy = nullptr, *gw = nullptr, *gmask = nullptr;
  int64_t gcap = 0;
  std::vector<GnnMember> data;
};

namespace {

// resident CTAs per SM, as shared memory allows (TMEM: 64, 128, 256, 64 of 512 columns each)
constexpr int kSms = 152;
constexpr size_t kSmemEncoder = kTileBytes + 64 * 128 + 2 * kTileBytes + 1024;
constexpr size_t kSmemLayerFwd = 3 * kTileBytes + 3 * 64 * 128 + 1024;
constexpr size_t kSmemLayerBwd = 5 * kTileBytes + 3 * 64 * 128 + 1024;
constexpr size_t kSmemEncoderBwd = 2 * kTileBytes + 1024;
constexpr int kFwdBlocks = 2 * kSms, kEncBlocks = 3 * kSms, kBwdBlocks = 2 * kSms;
unsigned gnn_grid(int64_t n, int most) { return (unsigned)std::min<int64_t>((n + kTile - 1) / kTile, most); }

void gnn_free_buffers(ufe_gnn *g) {
  for (auto &p : g->h) { dev_free(p); p = nullptr; }
  for (auto &p : g->t) { dev_free(p); p = nullptr; }
  for (auto &p : g->dacc) { dev_free(p); p = nullptr; }
  for (auto &p : g->dA) { dev_free(p); p = nullptr; }
  dev_free(g->ybuf);
  g->ybuf = nullptr;
  g->cap = 0;
}

void gnn_ensure(ufe_gnn *g, int64_t n) {
  if (g->cap >= n) return;
  gnn_free_buffers(g);
  const size_t rows = (size_t)n * kC;
  for (int l = 0; l < kLayers; ++l) g->h[l] = (float *)dev_alloc(rows * 4);
  for (auto &p : g->t) p = (uint16_t *)dev_alloc(rows * 2);
  for (auto &p : g->dacc) p = (float *)dev_alloc(rows * 4);
  for (auto &p : g->dA) p = (float *)dev_alloc(rows * 4);
  g->ybuf = (float *)dev_alloc((size_t)n * kGnnOut * 4);
  g->cap = n;
}

void gnn_ensure_scratch(ufe_gnn *g, int64_t n) {
  if (g->gcap >= n) return;
  g->gcap = 0;
  dev_replace(g->gnbr, 3 * (size_t)n);
  dev_replace(g->gx, kFin * (size_t)n);
  dev_replace(g->gy, kGnnOut * (size_t)n);
  dev_replace(g->gw, n);
  dev_replace(g->gmask, n);
  g->gcap = n;
}

void set_attrs() {
  static bool done = false;
  if (done) return;
  UFE_CUDA(cudaFuncSetAttribute(k_gnn_encoder, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemEncoder));
  auto smem = [](auto kern, size_t bytes) {
    UFE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  };
  smem(k_gnn_layer_fwd<false, false>, kSmemLayerFwd);
  smem(k_gnn_layer_fwd<false, true>, kSmemLayerFwd);
  smem(k_gnn_layer_fwd<true, false>, kSmemLayerFwd);
  smem(k_gnn_layer_fwd<true, true>, kSmemLayerFwd);
  smem(k_gnn_layer_bwd, kSmemLayerBwd);
  smem(k_gnn_encoder_bwd, kSmemEncoderBwd);
  done = true;
}

// forward over a graph already on the device; ybuf gets the outputs.  With targets: loss and decoder-gradient partials,
// dy (in ybuf) and the activations the backward pass reads.
void gnn_forward(ufe_gnn *g, cudaStream_t s, const Graph &gr, const float *x, const float *target, const float *w) {
  set_attrs();
  gnn_ensure(g, gr.n);
  const unsigned G = gnn_grid(gr.n, kFwdBlocks);
  k_gnn_encoder<<<gnn_grid(gr.n, kEncBlocks), kGnnThreads, kSmemEncoder, s>>>(gr, x, g->wbf, g->prm, g->h[0], g->err);
  UFE_CUDA(cudaGetLastError());
  const DecoderArgs dec{g->ybuf, target, w, g->loss_part, g->dpart};
  for (int l = 0; l < kLayers; ++l) {
    const bool last = l == kLayers - 1;
    auto kern = target ? (last ? k_gnn_layer_fwd<true, true> : k_gnn_layer_fwd<true, false>)
                       : (last ? k_gnn_layer_fwd<false, true> : k_gnn_layer_fwd<false, false>);
    kern<<<G, kGnnThreads, kSmemLayerFwd, s>>>(gr, l, g->wbf, g->prm, g->h[l], last ? nullptr : g->h[l + 1], g->t[l],
                                               dec, g->err);
    UFE_CUDA(cudaGetLastError());
  }
}

// backward after gnn_forward with targets: the full gradient in g->grad
void gnn_backward(ufe_gnn *g, cudaStream_t s, const Graph &gr, const float *x) {
  const int G = (int)gnn_grid(gr.n, kBwdBlocks), D = (int)gnn_grid(gr.n, kFwdBlocks);
  if (g->part_ctas < G) {   // networks that only predict have none
    g->part_ctas = 0;
    dev_replace(g->part, (size_t)kPartSets * G * kPart);
    g->part_ctas = G;
  }
  auto set = [&](int q) { return g->part + (int64_t)q * G * kPart; };
  GradIn in{nullptr, nullptr, g->ybuf};
  for (int l = kLayers - 1, c = 0; l >= 0; --l, c ^= 1) {
    k_gnn_layer_bwd<<<G, kGnnThreads, kSmemLayerBwd, s>>>(gr, l, g->wbf, g->prm, in, g->t[l], g->h[l], g->dacc[c],
                                                          g->dA[c], set(1 + 2 * l), set(2 + 2 * l), g->err);
    UFE_CUDA(cudaGetLastError());
    in = GradIn{g->dacc[c], g->dA[c], nullptr};
  }
  k_gnn_encoder_bwd<<<G, kGnnThreads, kSmemEncoderBwd, s>>>(gr, x, in, g->h[0], set(0), g->err);
  UFE_CUDA(cudaGetLastError());
  k_gnn_reduce<<<kReduceBlocks, 256, 0, s>>>(G, D, g->part, g->dpart, g->grad);
  UFE_CUDA(cudaGetLastError());
}

double gnn_loss(ufe_gnn *g, cudaStream_t s, int64_t n) {
  const int64_t nb = gnn_grid(n, kFwdBlocks);
  UFE_CUDA(cudaMemcpyAsync(g->loss_host, g->loss_part, sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
  UFE_CUDA(cudaStreamSynchronize(s));
  double l = 0.0;
  for (int64_t b = 0; b < nb; ++b) l += g->loss_host[b];
  return l;
}

void gnn_check(ufe_gnn *g, cudaStream_t s) {
  int h = 0;
  UFE_CUDA(cudaMemcpyAsync(&h, g->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  UFE_CUDA(cudaStreamSynchronize(s));
  UFE_REQUIRE(h == 0, UFE_ERR_DEVICE, "learned start: a tensor-core completion timed out");
}

void gnn_adam(ufe_gnn *g, cudaStream_t s, float lr) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  g->adam_t += 1;
  const float c1 = 1.f - (float)std::pow((double)b1, (double)g->adam_t);
  const float c2 = 1.f - (float)std::pow((double)b2, (double)g->adam_t);
  k_gnn_adam<<<(kParams + 255) / 256, 256, 0, s>>>(kParams, g->prm, g->grad, g->m, g->v, lr, b1, b2, eps, c1, c2);
  UFE_CUDA(cudaGetLastError());
  k_gnn_pack<<<(kC * 2 * kC + 255) / 256, 256, 0, s>>>(g->prm, g->wbf);
  UFE_CUDA(cudaGetLastError());
}

// weights: He-style uniform initialisation from a 64-bit LCG (host), biases zero
std::vector<float> init_params(uint64_t seed) {
  std::vector<float> p(kParams, 0.f);
  uint64_t st = seed * 6364136223846793005ull + 1442695040888963407ull;
  auto uni = [&]() {
    st = st * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(st >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
  };
  auto fill = [&](int off, int out, int in, double gain) {
    const double a = gain * std::sqrt(3.0 / in);
    for (int i = 0; i < out * in; ++i) p[off + i] = (float)(a * uni());
  };
  fill(kOffWe, kC, kFin, std::sqrt(2.0));
  for (int l = 0; l < kLayers; ++l) {
    fill(off_W1(l), kC, 2 * kC, std::sqrt(2.0));
    fill(off_W2(l), kC, kC, 0.5);   // small residual branches at the start
  }
  fill(kOffWd, kGnnOut, kC, 1.0);
  return p;
}

Graph upload_graph(ufe_gnn *g, cudaStream_t s, int64_t n, const int32_t *nbr, const float *x) {
  gnn_ensure_scratch(g, n);
  for (int64_t i = 0; i < 3 * n; ++i)
    UFE_REQUIRE(nbr[i] >= -1 && nbr[i] < n, UFE_ERR_INVALID, "learned start: neighbour index out of range");
  UFE_CUDA(cudaMemcpyAsync(g->gnbr, nbr, sizeof(int32_t) * 3 * n, cudaMemcpyHostToDevice, s));
  UFE_CUDA(cudaMemcpyAsync(g->gx, x, sizeof(float) * kFin * n, cudaMemcpyHostToDevice, s));
  return Graph{n, g->gnbr};
}

}  // namespace

extern "C" int32_t ufe_gnn_param_count(void) { return kParams; }

extern "C" int32_t ufe_gnn_create(ufe_ctx *ctx, uint64_t seed, ufe_gnn **out) {
  if (!out) return UFE_ERR_INVALID;
  *out = nullptr;
  return guarded(ctx, [&]() -> int32_t {
    UFE_CUDA(cudaSetDevice(ctx->device));
    ufe_gnn *g = new ufe_gnn();
    g->ctx = ctx;
    g->device = ctx->device;
    try {
      g->prm = (float *)dev_alloc(sizeof(float) * kParams);
      g->grad = (float *)dev_alloc(sizeof(float) * kParams);
      g->m = (float *)dev_alloc(sizeof(float) * kParams);
      g->v = (float *)dev_alloc(sizeof(float) * kParams);
      g->wbf = (uint16_t *)dev_alloc(sizeof(uint16_t) * kBfTotal);
      g->err = (int *)dev_alloc(sizeof(int));
      g->dpart = (float *)dev_alloc(sizeof(float) * kFwdBlocks * kDecParts);
      g->loss_part = (double *)dev_alloc(sizeof(double) * kFwdBlocks);
      UFE_CUDA(cudaMallocHost(&g->loss_host, sizeof(double) * kFwdBlocks));
      cudaStream_t s = ctx->stream;
      const std::vector<float> p = init_params(seed);
      UFE_CUDA(cudaMemcpyAsync(g->prm, p.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice, s));
      UFE_CUDA(cudaMemsetAsync(g->grad, 0, sizeof(float) * kParams, s));
      UFE_CUDA(cudaMemsetAsync(g->m, 0, sizeof(float) * kParams, s));
      UFE_CUDA(cudaMemsetAsync(g->v, 0, sizeof(float) * kParams, s));
      UFE_CUDA(cudaMemsetAsync(g->wbf, 0, sizeof(uint16_t) * kBfTotal, s));
      UFE_CUDA(cudaMemsetAsync(g->err, 0, sizeof(int), s));
      k_gnn_pack<<<(kC * 2 * kC + 255) / 256, 256, 0, s>>>(g->prm, g->wbf);
      UFE_CUDA(cudaGetLastError());
      UFE_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
      ufe_gnn_destroy(g);
      throw;
    }
    *out = g;
    return UFE_OK;
  });
}

extern "C" void ufe_gnn_destroy(ufe_gnn *g) {
  if (!g) return;
  // the owning context may already be gone: free through the device, not its stream
  cudaSetDevice(g->device);
  cudaDeviceSynchronize();
  for (auto &m : g->data) {
    dev_free(m.nbr);
    dev_free(m.x);
    dev_free(m.y);
    dev_free(m.w);
  }
  gnn_free_buffers(g);
  void *ptrs[] = {g->prm, g->grad, g->m, g->v, g->wbf, g->err, g->part, g->dpart, g->loss_part,
                  g->gnbr, g->gx, g->gy, g->gw, g->gmask};
  for (void *p : ptrs) dev_free(p);
  if (g->loss_host) cudaFreeHost(g->loss_host);
  delete g;
}

extern "C" int32_t ufe_gnn_get_params(ufe_gnn *g, float *params) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(params, UFE_ERR_INVALID, "NULL params");
    UFE_CUDA(cudaMemcpyAsync(params, g->prm, sizeof(float) * kParams, cudaMemcpyDeviceToHost, g->ctx->stream));
    UFE_CUDA(cudaStreamSynchronize(g->ctx->stream));
    return UFE_OK;
  });
}

extern "C" int32_t ufe_gnn_set_params(ufe_gnn *g, const float *params) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(params, UFE_ERR_INVALID, "NULL params");
    cudaStream_t s = g->ctx->stream;
    UFE_CUDA(cudaMemcpyAsync(g->prm, params, sizeof(float) * kParams, cudaMemcpyHostToDevice, s));
    UFE_CUDA(cudaMemsetAsync(g->m, 0, sizeof(float) * kParams, s));
    UFE_CUDA(cudaMemsetAsync(g->v, 0, sizeof(float) * kParams, s));
    g->adam_t = 0;
    k_gnn_pack<<<(kC * 2 * kC + 255) / 256, 256, 0, s>>>(g->prm, g->wbf);
    UFE_CUDA(cudaGetLastError());
    UFE_CUDA(cudaStreamSynchronize(s));
    return UFE_OK;
  });
}

extern "C" int32_t ufe_gnn_forward(ufe_gnn *g, int64_t n, const int32_t *nbr, const float *x, float *y) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(n >= 1 && nbr && x && y, UFE_ERR_INVALID, "gnn forward: bad arguments");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    cudaStream_t s = g->ctx->stream;
    const Graph gr = upload_graph(g, s, n, nbr, x);
    gnn_forward(g, s, gr, g->gx, nullptr, nullptr);
    UFE_CUDA(cudaMemcpyAsync(y, g->ybuf, sizeof(float) * kGnnOut * n, cudaMemcpyDeviceToHost, s));
    gnn_check(g, s);
    return UFE_OK;
  });
}

extern "C" int32_t ufe_gnn_loss_grad(ufe_gnn *g, int64_t n, const int32_t *nbr, const float *x, const float *target,
                                     const float *w, double *loss, float *grad) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(n >= 1 && nbr && x && target && w, UFE_ERR_INVALID, "gnn loss/grad: bad arguments");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    cudaStream_t s = g->ctx->stream;
    const Graph gr = upload_graph(g, s, n, nbr, x);
    UFE_CUDA(cudaMemcpyAsync(g->gy, target, sizeof(float) * kGnnOut * n, cudaMemcpyHostToDevice, s));
    UFE_CUDA(cudaMemcpyAsync(g->gw, w, sizeof(float) * n, cudaMemcpyHostToDevice, s));
    gnn_forward(g, s, gr, g->gx, g->gy, g->gw);
    gnn_backward(g, s, gr, g->gx);
    if (grad) UFE_CUDA(cudaMemcpyAsync(grad, g->grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost, s));
    const double l = gnn_loss(g, s, n);
    if (loss) *loss = l;
    gnn_check(g, s);
    return UFE_OK;
  });
}

// ---- the mesh path: training data from solves, warm start of a solve ---------------------------
extern "C" int32_t ufe_gnn_dataset_add(ufe_gnn *g, ufe_ctx *mesh_ctx, const float *features_before) {
  if (!g || !mesh_ctx) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(mesh_ctx->device == g->ctx->device, UFE_ERR_INVALID, "gnn and mesh contexts on different devices");
    UFE_REQUIRE(mesh_ctx->has_mesh && mesh_ctx->work, UFE_ERR_INVALID, "gnn dataset: no solved ice state");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    UFE_CUDA(cudaStreamSynchronize(g->ctx->stream));
    cudaStream_t s = mesh_ctx->stream;
    const int64_t n = mesh_ctx->nTri;
    GnnMember m;
    m.n = n;
    m.nbr = (int32_t *)dev_alloc(sizeof(int32_t) * 3 * n);
    m.x = (float *)dev_alloc(sizeof(float) * kFin * n);
    m.y = (float *)dev_alloc(sizeof(float) * kGnnOut * n);
    m.w = (float *)dev_alloc(sizeof(float) * n);
    try {
      gnn_mesh_graph(mesh_ctx, s, m.nbr);
      if (features_before) {
        // features the caller took before the solve (ufe_gnn_features), in the caller's triangle order
        std::vector<float> xi((size_t)kFin * n);
        const std::vector<int32_t> &pt = mesh_ctx->perm_t_h;
        for (int64_t t = 0; t < n; ++t)
          for (int k = 0; k < kFin; ++k) xi[(size_t)t * kFin + k] = features_before[(size_t)pt[t] * kFin + k];
        UFE_CUDA(cudaMemcpyAsync(m.x, xi.data(), sizeof(float) * kFin * n, cudaMemcpyHostToDevice, s));
        UFE_CUDA(cudaStreamSynchronize(s));
      } else {
        gnn_mesh_features(mesh_ctx, s, 0, m.x, nullptr);
      }
      gnn_mesh_velocity(mesh_ctx, s, m.y, false, nullptr);
      gnn_mesh_viscosity(mesh_ctx, s, m.y, false, nullptr);
      // loss weights: triangles with ice, equal weights summing to one
      std::vector<float> hx((size_t)kFin * n);
      UFE_CUDA(cudaMemcpyAsync(hx.data(), m.x, sizeof(float) * kFin * n, cudaMemcpyDeviceToHost, s));
      UFE_CUDA(cudaStreamSynchronize(s));
      int64_t cnt = 0;
      for (int64_t t = 0; t < n; ++t) cnt += hx[(size_t)t * kFin + 13] > 0.f;
      std::vector<float> hw(n);
      for (int64_t t = 0; t < n; ++t) hw[t] = (hx[(size_t)t * kFin + 13] > 0.f && cnt > 0) ? 1.f / (float)cnt : 0.f;
      UFE_CUDA(cudaMemcpyAsync(m.w, hw.data(), sizeof(float) * n, cudaMemcpyHostToDevice, s));
      UFE_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
      dev_free(m.nbr);
      dev_free(m.x);
      dev_free(m.y);
      dev_free(m.w);
      throw;
    }
    g->data.push_back(m);
    return (int32_t)g->data.size();
  });
}

extern "C" int32_t ufe_gnn_dataset_clear(ufe_gnn *g) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_CUDA(cudaStreamSynchronize(g->ctx->stream));
    for (auto &m : g->data) {
      dev_free(m.nbr);
      dev_free(m.x);
      dev_free(m.y);
      dev_free(m.w);
    }
    g->data.clear();
    return UFE_OK;
  });
}

// Features of the mesh context's resident ice state, in the caller's triangle order (nTri x 16).
extern "C" int32_t ufe_gnn_features(ufe_gnn *g, ufe_ctx *mesh_ctx, int32_t use_prev_velocity, float *x) {
  if (!g || !mesh_ctx) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(mesh_ctx->device == g->ctx->device, UFE_ERR_INVALID, "gnn and mesh contexts on different devices");
    UFE_REQUIRE(mesh_ctx->has_mesh && mesh_ctx->work && x, UFE_ERR_INVALID, "gnn features: no ice state");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    cudaStream_t s = mesh_ctx->stream;
    const int64_t n = mesh_ctx->nTri;
    gnn_ensure_scratch(g, n);
    gnn_mesh_features(mesh_ctx, s, use_prev_velocity, g->gx, nullptr);
    std::vector<float> xi((size_t)kFin * n);
    UFE_CUDA(cudaMemcpyAsync(xi.data(), g->gx, sizeof(float) * kFin * n, cudaMemcpyDeviceToHost, s));
    UFE_CUDA(cudaStreamSynchronize(s));
    const std::vector<int32_t> &pt = mesh_ctx->perm_t_h;
    for (int64_t t = 0; t < n; ++t)
      for (int k = 0; k < kFin; ++k) x[(size_t)pt[t] * kFin + k] = xi[(size_t)t * kFin + k];
    return UFE_OK;
  });
}

// Train on the stored members: `epochs` passes, one member per Adam step, member order shuffled
// per epoch with `seed`.  loss_per_epoch (optional, epochs entries): mean training loss.
extern "C" int32_t ufe_gnn_train(ufe_gnn *g, int32_t epochs, float lr, uint64_t seed, float *loss_per_epoch,
                                 double *device_ms) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(epochs >= 0 && lr > 0.f, UFE_ERR_INVALID, "gnn train: bad arguments");
    UFE_REQUIRE(!g->data.empty(), UFE_ERR_INVALID, "gnn train: empty dataset");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    cudaStream_t s = g->ctx->stream;
    std::vector<int> order(g->data.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    uint64_t st = seed * 2862933555777941757ull + 3037000493ull;
    float total_ms = 0.f;
    for (int e = 0; e < epochs; ++e) {
      for (size_t i = order.size(); i > 1; --i) {   // Fisher-Yates
        st = st * 6364136223846793005ull + 1442695040888963407ull;
        std::swap(order[i - 1], order[(size_t)((st >> 33) % i)]);
      }
      double sum = 0.0;
      UFE_CUDA(cudaEventRecord(g->ctx->ev0, s));
      for (int idx : order) {
        const GnnMember &m = g->data[idx];
        const Graph gr{m.n, m.nbr};
        gnn_forward(g, s, gr, m.x, m.y, m.w);
        gnn_backward(g, s, gr, m.x);
        gnn_adam(g, s, lr);
        if (loss_per_epoch) sum += gnn_loss(g, s, m.n);
      }
      UFE_CUDA(cudaEventRecord(g->ctx->ev1, s));
      UFE_CUDA(cudaEventSynchronize(g->ctx->ev1));
      float ms = 0.f;
      UFE_CUDA(cudaEventElapsedTime(&ms, g->ctx->ev0, g->ctx->ev1));
      total_ms += ms;
      if (loss_per_epoch) loss_per_epoch[e] = (float)(sum / (double)order.size());
    }
    gnn_check(g, s);
    if (device_ms) *device_ms = total_ms;
    return UFE_OK;
  });
}

// Mean loss of the stored members (evaluation; no update).
extern "C" int32_t ufe_gnn_evaluate(ufe_gnn *g, double *mean_loss) {
  if (!g) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(!g->data.empty() && mean_loss, UFE_ERR_INVALID, "gnn evaluate: empty dataset");
    cudaStream_t s = g->ctx->stream;
    double sum = 0.0;
    for (const GnnMember &m : g->data) {
      gnn_forward(g, s, Graph{m.n, m.nbr}, m.x, m.y, m.w);
      sum += gnn_loss(g, s, m.n);
    }
    gnn_check(g, s);
    *mean_loss = sum / (double)g->data.size();
    return UFE_OK;
  });
}

// Warm start: predict the velocity of the mesh context's resident ice state and store it as the
// resident velocity, so that ufe_solve_ssa_resident / ufe_solve_diva_resident with cold_start = 0
// start the Picard loop from it; `smooth_passes` averaging passes over each triangle and its
// neighbours take the prediction's small-scale noise out first.  With `with_viscosity` the
// predicted vertically averaged viscosity is stored on the vertices as well and the next solve's
// first Picard iteration uses it in place of Glen's law (SSA: the viscosity; DIVA: every layer).
// Kernels one prediction launches: graph, features, encoder, the layers (the last with the decoder), velocity store,
// two per smoothing pass, and the viscosity store.
extern "C" int32_t ufe_gnn_predict_kernels(int32_t smooth_passes) {
  return 1 + 1 + (1 + kLayers) + 1 + 2 * (smooth_passes > 0 ? smooth_passes : 0);
}

extern "C" int32_t ufe_gnn_predict_start(ufe_gnn *g, ufe_ctx *mesh_ctx, int32_t use_prev_velocity,
                                         int32_t smooth_passes, int32_t with_viscosity, double *device_ms) {
  if (!g || !mesh_ctx) return UFE_ERR_INVALID;
  return guarded(g->ctx, [&]() -> int32_t {
    UFE_REQUIRE(mesh_ctx->device == g->ctx->device, UFE_ERR_INVALID, "gnn and mesh contexts on different devices");
    UFE_REQUIRE(mesh_ctx->has_mesh && mesh_ctx->work, UFE_ERR_INVALID, "gnn predict: upload the ice state first");
    UFE_CUDA(cudaSetDevice(g->ctx->device));
    UFE_CUDA(cudaStreamSynchronize(g->ctx->stream));
    cudaStream_t s = mesh_ctx->stream;
    const int64_t n = mesh_ctx->nTri;
    gnn_ensure_scratch(g, n);
    UFE_CUDA(cudaEventRecord(mesh_ctx->ev0, s));
    gnn_mesh_graph(mesh_ctx, s, g->gnbr);
    gnn_mesh_features(mesh_ctx, s, use_prev_velocity, g->gx, g->gmask);
    gnn_forward(g, s, Graph{n, g->gnbr}, g->gx, nullptr, nullptr);
    gnn_mesh_velocity(mesh_ctx, s, g->ybuf, true, g->gmask);
    if (smooth_passes > 0) gnn_mesh_smooth(mesh_ctx, s, smooth_passes, g->gmask);
    if (with_viscosity) gnn_mesh_viscosity(mesh_ctx, s, g->ybuf, true, g->gmask);
    UFE_CUDA(cudaEventRecord(mesh_ctx->ev1, s));
    gnn_check(g, s);
    if (device_ms) {
      float ms = 0.f;
      UFE_CUDA(cudaEventElapsedTime(&ms, mesh_ctx->ev0, mesh_ctx->ev1));
      *device_ms = ms;
    }
    return UFE_OK;
  });
}

extern "C" int32_t ufe_gnn_predict_velocity(ufe_gnn *g, ufe_ctx *mesh_ctx, int32_t use_prev_velocity,
                                            int32_t smooth_passes, double *device_ms) {
  return ufe_gnn_predict_start(g, mesh_ctx, use_prev_velocity, smooth_passes, 0, device_ms);
}
