// e2d_mlp_deep.cu — the deep warm-start network on the tensor cores: 5 input
// features (padded to 16), four hidden layers of 256 units with GELU (tanh
// form), 4 outputs (padded to 16).
//
//   net_kernel<false>  rows -> outputs: all five layers of a 128-row tile in one
//                      kernel, the activations in shared memory between layers
//   net_kernel<true>   forward, loss and the deltas of every layer of a tile,
//                      leaving activations and deltas (BF16) for dw_kernel
//   dw_kernel          every layer's weight and bias gradients from them
//   adam_kernel        the update, and the BF16 copies of the new weights
//
// A pair of CTAs (a cluster) shares a tile: each computes 128 of a layer's
// 256 columns, so its half of the weights (64 KB) and two activation buffers
// (64 KB each) fit one SM, and writes its half of the next activations into
// both CTAs' shared memory.  The 64 tiles of an 8,192-row minibatch thus use
// 128 SMs.  What bounds net_kernel is the epilogue: tanhf and the GELU
// arithmetic, about 34 instructions per activation (16 warps per SM to issue
// them, issue active 46 %), and the pair's exchange between layers; the next
// weights arrive (cp.async.bulk) under it.  Measured against a kernel per
// layer with activations in HBM and 4 warps per SM (B200): prediction of 300,007
// rows 2,005 -> 593 us, a training step on 8,192 rows 753 -> 94 us
// (net_kernel 46, dw_kernel 34, adam_kernel 7; 105 us before the kernels of a
// step were programmatic dependents of one another and read the minibatch's
// rows from host memory instead of after a copy).  Swizzled operand tiles were
// measured too (no faster: the products are not the bound; their strided
// writes to the peer cost 10 %).
//
// Every product is one elected thread issuing tcgen05.mma of BF16 operands
// in shared memory (e2d_tc.cuh) into an FP32 TMEM accumulator, committed to an
// mbarrier that is waited on with a bounded spin; a wait that runs out sets the
// error word, the remaining products are skipped and the TMEM is freed.
// Activations, deltas and weights live in global memory in the canonical
// operand layout (tiles of 128 rows), so that a tile, half or chunk of one is
// a plain bulk copy, and the weight gradients read the same tiles as MN-major
// operands: no transposed copies.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "../../include/cffc_e2d.h"
#include "e2d_pdl.cuh"
#include "e2d_tc.cuh"

using namespace e2d;

namespace {

constexpr int DF = 16, DH = 256, DO = 16, DO_USED = 4, DNL = 4;  // features, width, outputs (padded), hidden layers
constexpr int NLAYER = DNL + 1;
constexpr int TILE = 128;          // rows per tile (UMMA M)
constexpr int HALF = DH / 2;       // columns of a layer per CTA of a pair
constexpr int NT = 512;            // threads of net_kernel: 4 warps per 32 TMEM lanes
constexpr int RC = 64;             // rows per chunk of the weight-gradient product
constexpr uint32_t WAIT_ITERS = 1u << 22;

__host__ __device__ constexpr int layer_in(int l) { return l == 0 ? DF : DH; }
__host__ __device__ constexpr int layer_out(int l) { return l == DNL ? DO : DH; }
// flat parameter vector: W_l [out][in] then b_l [out], layers 0..4
__host__ __device__ constexpr int w_off(int l) {
  return l == 0 ? 0 : DH * DF + DH + (l - 1) * (DH * DH + DH) - (l == NLAYER ? (DH - DO) * (DH + 1) : 0);
}
__host__ __device__ constexpr int b_off(int l) { return w_off(l) + layer_out(l) * layer_in(l); }
constexpr int NPARAM = w_off(NLAYER);
static_assert(NPARAM == w_off(DNL) + DO * DH + DO, "parameter layout");

__device__ __forceinline__ uint16_t f2bf(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float(uint32_t(b) << 16); }

// GELU, tanh form, and its derivative (null: not wanted), from one tanh.
__device__ __forceinline__ float gelu(float z, float* prime) {
  const float u = 0.7978845608028654f * (z + 0.044715f * z * z * z);
  const float t = tanhf(u);
  if (prime) *prime = 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * 0.7978845608028654f * (1.0f + 0.134145f * z * z);
  return 0.5f * z * (1.0f + t);
}

__device__ __forceinline__ uint4 pack8(const float* v) {
  uint32_t k[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) k[q] = uint32_t(f2bf(v[2 * q])) | (uint32_t(f2bf(v[2 * q + 1])) << 16);
  return make_uint4(k[0], k[1], k[2], k[3]);
}

__device__ __forceinline__ void cta_sync_async() {
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
}

// Commit (thread 0) and bounded wait of every thread; CTA-uniform result.
__device__ __forceinline__ bool complete(uint64_t* bar, uint32_t& phase) {
  if (threadIdx.x == 0) tc::mma_commit(bar);
  const bool ok = tc::mbar_wait_warp(bar, phase, WAIT_ITERS);
  phase ^= 1u;
  tc::fence_after_sync();
  return __syncthreads_and(ok) != 0;
}

// Tiles of 128 rows (activations, deltas, features) are column-chunk tiles
// (e2d_tc.cuh): any range of columns is contiguous, so a CTA's half of a tile
// goes to global memory, and a piece of one to the weight gradients, as one
// bulk copy, and a warp's 32 rows of a chunk are 512 bytes on end.  Weights
// are K-major by row group: a half of the rows is contiguous.
constexpr int CHUNK = TILE * 16;
__device__ __forceinline__ uint32_t tile_off(int r, int k) {  // byte of element (r, k)
  return uint32_t((k >> 3) * CHUNK + r * 16 + (k & 7) * 2);
}

// D[128][N] = A[128][K] B[N][K]^T, one thread: A a tile, B weights.
__device__ __forceinline__ void product(uint32_t d, const uint8_t* A, const uint8_t* Bm, int K, int N) {
  const uint32_t id = tc::idesc_bf16(TILE, N), a0 = tc::smem_addr(A), b0 = tc::smem_addr(Bm);
  for (int t = 0; t < K / 16; ++t)
    tc::mma_bf16(d, tc::smem_desc(a0 + 2 * CHUNK * t, CHUNK, 128), tc::smem_desc(b0 + 256 * t, 128, K * 16), id,
                 t > 0 ? 1u : 0u);
}

// Four floats of a caller's array: one 16-byte access where its base is
// 16-byte aligned (vec), else four.
__device__ __forceinline__ float4 ld4(const float* p, int vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

struct NetArgs {
  const float *X, *T;         // [*][16], [*][4]
  int vec;                    // X, T and Y are 16-byte aligned
  const int* idx;             // rows of the pass, in host memory (null: 0 .. n-1)
  int n;
  float inv_n;
  const uint16_t *wk, *wt;    // BF16 weights and transposes, canonical tiles at the parameter offsets
  const float* p;             // FP32 parameters (biases)
  float* Y;                   // [n][4] (forward)
  uint16_t *xb, *dy;          // tiles [128][16] (train)
  uint16_t *act[DNL], *dz[DNL];  // tiles [128][256] (train)
  float* gp;                  // GELU' of the CTA's current tile, [CTA][4][128 x 128] (train)
  double* lpart;              // loss sums, [clusters] (train)
  int* err;
};

struct NetSmem {
  uint8_t A[2][TILE * DH * 2];    // activations / deltas, [128][256]
  uint8_t W[HALF * DH * 2];       // this CTA's half of a hidden layer's weights or transpose
  uint8_t W0[HALF * DF * 2], W4[DO * DH * 2], W4T[HALF * DO * 2];
  uint8_t X[TILE * DF * 2], dY[TILE * DO * 2];
  float b[DNL][HALF], b4[DO];
  int idx[TILE];                  // rows of the tile
  double lw[4];
  uint64_t bar, wbar;
  uint32_t taddr;
};

template <bool TRAIN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NT, 1) net_kernel(const __grid_constant__ NetArgs a) {
  extern __shared__ __align__(1024) uint8_t smraw[];
  NetSmem& s = *reinterpret_cast<NetSmem*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = tc::cluster_rank();
  const int cluster = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  const int ntiles = (a.n + TILE - 1) / TILE;
  // what depends on no earlier kernel: barriers, TMEM, the first tile's rows
  if (tid == 0) {
    tc::mbar_init(&s.bar, 1);
    tc::mbar_init(&s.wbar, 1);
  }
  if (warp == 0) tc::tmem_alloc(&s.taddr, 256);
  auto row_of = [&](int tile) {
    const int g = tile * TILE + tid;
    return tid < TILE && g < a.n ? (a.idx ? a.idx[g] : g) : 0;
  };
  int next_row = row_of(cluster);
  pdl_wait();
  // constant operands (16 bytes a thread) and biases
  auto copy = [&](uint8_t* dst, const uint16_t* src, int bytes) {
    for (int q = tid; q < bytes / 16; q += NT) reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<const uint4*>(src)[q];
  };
  copy(s.W0, a.wk + w_off(0) + rank * HALF * DF, HALF * DF * 2);
  copy(s.W4, a.wk + w_off(DNL), DO * DH * 2);
  if (TRAIN) copy(s.W4T, a.wt + w_off(DNL) + rank * HALF * DO, HALF * DO * 2);
  if (tid < HALF)
    for (int l = 0; l < DNL; ++l) s.b[l][tid] = a.p[b_off(l) + rank * HALF + tid];
  if (tid < DO) s.b4[tid] = a.p[b_off(DNL) + tid];
  cta_sync_async();
  tc::cluster_sync();  // the peer runs: its shared memory may be written
  const uint32_t tm = s.taddr, td = tm, ty = tm + HALF;  // hidden products, outputs
  // this thread's TMEM lane (row of the tile) and 32 of the CTA's 128 columns
  const int row = 32 * (warp & 3) + lane, cg = warp >> 2;
  const uint32_t lane_base = uint32_t(32 * (warp & 3)) << 16;
  const uint32_t roff = tile_off(row, 0);
  const uint32_t peer = rank ^ 1u;
  const uint32_t pA[2] = {tc::peer_addr(tc::smem_addr(s.A[0]), peer), tc::peer_addr(tc::smem_addr(s.A[1]), peer)};
  float4* gp = TRAIN ? reinterpret_cast<float4*>(a.gp) + size_t(blockIdx.x) * (DNL * TILE * HALF / 4) : nullptr;
  uint32_t phase = 0, wphase = 0;
  int wissued = 0, wwaited = 0;
  bool ok = true;
  double lsum = 0.0;
  // one hidden layer's weights (its transpose for the deltas) into s.W
  auto load_w = [&](const uint16_t* src) {
    ++wissued;
    if (tid == 0) {
      tc::mbar_expect_tx(&s.wbar, HALF * DH * 2);
      for (int q = 0; q < 4; ++q)
        tc::bulk_load(s.W + q * (HALF * DH / 2), src + rank * HALF * DH + q * (HALF * DH / 4), HALF * DH / 2, &s.wbar);
    }
  };
  auto wait_w = [&]() {
    const bool got = tc::mbar_wait_warp(&s.wbar, wphase, WAIT_ITERS);
    wphase ^= 1u;
    ++wwaited;
    ok = __syncthreads_and(got && ok) != 0;
  };
  // both CTAs' halves of the next operand are in buffer nxt; this CTA's half
  // goes to global memory too (out not null)
  auto pair_sync = [&](int nxt, uint16_t* out) {
    asm volatile("fence.proxy.async;" ::: "memory");
    tc::fence_before_sync();
    tc::cluster_sync();
    tc::fence_after_sync();
    if (tid == 0) {
      asm volatile("fence.proxy.async;" ::: "memory");
      if (out) tc::bulk_store(out + rank * HALF * TILE, s.A[nxt] + rank * HALF * TILE * 2, HALF * TILE * 2);
    }
  };
  // 16 values of this thread's row, columns rank * 128 + 32 cg + 16 h of a
  // layer, as BF16 into buffer nxt, the peer's too (both)
  auto put16 = [&](const float* v, int h, int nxt, bool both) {
    const int c = rank * (HALF / 8) + 4 * cg + 2 * h;  // chunk of 8 columns
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint4 k = pack8(v + 8 * q);
      const uint32_t off = roff + (c + q) * CHUNK;
      *reinterpret_cast<uint4*>(s.A[nxt] + off) = k;
      if (both) tc::st_peer(pA[nxt] + off, k);
    }
  };
  if (cluster < ntiles) load_w(a.wk + w_off(1));
  for (int tile = cluster; tile < ntiles; tile += nclusters) {
    const int grow = tile * TILE + row;
    const bool valid = grow < a.n, more = tile + nclusters < ntiles;
    if (tid < TILE) s.idx[tid] = next_row;
    if (more) next_row = row_of(tile + nclusters);
    __syncthreads();
    if (tid < 2 * TILE) {  // X: 8 features a thread
      const int r = tid & (TILE - 1), c = tid >> 7, g = tile * TILE + r;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (g < a.n) {
        const float* x = a.X + size_t(s.idx[r]) * DF + 8 * c;
        const float4 x0 = ld4(x, a.vec), x1 = ld4(x + 4, a.vec);
        v[0] = x0.x; v[1] = x0.y; v[2] = x0.z; v[3] = x0.w; v[4] = x1.x; v[5] = x1.y; v[6] = x1.z; v[7] = x1.w;
      }
      const uint4 k = pack8(v);
      const uint32_t off = tile_off(r, 8 * c);
      *reinterpret_cast<uint4*>(s.X + off) = k;
      if (TRAIN && rank == 0)
        *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(a.xb) + size_t(tile) * (TILE * DF * 2) + off) = k;
    }
    cta_sync_async();
    // ---- hidden layers: H_l = gelu(A W_l^T + b_l) --------------------------
    for (int l = 0; l < DNL; ++l) {
      if (l > 0) wait_w();
      if (ok) {
        if (tid == 0) {
          if (l == 0) product(td, s.X, s.W0, DF, HALF);
          else product(td, s.A[(l - 1) & 1], s.W, DH, HALF);
          if (TRAIN) tc::bulk_store_read<1>();  // the buffer written next has reached global memory
        }
        ok = complete(&s.bar, phase);
      }
      if (l > 0) {  // the weights are read: the next ones arrive under the epilogue
        if (l < DNL - 1) load_w(a.wk + w_off(l + 1));
        else if (TRAIN) load_w(a.wt + w_off(DNL - 1));
        else if (more) load_w(a.wk + w_off(1));
      }
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        float v[16], g[16];
        tc::tmem_ld16(td + lane_base + uint32_t(32 * cg + 16 * h), v);
        const float4* b = reinterpret_cast<const float4*>(&s.b[l][32 * cg + 16 * h]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 bq = b[q];
          v[4 * q] += bq.x; v[4 * q + 1] += bq.y; v[4 * q + 2] += bq.z; v[4 * q + 3] += bq.w;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float y = gelu(v[q], TRAIN ? &g[q] : nullptr);
          v[q] = !TRAIN || valid ? y : 0.0f;  // rows past the last stay zero in the gradients
        }
        if (TRAIN)
#pragma unroll
          for (int q = 0; q < 4; ++q)
            gp[(((l * 4 + cg) * 2 + h) * 4 + q) * TILE + row] =
                make_float4(g[4 * q], g[4 * q + 1], g[4 * q + 2], g[4 * q + 3]);
        put16(v, h, l & 1, true);
      }
      pair_sync(l & 1, TRAIN ? a.act[l] + size_t(tile) * (TILE * DH) : nullptr);
    }
    // ---- outputs -------------------------------------------------------------
    if (ok && (TRAIN || rank == 0)) {
      if (tid == 0) product(ty, s.A[(DNL - 1) & 1], s.W4, DH, DO);
      ok = complete(&s.bar, phase);
    }
    if (!TRAIN) {
      if (rank == 0 && warp < 4) {
        float y[16];
        tc::tmem_ld16(ty + lane_base, y);
        float* o = a.Y + size_t(grow) * DO_USED;
        if (valid && a.vec)
          *reinterpret_cast<float4*>(o) = make_float4(y[0] + s.b4[0], y[1] + s.b4[1], y[2] + s.b4[2], y[3] + s.b4[3]);
        else if (valid)
#pragma unroll
          for (int q = 0; q < DO_USED; ++q) o[q] = y[q] + s.b4[q];
      }
      tc::fence_before_sync();
      continue;
    }
    // ---- loss and the output deltas dY = bf16(2 (y - t) / n) -------------------
    if (warp < 4) {
      float y[16], d[16];
      tc::tmem_ld16(ty + lane_base, y);
#pragma unroll
      for (int q = 0; q < 16; ++q) d[q] = 0.0f;
      if (valid) {
        const float4 t = ld4(a.T + size_t(s.idx[row]) * DO_USED, a.vec);
        const float tq[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int q = 0; q < DO_USED; ++q) {
          const float e = (y[q] + s.b4[q]) - tq[q];
          lsum += double(e) * double(e);
          d[q] = 2.0f * e * a.inv_n;
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint4 k = pack8(d + 8 * q);
        const uint32_t off = tile_off(row, 8 * q);
        *reinterpret_cast<uint4*>(s.dY + off) = k;
        if (rank == 0)
          *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(a.dy) + size_t(tile) * (TILE * DO * 2) + off) = k;
      }
    }
    cta_sync_async();
    // ---- hidden deltas: dZ_l = (dZ_{l+1} W_{l+1}) * gelu'(Z_l) -----------------
    for (int l = DNL - 1; l >= 0; --l) {
      const bool top = l == DNL - 1;
      if (!top) wait_w();
      if (ok) {
        if (tid == 0) {
          if (top) product(td, s.dY, s.W4T, DO, HALF);
          else product(td, s.A[l & 1], s.W, DH, HALF);
          tc::bulk_store_read<1>();
        }
        ok = complete(&s.bar, phase);
      }
      if (!top) {
        if (l > 0) load_w(a.wt + w_off(l));
        else if (more) load_w(a.wk + w_off(1));
      }
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        float v[16];
        tc::tmem_ld16(td + lane_base + uint32_t(32 * cg + 16 * h), v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 g = gp[(((l * 4 + cg) * 2 + h) * 4 + q) * TILE + row];
          v[4 * q] *= g.x; v[4 * q + 1] *= g.y; v[4 * q + 2] *= g.z; v[4 * q + 3] *= g.w;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = valid ? v[q] : 0.0f;
        // the next product (layer l - 1) reads buffer (l - 1) & 1
        put16(v, h, (l - 1) & 1, l > 0);
      }
      pair_sync((l - 1) & 1, a.dz[l] + size_t(tile) * (TILE * DH));
    }
  }
  if (TRAIN && rank == 0 && warp < 4) {
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) s.lw[warp] = lsum;
  }
  if (wissued > wwaited) tc::mbar_wait(&s.wbar, wphase, WAIT_ITERS);  // no copy outlives the CTA
  if (TRAIN && tid == 0) tc::bulk_store_done();
  if (!ok && tid == 0) atomicExch(a.err, 1);
  tc::fence_before_sync();
  tc::cluster_sync();
  tc::fence_after_sync();
  if (TRAIN && rank == 0 && tid == 0) a.lpart[cluster] = ((s.lw[0] + s.lw[1]) + s.lw[2]) + s.lw[3];
  if (warp == 0) tc::tmem_dealloc(tm, 256);
}

// ---- weight and bias gradients -----------------------------------------------
// dW_l = sum over rows of dZ_l^T A_l, the rows in groups of `rows` (a multiple
// of 64): a group is accumulated by the tensor core, the groups are added in
// order in FP32 registers, so the sum is the same whichever SM forms it.  One
// CTA per 128 x DWN piece of a layer's gradient walks all groups: one warp
// brings the tiles' columns of both operands (one bulk copy each, a ring of
// DWS stages), DWI warps issue the products of a group each in turn (a product
// of 64 rows is four small MMAs, so one thread's issue rate bounds it: 74 us
// with one such warp, 34 with four, 8,192 rows), four warps add.  Before,
// every group's gradient went to a slot and the slots were summed: 33 MB a
// layer each way, 430 us a step.
constexpr int DWN = 32;                            // columns of a piece
constexpr int DWS = 5;                             // stages
constexpr int DWB = 256 / DWN;                             // accumulators: a group's product, read and release overlap the others'
constexpr int DW_P = TILE * HALF * 2, DW_Q = TILE * DWN * 2;  // bytes of a tile's operands
constexpr int DW_HID = (DNL - 1) * 2 * (DH / DWN);  // pieces of the 256 x 256 layers
constexpr int DW_ITEMS = DW_HID + 4;               // and two halves each of the first and the output layer
constexpr int BCOLS = 16;                          // columns of a bias piece: two threads a row, 144 groups at a time
constexpr int DW_BIAS = DNL * (DH / BCOLS) + 1;    // bias pieces of the hidden layers, and the outputs'
constexpr int DWI = 4;                             // warps that issue products, a group each in turn
constexpr int DW_THREADS = 32 * (4 + 1 + DWI);
static_assert(DWB * DWN == 256, "TMEM columns: a power of two, at least 32");
static_assert(DWB / 2 <= DWS, "a summed group lies within the ring");
static_assert(DF == 16 && DO == 16, "the narrow layers are one piece of 16 columns");

struct DwArgs {
  const uint16_t *xb, *dy;
  const uint16_t *act[DNL], *dz[DNL];
  int n, rows, brows;  // rows per group of the products, of the bias sums
  float* g;
  int* err;
};
struct DwSmem {
  uint8_t P[DWS][DW_P], Q[DWS][DW_Q];
  uint64_t full[DWS], empty[DWS], dfull[DWB], dempty[DWB], turn[DWI];
  uint32_t taddr;
};
constexpr int BIAS_MAX_GROUPS = 512;  // at most one group per SM
static_assert(DO == BCOLS && sizeof(DwSmem) >= BIAS_MAX_GROUPS * BCOLS * 4, "bias partial sums fit");

// db_l: the rows in groups of brows, each summed in row order, then the
// groups in order.  A thread sums 8 columns (16 bytes a row).
__device__ void bias_piece(const DwArgs& a, int item, float* part) {
  const bool hid = item < DNL * (DH / BCOLS);
  const int l = hid ? item / (DH / BCOLS) : DNL, c0 = hid ? BCOLS * (item % (DH / BCOLS)) : 0;
  const int sub = threadIdx.x / (BCOLS / 8), c = threadIdx.x % (BCOLS / 8), nsub = DW_THREADS / (BCOLS / 8);
  const uint8_t* D = reinterpret_cast<const uint8_t*>(hid ? a.dz[l] : a.dy) + tile_off(0, c0 + 8 * c);
  const size_t tile = TILE * 2 * (hid ? DH : DO);
  const int groups = (a.n + a.brows - 1) / a.brows;
  for (int k = sub; k < groups; k += nsub) {
    const int r0 = k * a.brows, r1 = min(a.n, r0 + a.brows);
    float t[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
    for (int r = r0; r < r1; ++r) {
      const uint4 v = *reinterpret_cast<const uint4*>(D + (r >> 7) * tile + tile_off(r & (TILE - 1), 0));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        t[2 * e] += bf2f(uint16_t(w[e]));
        t[2 * e + 1] += bf2f(uint16_t(w[e] >> 16));
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) part[k * BCOLS + 8 * c + e] = t[e];
  }
  __syncthreads();
  if (threadIdx.x < BCOLS) {
    float t = 0.0f;
#pragma unroll 8
    for (int k = 0; k < groups; ++k) t += part[k * BCOLS + threadIdx.x];
    a.g[b_off(l) + c0 + threadIdx.x] = hid || threadIdx.x < DO_USED ? t : 0.0f;
  }
}

__global__ void __launch_bounds__(DW_THREADS, 1) dw_kernel(const __grid_constant__ DwArgs a) {
  extern __shared__ __align__(1024) uint8_t smraw[];
  DwSmem& s = *reinterpret_cast<DwSmem*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, item = blockIdx.x;
  if (item >= DW_ITEMS) {
    pdl_wait();
    bias_piece(a, item - DW_ITEMS, reinterpret_cast<float*>(smraw));
    return;
  }
  const bool hid = item < DW_HID, last = item >= DW_HID + 2;
  const int l = hid ? 1 + item / (2 * (DH / DWN)) : (last ? DNL : 0);
  const int half = hid ? (item / (DH / DWN)) & 1 : item & 1, nt = hid ? item % (DH / DWN) : 0;
  const int ncol = hid ? DWN : 16;
  const uint32_t qbytes = TILE * 2 * ncol;
  const uint8_t* P = reinterpret_cast<const uint8_t*>(last ? a.act[DNL - 1] : a.dz[l]) + half * DW_P;
  const uint8_t* Q = reinterpret_cast<const uint8_t*>(hid ? a.act[l - 1] : (last ? a.dy : a.xb)) + nt * DW_Q;
  const size_t qtile = hid ? TILE * DH * 2 : qbytes;  // bytes of a tile of Q's array
  if (tid == 0) {
    for (int k = 0; k < DWS; ++k) {
      tc::mbar_init(&s.full[k], 1);
      tc::mbar_init(&s.empty[k], 2);  // the tile's two chunks of 64 rows
    }
    for (int k = 0; k < DWB; ++k) {
      tc::mbar_init(&s.dfull[k], 1);
      tc::mbar_init(&s.dempty[k], 4);
    }
    for (int k = 0; k < DWI; ++k) tc::mbar_init(&s.turn[k], 1);
  }
  if (warp == 0) tc::tmem_alloc(&s.taddr, DWB * DWN);
  pdl_wait();
  cta_sync_async();
  const uint32_t tm = s.taddr;
  const int nchunk = (a.n + RC - 1) / RC, per = a.rows / RC, ngroup = (nchunk + per - 1) / per;
  float acc[DWN];
#pragma unroll
  for (int q = 0; q < DWN; ++q) acc[q] = 0.0f;
  bool ok = true;
  const int ntiles = (a.n + TILE - 1) / TILE;
  if (warp == 4) {  // copies
    int k = 0;
    for (; k < ntiles; ++k) {
      const int st = k % DWS;
      if (k >= DWS) ok = tc::mbar_wait_warp(&s.empty[st], uint32_t(k / DWS - 1) & 1u, WAIT_ITERS);
      if (!ok) break;
      if (lane == 0) {
        tc::mbar_expect_tx(&s.full[st], DW_P + qbytes);
        tc::bulk_load(s.P[st], P + size_t(k) * (TILE * DH * 2), DW_P, &s.full[st]);
        tc::bulk_load(s.Q[st], Q + k * qtile, qbytes, &s.full[st]);
      }
      __syncwarp();
    }
    for (int j = max(0, k - DWS); j < k; ++j) {  // no product and, stopped early, no copy outlives the CTA
      if (ok) ok = tc::mbar_wait_warp(&s.empty[j % DWS], uint32_t(j / DWS) & 1u, WAIT_ITERS);
      else tc::mbar_wait(&s.full[j % DWS], uint32_t(j / DWS) & 1u, WAIT_ITERS);
    }
  } else if (warp > 4) {  // products: group after group, DWI warps in turn, 64 rows at a time
    // A wait on full[] tells a phase by its parity, so nobody may wait for a
    // tile before the one DWS earlier has landed.  With one chunk a group the
    // accumulators see to that: a group waits until the one DWB earlier, DWB / 2
    // tiles back, and all before it are summed.  Longer groups: a group's warp
    // hands on to the next group's once it has seen the last of its tiles; by
    // then every tile up to that one has been seen, in order.  (Handed on with
    // one chunk a group too, a training step on 8,192 rows took 100 us, not 94.)
    if (lane == 0) {
      const uint32_t id = tc::idesc_bf16_t(TILE, ncol);
      const bool turns = per > 1;
      uint32_t tphase = 0;
      for (int grp = warp - 5; grp < ngroup && ok; grp += DWI) {
        const int buf = grp % DWB, k1 = min(nchunk, (grp + 1) * per);
        if (grp >= DWB) ok = tc::mbar_wait(&s.dempty[buf], uint32_t(grp / DWB - 1) & 1u, WAIT_ITERS);
        if (turns && grp > 0) {
          ok = ok && tc::mbar_wait(&s.turn[warp - 5], tphase, WAIT_ITERS);
          tphase ^= 1u;
        }
        bool handed = !turns || grp + 1 >= ngroup;
        for (int k = grp * per; k < k1; ++k) {
          const int tile = k >> 1, st = tile % DWS;
          ok = ok && tc::mbar_wait(&s.full[st], uint32_t(tile / DWS) & 1u, WAIT_ITERS);
          if (!ok) break;
          if (!handed && tile == (k1 - 1) >> 1) {
            tc::mbar_arrive(&s.turn[(grp + 1) % DWI]);
            handed = true;
          }
          tc::fence_after_sync();
          const uint32_t p0 = tc::smem_addr(s.P[st]) + (k & 1) * (CHUNK / 2);
          const uint32_t q0 = tc::smem_addr(s.Q[st]) + (k & 1) * (CHUNK / 2);
#pragma unroll
          for (int t = 0; t < RC / 16; ++t)  // 16 rows: two row groups
            tc::mma_bf16(tm + buf * DWN, tc::smem_desc(p0 + 256 * t, 128, CHUNK), tc::smem_desc(q0 + 256 * t, 128, CHUNK),
                         id, (k > grp * per || t > 0) ? 1u : 0u);
          if (k == k1 - 1) tc::mma_commit(&s.dfull[buf]);
          tc::mma_commit(&s.empty[st]);
          if (k == nchunk - 1 && !(k & 1)) tc::mma_commit(&s.empty[st]);  // the last tile's missing half
        }
      }
    }
    ok = __shfl_sync(0xffffffffu, int(ok), 0) != 0;
  } else {  // sums: TMEM lane = row of the piece
    const uint32_t lane_base = uint32_t(32 * warp) << 16;
    for (int grp = 0; grp < ngroup && ok; ++grp) {
      const int buf = grp % DWB;
      ok = tc::mbar_wait_warp(&s.dfull[buf], uint32_t(grp / DWB) & 1u, WAIT_ITERS);
      if (!ok) break;
      tc::fence_after_sync();
      float v[DWN];  // (columns past a narrow piece's 16 are read and not used)
      tc::tmem_ld32(tm + lane_base + uint32_t(buf * DWN), v);
#pragma unroll
      for (int q = 0; q < DWN; ++q) acc[q] += v[q];
      tc::fence_before_sync();
      if (lane == 0) tc::mbar_arrive(&s.dempty[buf]);
    }
    const int f = half * HALF + 32 * warp + lane;
    if (last) {  // W5 [16][256]: rows past the used outputs stay 0
#pragma unroll
      for (int q = 0; q < DO; ++q) a.g[w_off(DNL) + q * DH + f] = q < DO_USED ? acc[q] : 0.0f;
    } else {
      float4* o = reinterpret_cast<float4*>(a.g + w_off(l) + f * layer_in(l) + nt * DWN);
#pragma unroll
      for (int q = 0; q < DWN / 4; ++q)
        if (4 * q < ncol) o[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
    }
  }
  if (!ok && lane == 0) atomicExch(a.err, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tm, DWB * DWN);
}

// The BF16 copies of weight q: of W_l [out][in] and, past the first layer, of
// its transpose [in][out].
__device__ __forceinline__ void put_weight(int q, float x, uint16_t* wk, uint16_t* wt) {
  int l = 0;
  while (l < NLAYER - 1 && q >= w_off(l + 1)) ++l;
  const int rel = q - w_off(l);
  if (rel >= layer_out(l) * layer_in(l)) return;  // a bias
  const int o = rel / layer_in(l), i = rel % layer_in(l);
  const uint16_t b = f2bf(x);
  wk[w_off(l) + tc::kmaj_off(o, i, layer_in(l)) / 2] = b;
  if (l > 0) wt[w_off(l) + tc::kmaj_off(i, o, layer_out(l)) / 2] = b;
}
__global__ void cast_kernel(const float* __restrict__ p, uint16_t* wk, uint16_t* wt) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < NPARAM) put_weight(q, p[q], wk, wt);
}

// Adam (Kingma & Ba, 2015), the BF16 copies of the new weights, and the
// step's loss from the clusters' sums.
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                            float eps, float c1, float c2, uint16_t* wk, uint16_t* wt, const double* lpart, int nl,
                            double rows, float* loss) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  if (q < NPARAM) {
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.0f - b1) * gq;
    const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    const float x = p[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
    p[q] = x;
    put_weight(q, x, wk, wt);
  }
  if (q == 0 && loss) {
    double t = 0.0;
    for (int c = 0; c < nl; ++c) t += lpart[c];
    *loss = float(t / rows);
  }
}

struct Pcg {
  uint64_t s, inc;
  uint32_t next() {
    const uint64_t old = s;
    s = old * 6364136223846793005ULL + inc;
    const uint32_t x = uint32_t(((old >> 18u) ^ old) >> 27u), r = uint32_t(old >> 59u);
    return (x >> r) | (x << ((32 - r) & 31));
  }
  double uniform() { return (next() + 0.5) / 4294967296.0; }
};

// Minibatch row lists in pinned host memory, read from there by net_kernel
// (512 bytes a CTA, before it waits for the step before; a copy to the device
// would stand between two steps' kernels), reused in two halves.
constexpr int IDX_RING = 8, IDX_HALF = IDX_RING / 2;

}  // namespace

// The network and its work arrays (cap: the rows of one pass).
struct e2d_mlp_deep {
  int device = 0, sms = 148, cap = 0, icap = 0, hcap = 0, adam_t = 0;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  uint16_t *wk = nullptr, *wt = nullptr;       // BF16 weights and transposes (canonical tiles, param offsets)
  uint16_t* xb = nullptr;                      // [cap][16] tiles
  uint16_t* act[DNL] = {};                     // H_1..H_4, [cap][256] tiles
  uint16_t* dy = nullptr;                      // [cap][16] tiles
  uint16_t* dz[DNL] = {};                      // deltas of the hidden layers, [cap][256] tiles
  float* gp = nullptr;                         // [CTAs][4][128 x 128] GELU' of the tiles in work
  double* lpart = nullptr;                     // [clusters] loss sums
  int* hidx = nullptr;                         // [IDX_RING][icap] minibatch rows (pinned host memory)
  cudaEvent_t read[2] = {};                    // the steps that read a half of hidx are done
  float* loss = nullptr;                       // [hcap] loss history of a training call
  int* err = nullptr;
  void* ws = nullptr;                          // the work arrays' memory (rebuilt on growth)
};

namespace {

void free_ws(e2d_mlp_deep* d) {
  if (d->ws) cudaFree(d->ws);
  d->ws = nullptr;
  d->cap = 0;
}

// CTAs of net_kernel over n rows: a pair per tile, at most one per SM.
int net_grid(const e2d_mlp_deep* d, int n) {
  const int ntiles = (n + TILE - 1) / TILE, most = d->sms / 2;
  return 2 * (ntiles < most ? ntiles : most);
}

// Work arrays of a gradient over `rows` rows (whole tiles), one allocation.
int ensure_cap(e2d_mlp_deep* d, int rows) {
  if (rows <= d->cap) return 0;
  free_ws(d);
  const size_t c = (size_t(rows) + TILE - 1) / TILE * TILE, narrow = c * DF * 2, wide = c * DH * 2;
  const size_t gp = size_t(net_grid(d, rows)) * DNL * TILE * HALF * 4;
  if (cudaMalloc(&d->ws, 2 * narrow + 2 * DNL * wide + gp) != cudaSuccess) {
    cudaGetLastError();
    d->ws = nullptr;
    return E2D_ERR_NOMEM;
  }
  uint8_t* q = static_cast<uint8_t*>(d->ws);
  auto take = [&](size_t bytes) { uint8_t* p = q; q += bytes; return p; };
  d->gp = reinterpret_cast<float*>(take(gp));
  d->xb = reinterpret_cast<uint16_t*>(take(narrow));
  d->dy = reinterpret_cast<uint16_t*>(take(narrow));
  for (int l = 0; l < DNL; ++l) {
    d->act[l] = reinterpret_cast<uint16_t*>(take(wide));
    d->dz[l] = reinterpret_cast<uint16_t*>(take(wide));
  }
  d->cap = rows;
  return 0;
}

void free_train(e2d_mlp_deep* d) {
  if (d->hidx) cudaFreeHost(d->hidx);
  d->hidx = nullptr;
  for (auto& e : d->read) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (d->loss) cudaFree(d->loss);
  d->loss = nullptr;
  d->icap = d->hcap = 0;
}

// The row lists of minibatches of `batch` rows and a history of `steps` losses.
int ensure_train(e2d_mlp_deep* d, int batch, int steps) {
  if (batch <= d->icap && steps <= d->hcap) return 0;
  if (batch < d->icap) batch = d->icap;
  if (steps < d->hcap) steps = d->hcap;
  free_train(d);
  bool ok = cudaMalloc(&d->loss, sizeof(float) * size_t(steps > 0 ? steps : 1)) == cudaSuccess;
  ok = ok && cudaMallocHost(&d->hidx, sizeof(int) * size_t(batch) * IDX_RING) == cudaSuccess;
  for (int k = 0; k < 2 && ok; ++k)
    ok = cudaEventCreateWithFlags(&d->read[k], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    free_train(d);
    return E2D_ERR_NOMEM;
  }
  d->icap = batch;
  d->hcap = steps;
  return 0;
}

NetArgs net_args(const e2d_mlp_deep* d, const float* X, const float* T, const int* idx, int n, float* Y) {
  NetArgs a{};
  a.X = X; a.T = T; a.idx = idx; a.Y = Y;
  a.vec = ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(T) | reinterpret_cast<uintptr_t>(Y)) & 15) == 0;
  a.n = n;
  a.inv_n = 1.0f / float(n);
  a.wk = d->wk; a.wt = d->wt; a.p = d->p;
  a.xb = d->xb; a.dy = d->dy;
  for (int l = 0; l < DNL; ++l) { a.act[l] = d->act[l]; a.dz[l] = d->dz[l]; }
  a.gp = d->gp;
  a.lpart = d->lpart;
  a.err = d->err;
  return a;
}

// Gradient of loss = sum over rows and the used outputs of (y - t)^2 / n over
// n rows (idx, or the first n) into d->g; the loss sums into d->lpart.  The
// rows are grouped as one group per SM, so that the sums' order depends on n
// alone.
int gradient_rows(e2d_mlp_deep* d, const float* X, const float* T, const int* idx, int n, cudaStream_t st) {
  if (launch_pdl(net_kernel<true>, net_grid(d, n), NT, sizeof(NetSmem), st, net_args(d, X, T, idx, n, nullptr)) !=
      cudaSuccess)
    return E2D_ERR_CUDA;
  DwArgs w{};
  w.xb = d->xb; w.dy = d->dy;
  for (int l = 0; l < DNL; ++l) { w.act[l] = d->act[l]; w.dz[l] = d->dz[l]; }
  w.n = n;
  w.brows = (n + d->sms - 1) / d->sms;
  w.rows = (w.brows + RC - 1) / RC * RC;
  w.g = d->g;
  w.err = d->err;
  return launch_pdl(dw_kernel, DW_ITEMS + DW_BIAS, DW_THREADS, sizeof(DwSmem), st, w) == cudaSuccess ? 0
                                                                                                      : E2D_ERR_CUDA;
}

int check_err(e2d_mlp_deep* d, cudaStream_t st) {
  int e = 0;
  if (cudaMemcpyAsync(&e, d->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return E2D_ERR_CUDA;
  return e ? E2D_ERR_CUDA : 0;
}

int refresh(e2d_mlp_deep* d, cudaStream_t st) {
  cast_kernel<<<(NPARAM + 255) / 256, 256, 0, st>>>(d->p, d->wk, d->wt);
  return cudaGetLastError() == cudaSuccess ? 0 : E2D_ERR_CUDA;
}

}  // namespace

extern "C" {

e2d_mlp_deep* e2d_mlp_deep_create(uint64_t seed, int* err) {
  if (err) *err = 0;
  e2d_mlp_deep* d = new e2d_mlp_deep;
  cudaGetDevice(&d->device);
  cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, d->device);
  bool ok = cudaMalloc(&d->p, 4 * size_t(NPARAM)) == cudaSuccess && cudaMalloc(&d->g, 4 * size_t(NPARAM)) == cudaSuccess &&
            cudaMalloc(&d->m, 4 * size_t(NPARAM)) == cudaSuccess && cudaMalloc(&d->v, 4 * size_t(NPARAM)) == cudaSuccess &&
            cudaMalloc(&d->wk, 2 * size_t(NPARAM)) == cudaSuccess && cudaMalloc(&d->wt, 2 * size_t(NPARAM)) == cudaSuccess &&
            cudaMalloc(&d->lpart, sizeof(double) * d->sms) == cudaSuccess &&
            cudaMalloc(&d->err, sizeof(int)) == cudaSuccess;
  if (ok && (cudaFuncSetAttribute(net_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(NetSmem))) ||
             cudaFuncSetAttribute(net_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(NetSmem))) ||
             cudaFuncSetAttribute(dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(DwSmem))))) {
    if (err) *err = E2D_ERR_CUDA;
    e2d_mlp_deep_destroy(d);
    return nullptr;
  }
  if (!ok) {
    if (err) *err = E2D_ERR_NOMEM;
    e2d_mlp_deep_destroy(d);
    return nullptr;
  }
  // Glorot-uniform weights, zero biases
  std::vector<float> h(NPARAM, 0.0f);
  Pcg rng{seed * 2 + 1, (seed << 1) | 1};
  for (int l = 0; l < NLAYER; ++l) {
    const int fan_in = l == 0 ? 5 : layer_in(l), fan_out = l == DNL ? DO_USED : layer_out(l);
    const double a = std::sqrt(6.0 / double(fan_in + fan_out));
    for (int o = 0; o < layer_out(l); ++o)
      for (int i = 0; i < layer_in(l); ++i) {
        const double u = (2.0 * rng.uniform() - 1.0) * a;
        // inputs past the 5 features and outputs past the 4 used ones start at zero
        const bool live = (l > 0 || i < 5) && (l < DNL || o < DO_USED);
        h[w_off(l) + o * layer_in(l) + i] = live ? float(u) : 0.0f;
      }
  }
  if (cudaMemcpy(d->p, h.data(), 4 * size_t(NPARAM), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(d->m, 0, 4 * size_t(NPARAM)) != cudaSuccess || cudaMemset(d->v, 0, 4 * size_t(NPARAM)) != cudaSuccess ||
      cudaMemset(d->g, 0, 4 * size_t(NPARAM)) != cudaSuccess || cudaMemset(d->wk, 0, 2 * size_t(NPARAM)) != cudaSuccess ||
      cudaMemset(d->wt, 0, 2 * size_t(NPARAM)) != cudaSuccess ||
      cudaMemset(d->err, 0, sizeof(int)) != cudaSuccess || refresh(d, 0) || cudaDeviceSynchronize() != cudaSuccess) {
    if (err) *err = E2D_ERR_CUDA;
    e2d_mlp_deep_destroy(d);
    return nullptr;
  }
  return d;
}

void e2d_mlp_deep_destroy(e2d_mlp_deep* d) {
  if (!d) return;
  free_ws(d);
  free_train(d);
  for (void* q : {(void*)d->p, (void*)d->g, (void*)d->m, (void*)d->v, (void*)d->wk, (void*)d->wt, (void*)d->lpart,
                  (void*)d->err})
    if (q) cudaFree(q);
  delete d;
}

int e2d_mlp_deep_nparams(void) { return NPARAM; }

int e2d_mlp_deep_params(e2d_mlp_deep* d, float* out, const float* in) {
  if (!d) return E2D_ERR_ARG;
  if (in) {
    if (cudaMemcpy(d->p, in, 4 * size_t(NPARAM), cudaMemcpyHostToDevice) != cudaSuccess) return E2D_ERR_CUDA;
    if (refresh(d, 0) || cudaDeviceSynchronize() != cudaSuccess) return E2D_ERR_CUDA;
  }
  if (out && cudaMemcpy(out, d->p, 4 * size_t(NPARAM), cudaMemcpyDeviceToHost) != cudaSuccess) return E2D_ERR_CUDA;
  return 0;
}

int e2d_mlp_deep_forward(e2d_mlp_deep* d, const float* X, int n, float* Y, void* stream) {
  if (!d || !X || !Y || n < 1) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  net_kernel<false><<<net_grid(d, n), NT, sizeof(NetSmem), st>>>(net_args(d, X, nullptr, nullptr, n, Y));
  if (cudaGetLastError() != cudaSuccess) return E2D_ERR_CUDA;
  return check_err(d, st);
}

int e2d_mlp_deep_gradient(e2d_mlp_deep* d, const float* X, const float* T, int n, float* grad, double* loss,
                          void* stream) {
  if (!d || !X || !T || n < 1) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc;
  if ((rc = ensure_cap(d, n)) || (rc = gradient_rows(d, X, T, nullptr, n, st))) return rc;
  const int nl = net_grid(d, n) / 2;
  std::vector<double> lp(nl);
  if (cudaMemcpyAsync(lp.data(), d->lpart, sizeof(double) * nl, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return E2D_ERR_CUDA;
  if ((rc = check_err(d, st))) return rc;
  if (grad && cudaMemcpy(grad, d->g, 4 * size_t(NPARAM), cudaMemcpyDeviceToHost) != cudaSuccess) return E2D_ERR_CUDA;
  double l = 0.0;
  for (double x : lp) l += x;
  if (loss) *loss = l / double(n);
  return 0;
}

// Three launches a step and no wait for the device: the host draws the next
// minibatches' rows (through a ring of pinned lists) while the device works,
// and reads the losses once at the end.
int e2d_mlp_deep_train(e2d_mlp_deep* d, const float* X, const float* T, int n, int steps, int batch, float lr,
                       uint64_t seed, float* loss_hist, void* stream) {
  if (!d || !X || !T || n < 1 || steps < 0 || batch < 1 || !(lr > 0.0f)) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int b = batch < n ? batch : n;
  int rc;
  if ((rc = ensure_cap(d, b)) || (rc = ensure_train(d, b, steps))) return rc;
  Pcg rng{seed * 2 + 1, (seed << 1) | 1};
  std::vector<int> perm(n);
  for (int q = 0; q < n; ++q) perm[q] = q;
  int pos = n;  // reshuffle at the first step
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const int nl = net_grid(d, b) / 2;
  for (int k = 0; k < steps; ++k) {
    const int slot = k % IDX_RING, half = slot / IDX_HALF;
    // the half's last readers are done (an earlier call's included)
    if (slot % IDX_HALF == 0 && cudaEventSynchronize(d->read[half]) != cudaSuccess) return E2D_ERR_CUDA;
    int* hidx = d->hidx + size_t(slot) * d->icap;
    for (int q = 0; q < b;) {
      if (pos >= n) {  // Fisher-Yates shuffle of the rows per epoch
        for (int i = n - 1; i > 0; --i) std::swap(perm[i], perm[int(rng.next() % uint32_t(i + 1))]);
        pos = 0;
      }
      const int take = b - q < n - pos ? b - q : n - pos;
      std::copy(perm.begin() + pos, perm.begin() + pos + take, hidx + q);
      q += take;
      pos += take;
    }
    if ((rc = gradient_rows(d, X, T, hidx, b, st))) return rc;
    ++d->adam_t;
    const float c1 = 1.0f - powf(b1, float(d->adam_t)), c2 = 1.0f - powf(b2, float(d->adam_t));
    if (launch_pdl(adam_kernel, (NPARAM + 255) / 256, 256, 0, st, d->p, d->g, d->m, d->v, lr, b1, b2, eps, c1, c2, d->wk,
                   d->wt, d->lpart, nl, double(b), loss_hist ? d->loss + k : nullptr) != cudaSuccess ||
        ((slot % IDX_HALF == IDX_HALF - 1 || k == steps - 1) && cudaEventRecord(d->read[half], st) != cudaSuccess))
      return E2D_ERR_CUDA;
  }
  if (loss_hist && steps > 0 &&
      cudaMemcpyAsync(loss_hist, d->loss, sizeof(float) * size_t(steps), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return E2D_ERR_CUDA;
  return check_err(d, st);
}

}  // extern "C"
