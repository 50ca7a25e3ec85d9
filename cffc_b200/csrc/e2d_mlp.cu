// e2d_mlp.cu — the learned warm start's network on the tensor cores: a
// per-cell MLP (16 input features -> 128 -> 128 -> 16 outputs, tanh hidden
// layers) whose forward pass (inference) and forward + backward pass
// (training) are hand-written tcgen05 kernels: BF16 operands resident in
// shared memory, FP32 accumulators in TMEM, one persistent CTA over tiles of
// 128 cells, every matrix product an M = 128 UMMA.
//
// Training products per tile (cells c, hidden h, outputs o, features f):
//   forward   D1 = X W1^T, H1 = tanh(D1 + b1); D2 = H1 W2^T, H2 = tanh(..);
//             Y = H2 W3^T + b3
//   backward  dY = 2 (Y - T) / n  (the four used outputs)
//             dH2 = dY W3           (M = c)     dW3^T = H2^T dY  (M = h, K = c)
//             dZ2 = dH2 (1 - H2^2)
//             dH1 = dZ2 W2          (M = c)     dW2 = dZ2^T H1   (M = o, K = c)
//             dZ1 = dH1 (1 - H1^2);             dW1 = dZ1^T X    (M = h, K = c)
// Each CTA accumulates its tiles' weight gradients in TMEM (FP32) and
// writes them to its own slot; the slots are summed in CTA order, so
// training is deterministic.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/cffc_e2d.h"
#include <cuda_bf16.h>

#include "e2d_tc.cuh"

using namespace e2d;

namespace {

constexpr uint32_t WAIT_ITERS = 1u << 22;  // bounded mbarrier waits (about a second)

// ---------------------------------------------------------------------------
// Self-test of the building blocks: D[128 x N] = A[128 x K] B[N x K]^T.
__global__ void __launch_bounds__(128) tc_selftest_kernel(const uint16_t* A, const uint16_t* Bm, float* D, int N,
                                                          int K, uint32_t ncols, int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t taddr;
  uint8_t* As = sm;
  uint8_t* Bs = sm + 128 * K * 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int idx = tid; idx < 128 * K; idx += 128)
    *reinterpret_cast<uint16_t*>(As + tc::kmaj_off(idx / K, idx % K, K)) = A[idx];
  for (int idx = tid; idx < N * K; idx += 128)
    *reinterpret_cast<uint16_t*>(Bs + tc::kmaj_off(idx / K, idx % K, K)) = Bm[idx];
  if (tid == 0) tc::mbar_init(&bar, 1);
  if (warp == 0) tc::tmem_alloc(&taddr, ncols);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t t0 = taddr;
  if (tid == 0) {
    const uint32_t id = tc::idesc_bf16(128, N);
    for (int t = 0; t < K / 16; ++t)
      tc::mma_bf16(t0, tc::smem_desc(tc::smem_addr(As) + 256 * t, 128, K * 16),
                   tc::smem_desc(tc::smem_addr(Bs) + 256 * t, 128, K * 16), id, t > 0);
    tc::mma_commit(&bar);
  }
  __syncwarp();
  // warp-uniform outcome: the TMEM loads below are .sync.aligned
  const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&bar, 0, WAIT_ITERS));
  tc::fence_after_sync();
  if (!ok) {
    if (lane == 0) atomicExch(err, 1);
  } else {
    const int row = 32 * warp + lane;
    for (int col = 0; col < N; col += 16) {
      float v[16];
      tc::tmem_ld16(t0 + (uint32_t(32 * warp) << 16) + uint32_t(col), v);
#pragma unroll
      for (int q = 0; q < 16; ++q) D[size_t(row) * N + col + q] = v[q];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(t0, ncols);
}

}  // namespace

extern "C" int e2d_tc_selftest(const uint16_t* A, const uint16_t* B, float* D, int N, int K) {
  if (!A || !B || !D || N < 16 || N > 256 || N % 16 || K < 16 || K > 128 || K % 16) return E2D_ERR_ARG;
  uint16_t *dA = nullptr, *dB = nullptr;
  float* dD = nullptr;
  int* derr = nullptr;
  int rc = 0;
  const size_t smem = size_t(128) * K * 2 + size_t(N) * K * 2;
  uint32_t ncols = 32;
  while (ncols < uint32_t(N)) ncols <<= 1;
  if (cudaMalloc(&dA, 2 * 128 * K) || cudaMalloc(&dB, 2 * size_t(N) * K) || cudaMalloc(&dD, 4 * 128 * size_t(N)) ||
      cudaMalloc(&derr, sizeof(int))) {
    rc = E2D_ERR_NOMEM;
  } else if (cudaMemcpy(dA, A, 2 * 128 * K, cudaMemcpyHostToDevice) ||
             cudaMemcpy(dB, B, 2 * size_t(N) * K, cudaMemcpyHostToDevice) || cudaMemset(derr, 0, sizeof(int)) ||
             cudaFuncSetAttribute(tc_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))) {
    rc = E2D_ERR_CUDA;
  } else {
    tc_selftest_kernel<<<1, 128, smem>>>(dA, dB, dD, N, K, ncols, derr);
    int herr = 0;
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost) ||
        cudaMemcpy(D, dD, 4 * 128 * size_t(N), cudaMemcpyDeviceToHost))
      rc = E2D_ERR_CUDA;
    else if (herr)
      rc = E2D_ERR_CUDA;
  }
  cudaFree(dA); cudaFree(dB); cudaFree(dD); cudaFree(derr);
  return rc;
}

// ===========================================================================
// The warm-start network.
namespace {

constexpr int MF = 16;    // input features
constexpr int MH = 128;   // hidden units (both layers)
constexpr int MO = 16;    // outputs computed (the first MO_USED are trained)
constexpr int MO_USED = 4;
constexpr int TILE = 128; // cells per tile (the UMMA M)
constexpr int NPARAM = MH * MF + MH + MH * MH + MH + MO * MH + MO;
// offsets of the flat parameter vector
constexpr int P_W1 = 0, P_B1 = P_W1 + MH * MF, P_W2 = P_B1 + MH, P_B2 = P_W2 + MH * MH, P_W3 = P_B2 + MH,
              P_B3 = P_W3 + MO * MH;

// BF16 copies of the weights, row-major: W1 [MH][MF], W2 [MH][MH], W3 [MO][MH].
struct MlpDev {
  const uint16_t *w1, *w2, *w3;
  const float* p;  // FP32 parameters (biases read from here)
};

constexpr int EPI = 512;        // epilogue threads: 4 warps per 32 TMEM lanes, 32 columns a warp
constexpr int NT = EPI + 32;    // and the warp that issues the products
constexpr int CHUNK = TILE * 16;  // bytes of 8 columns of a 128-row tile

// Shared memory (bytes): column-chunk tiles (e2d_tc.cuh), each read K-major
// by one product and MN-major by another.
template <bool TRAIN>
struct MlpSmem {
  uint8_t W2[MH * MH * 2];          // [MH][MH]     B of F2, of dH1
  uint8_t H1[TILE * MH * 2];        // [cells][MH]  A of F2, B of dW2 (inference: then H2)
  uint8_t H2[TRAIN ? TILE * MH * 2 : 16];   // [cells][MH]  A of F3, of dW3^T; then dZ1, A of dW1
  uint8_t dZ2[TRAIN ? TILE * MH * 2 : 16];  // [cells][MH]  A of dH1, of dW2
  uint8_t dY[TRAIN ? TILE * MO * 2 : 16];   // [cells][MO]  A of dH2, B of dW3^T
  uint8_t X[2][TILE * MF * 2];      // [cells][MF]  A of F1, B of dW1; the next tile's beside
  uint8_t W1[MH * MF * 2];          // [MH][MF]     B of F1
  uint8_t W3[MO * MH * 2];          // [MO][MH]     B of F3, of dH2
  float b1[MH], b2[MH], b3[MO];
  float gb1[4][MH], gb2[4][MH], gb3[4][MO];  // bias gradients of each 32 rows (train)
  double lw[4];                              // their loss sums
  uint64_t bar;
  uint32_t taddr;
};

__device__ __forceinline__ uint16_t f2bf(float x) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) { return uint32_t(f2bf(a)) | (uint32_t(f2bf(b)) << 16); }
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Global BF16 [rows][K] row-major -> shared column-chunk tile.
__device__ void stage_tile(uint8_t* dst, const uint16_t* src, int rows, int K) {
  for (int q = threadIdx.x; q < rows * (K / 8); q += NT)
    *reinterpret_cast<uint4*>(dst + 16 * q) = *reinterpret_cast<const uint4*>(src + (q % rows) * K + 8 * (q / rows));
}

// A tile as an operand: its descriptor walk over 16 values of the contraction.
struct Operand {
  uint32_t base, lbo, sbo, step;
};
// contraction over the columns of a tile of `rows` rows
__device__ __forceinline__ Operand kmaj(const uint8_t* t, int rows) {
  return {tc::smem_addr(t), uint32_t(rows * 16), 128u, uint32_t(rows * 32)};
}
// contraction over its rows
__device__ __forceinline__ Operand mnmaj(const uint8_t* t, int rows) {
  return {tc::smem_addr(t), 128u, uint32_t(rows * 16), 256u};
}
// D[128][N] (+)= A B^T over K (a multiple of 16), one thread.
__device__ __forceinline__ void product(uint32_t d, Operand a, Operand b, uint32_t id, int K, bool acc) {
  for (int t = 0; t < K / 16; ++t)
    tc::mma_bf16(d, tc::smem_desc(a.base + a.step * t, a.lbo, a.sbo), tc::smem_desc(b.base + b.step * t, b.lbo, b.sbo),
                 id, (acc || t > 0) ? 1u : 0u);
}

// Every generic shared-memory write and TMEM read before, every product
// after; false for all as soon as one wait has run out.
__device__ __forceinline__ bool cta_sync_async(bool ok) {
  tc::fence_async_smem();
  tc::fence_before_sync();
  ok = __syncthreads_and(ok) != 0;
  tc::fence_after_sync();
  return ok;
}

__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Column sums over the warp's 32 rows of 16 columns, in warp_sum's order:
// each exchange halves the columns a lane carries; column (lane >> 1) ends in
// lanes 2 c and 2 c + 1.  16 shuffles where a sum per column takes 80.
__device__ __forceinline__ float column_sums16(float* v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = 8; n >= 1; n >>= 1) {  // lanes 2 n apart
    const bool up = lane & (2 * n);
#pragma unroll
    for (int q = 0; q < n; ++q) {
      const float keep = up ? v[q + n] : v[q], give = up ? v[q] : v[q + n];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// TMEM columns: D1, D3 and dH2 share [0,128) (each is read out before the
// next is written), D2 / dH1 [128,256); training accumulators dW3^T
// [256,272), dW1 [272,288), dW2 [384,512).  Inference allocates 256 columns,
// training 512.
constexpr uint32_t C_D1 = 0, C_D2 = 128, C_D3 = 0, C_GW3 = 256, C_GW1 = 272, C_GW2 = 384;

// h = tanh(d + b) of 32 columns of this thread's row, to the tile and packed.
__device__ __forceinline__ void activate(uint32_t taddr, const float* bias, uint8_t* dst, uint32_t* h) {
#pragma unroll
  for (int c0 = 0; c0 < 32; c0 += 16) {
    float v[16];
    tc::tmem_ld16(taddr + c0, v);
#pragma unroll
    for (int q = 0; q < 16; q += 2)
      h[(c0 + q) / 2] = pack2(tanhf(v[q] + bias[c0 + q]), tanhf(v[q + 1] + bias[c0 + q + 1]));
#pragma unroll
    for (int q = 0; q < 16; q += 8) {
      const uint32_t* w = h + (c0 + q) / 2;
      *reinterpret_cast<uint4*>(dst + (c0 + q) / 8 * CHUNK) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// dz = d (1 - h^2) of 32 columns of this thread's row, to the tile; the
// columns' sums over the warp's rows are added to gb (column_sums16's lanes).
__device__ __forceinline__ void deltas(uint32_t taddr, const uint32_t* h, bool valid, uint8_t* dst, float* gb) {
#pragma unroll
  for (int c0 = 0; c0 < 32; c0 += 16) {
    float v[16];
    tc::tmem_ld16(taddr + c0, v);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const uint32_t w = h[(c0 + q) / 2];
      const float a = (q & 1) ? bf_hi(w) : bf_lo(w);
      v[q] = valid ? v[q] * (1.0f - a * a) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 16; q += 8)
      *reinterpret_cast<uint4*>(dst + (c0 + q) / 8 * CHUNK) =
          make_uint4(pack2(v[q], v[q + 1]), pack2(v[q + 2], v[q + 3]), pack2(v[q + 4], v[q + 5]), pack2(v[q + 6], v[q + 7]));
    gb[c0 / 16] += column_sums16(v);
  }
}

// Persistent kernel over tiles of 128 cells.  TRAIN = false: Y = f(X) for the
// rows of the tiles.  TRAIN = true: the gradient of
// loss = sum over rows and the four outputs of (y - t)^2 / n_total,
// accumulated in TMEM over the CTA's tiles and written to the CTA's slot of
// grad (and of loss).
//
// Bound by the epilogues (two tanhf per hidden unit and cell, about 35
// instructions each) and the chain product -> commit -> epilogue -> barrier,
// six products deep.  So: 16 warps share a tile's epilogue (a thread has 32
// columns of one row), 16-byte stores, the weights stay in shared memory, the
// transposed operands are the same tiles read MN-major, the weight-gradient
// products are issued by a warp of their own behind the product that the
// epilogue waits for, and the next tile's X is loaded and its first product
// issued before this tile's last.  Measured (B200) against 128 threads a tile
// with 2-byte staging, transposed copies of every operand and a shuffle sum
// per column: a training step over 151,552 rows 580 -> 94 us (1,184 tiles, eight
// a CTA), and the same gradients bit for bit.
// vec: X, T and Y are 16-byte aligned.
template <bool TRAIN>
__global__ void __launch_bounds__(NT, TRAIN ? 1 : 2) mlp_kernel(MlpDev w, const float* __restrict__ X,
                                                                const float* __restrict__ T, int n, float inv_n,
                                                                float* __restrict__ Y, float* grad, double* loss,
                                                                int vec, int* err) {
  extern __shared__ __align__(1024) uint8_t smraw[];
  MlpSmem<TRAIN>& s = *reinterpret_cast<MlpSmem<TRAIN>*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool epi = tid < EPI;
  const int quad = warp & 3, cg = warp >> 2;  // 32 rows (TMEM lanes) and 32 columns of an epilogue warp
  const int r = 32 * quad + lane;             // this thread's row of the tile
  const uint32_t ncols = TRAIN ? 512u : 256u;
  const int ntiles = (n + TILE - 1) / TILE;
  auto ld4 = [&](const float* p) {
    return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
  };
  // four features of a row of the tile per thread
  auto load_x = [&](int tile) {
    const int row = tile * TILE + (tid >> 2);
    return epi && tile < ntiles && row < n ? ld4(X + size_t(row) * MF + 4 * (tid & 3)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto stage_x = [&](uint8_t* dst, const float4& x) {
    const int row = tid >> 2, part = tid & 3;
    if (epi)
      *reinterpret_cast<uint2*>(dst + (part >> 1) * CHUNK + row * 16 + (part & 1) * 8) =
          make_uint2(pack2(x.x, x.y), pack2(x.z, x.w));
  };
  // constant operands and the first tile
  const float4 x0 = load_x(blockIdx.x);
  stage_tile(s.W1, w.w1, MH, MF);
  stage_tile(s.W2, w.w2, MH, MH);
  stage_tile(s.W3, w.w3, MO, MH);
  stage_x(s.X[0], x0);
  if (TRAIN && epi && cg == 1)  // the unused outputs' deltas stay zero
    *reinterpret_cast<uint4*>(s.dY + CHUNK + r * 16) = make_uint4(0u, 0u, 0u, 0u);
  for (int k = tid; k < MH; k += NT) {
    s.b1[k] = w.p[P_B1 + k];
    s.b2[k] = w.p[P_B2 + k];
  }
  if (tid < MO) s.b3[tid] = w.p[P_B3 + tid];
  if (tid == 0) tc::mbar_init(&s.bar, 1);
  if (warp == 0) tc::tmem_alloc(&s.taddr, ncols);
  bool ok = cta_sync_async(true);
  const uint32_t tm = s.taddr;
  const uint32_t tw = tm + (uint32_t(32 * quad) << 16) + 32 * cg;  // this warp's lanes and columns
  const bool issuer = tid == EPI;
  uint8_t* const h2 = TRAIN ? s.H2 : s.H1;
  uint8_t* const row_h1 = s.H1 + 4 * cg * CHUNK + r * 16;  // this thread's row and columns of a tile
  uint8_t* const row_h2 = h2 + 4 * cg * CHUNK + r * 16;
  uint8_t* const row_dz2 = (TRAIN ? s.dZ2 : s.H1) + 4 * cg * CHUNK + r * 16;
  constexpr uint32_t ID = tc::idesc_bf16(128, MH), ID_O = tc::idesc_bf16(128, MO);
  constexpr uint32_t ID_BT = tc::idesc_bf16(128, MH) | (1u << 16);  // B MN-major
  constexpr uint32_t ID_T = tc::idesc_bf16_t(128, MH), ID_OT = tc::idesc_bf16_t(128, MO);
  uint32_t phase = 0;
  auto wait = [&]() {
    if (epi && ok) ok = tc::mbar_wait_warp(&s.bar, phase, WAIT_ITERS);
    phase ^= 1u;
    tc::fence_after_sync();
  };
  if (issuer) {
    product(tm + C_D1, kmaj(s.X[0], TILE), kmaj(s.W1, MH), ID, MF, false);
    tc::mma_commit(&s.bar);
  }
  double lsum = 0.0;
  float gb1[2] = {0.0f, 0.0f}, gb2[2] = {0.0f, 0.0f}, gb3[MO_USED] = {0.0f, 0.0f, 0.0f, 0.0f};
  int it = 0;
  for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
    const int row = tile * TILE + r;
    const bool valid = row < n, more = tile + int(gridDim.x) < ntiles;
    const float4 xn = load_x(tile + gridDim.x);
    float4 t4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (TRAIN && epi && cg == 0 && valid) t4 = ld4(T + size_t(row) * MO_USED);
    uint32_t p1[16], p2[16];  // H1, H2 of this thread's row and columns
    // ---- F1 (issued with the tile before): H1 = tanh(X W1^T + b1) ----------
    wait();
    if (epi) activate(tw + C_D1, s.b1 + 32 * cg, row_h1, p1);
    ok = cta_sync_async(ok);
    // ---- F2: H2 = tanh(H1 W2^T + b2) ---------------------------------------
    if (issuer && ok) {
      product(tm + C_D2, kmaj(s.H1, TILE), kmaj(s.W2, MH), ID, MH, false);
      tc::mma_commit(&s.bar);
    }
    wait();
    if (epi) activate(tw + C_D2, s.b2 + 32 * cg, row_h2, p2);
    if (!TRAIN) stage_x(s.X[(it + 1) & 1], xn);
    ok = cta_sync_async(ok);
    // ---- F3: Y = H2 W3^T + b3 ----------------------------------------------
    if (issuer && ok) {
      product(tm + C_D3, kmaj(h2, TILE), kmaj(s.W3, MO), ID_O, MH, false);
      tc::mma_commit(&s.bar);
    }
    wait();
    if (epi && cg == 0) {
      float y[16];
      tc::tmem_ld16(tw + C_D3, y);
#pragma unroll
      for (int q = 0; q < MO_USED; ++q) y[q] += s.b3[q];
      if (!TRAIN) {
        if (valid) {
          float* yr = Y + size_t(row) * MO_USED;
          if (vec) *reinterpret_cast<float4*>(yr) = make_float4(y[0], y[1], y[2], y[3]);
          else { yr[0] = y[0]; yr[1] = y[1]; yr[2] = y[2]; yr[3] = y[3]; }
        }
      } else {
        // dY, loss, b3 gradient
        const float tq[MO_USED] = {t4.x, t4.y, t4.z, t4.w};
        float dy[MO_USED];
#pragma unroll
        for (int q = 0; q < MO_USED; ++q) {
          dy[q] = 0.0f;
          if (valid) {
            const float e = y[q] - tq[q];
            lsum += double(e) * double(e);
            dy[q] = 2.0f * e * inv_n;
          }
          gb3[q] += warp_sum(dy[q]);
        }
        *reinterpret_cast<uint4*>(s.dY + r * 16) = make_uint4(pack2(dy[0], dy[1]), pack2(dy[2], dy[3]), 0u, 0u);
      }
    }
    ok = cta_sync_async(ok);
    if (!TRAIN) {
      if (issuer && ok && more) {
        product(tm + C_D1, kmaj(s.X[(it + 1) & 1], TILE), kmaj(s.W1, MH), ID, MF, false);
        tc::mma_commit(&s.bar);
      }
      continue;
    }
    // ---- B1: dH2 = dY W3; dW3^T += H2^T dY ---------------------------------
    if (issuer && ok) {
      product(tm + C_D1, kmaj(s.dY, TILE), mnmaj(s.W3, MO), ID_BT, MO, false);
      tc::mma_commit(&s.bar);
      product(tm + C_GW3, mnmaj(s.H2, TILE), mnmaj(s.dY, TILE), ID_OT, TILE, it > 0);
    }
    wait();
    if (epi) deltas(tw + C_D1, p2, valid, row_dz2, gb2);
    ok = cta_sync_async(ok);
    // ---- B2: dH1 = dZ2 W2; dW2 += dZ2^T H1 ---------------------------------
    if (issuer && ok) {
      product(tm + C_D2, kmaj(s.dZ2, TILE), mnmaj(s.W2, MH), ID_BT, MH, false);
      tc::mma_commit(&s.bar);
      product(tm + C_GW2, mnmaj(s.dZ2, TILE), mnmaj(s.H1, TILE), ID_T, TILE, it > 0);
    }
    wait();  // dW3^T is done as well: dZ1 goes where H2 was
    if (epi) deltas(tw + C_D2, p1, valid, row_h2, gb1);
    stage_x(s.X[(it + 1) & 1], xn);
    ok = cta_sync_async(ok);
    // ---- the next tile's F1; B3: dW1 += dZ1^T X -----------------------------
    if (issuer && ok) {
      if (more) {
        product(tm + C_D1, kmaj(s.X[(it + 1) & 1], TILE), kmaj(s.W1, MH), ID, MF, false);
        tc::mma_commit(&s.bar);
      }
      product(tm + C_GW1, mnmaj(s.H2, TILE), mnmaj(s.X[it & 1], TILE), ID_OT, TILE, it > 0);
    }
  }
  if (TRAIN) {  // the last weight-gradient products
    if (issuer) tc::mma_commit(&s.bar);
    wait();
    if (epi) {
      // a column's sum stands in two lanes: both write the same value
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        s.gb1[quad][32 * cg + 16 * k + (lane >> 1)] = gb1[k];
        s.gb2[quad][32 * cg + 16 * k + (lane >> 1)] = gb2[k];
      }
      if (cg == 0 && lane < MO_USED) s.gb3[quad][lane] = lane == 0 ? gb3[0] : lane == 1 ? gb3[1] : lane == 2 ? gb3[2] : gb3[3];
      double sum = lsum;
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (cg == 0 && lane == 0) s.lw[quad] = sum;
    }
    ok = cta_sync_async(ok);
    if (ok && epi) {
      // the CTA's accumulated gradients into its own slot of grad (summed
      // over the CTAs in CTA order by mlp_step_kernel: training is
      // deterministic); TMEM lane = output row
      float* gs = grad + size_t(blockIdx.x) * NPARAM;
      float v[16];
      if (cg == 0) {  // dW3^T: row h, columns o
        tc::tmem_ld16(tw + C_GW3, v);
#pragma unroll
        for (int q = 0; q < MO; ++q) gs[P_W3 + q * MH + r] = q < MO_USED ? v[q] : 0.0f;
      } else if (cg == 1) {  // dW1: row h, columns f
        tc::tmem_ld16(tw - 32 + C_GW1, v);
#pragma unroll
        for (int q = 0; q < MF; q += 4)
          *reinterpret_cast<float4*>(gs + P_W1 + r * MF + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
      }
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 16) {  // dW2: row o, columns h
        tc::tmem_ld16(tw + C_GW2 + c0, v);
#pragma unroll
        for (int q = 0; q < 16; q += 4)
          *reinterpret_cast<float4*>(gs + P_W2 + r * MH + 32 * cg + c0 + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
      }
      if (tid < MH) {
        gs[P_B1 + tid] = ((s.gb1[0][tid] + s.gb1[1][tid]) + s.gb1[2][tid]) + s.gb1[3][tid];
        gs[P_B2 + tid] = ((s.gb2[0][tid] + s.gb2[1][tid]) + s.gb2[2][tid]) + s.gb2[3][tid];
        if (tid < MO)
          gs[P_B3 + tid] = tid < MO_USED ? ((s.gb3[0][tid] + s.gb3[1][tid]) + s.gb3[2][tid]) + s.gb3[3][tid] : 0.0f;
        if (tid == 0) loss[blockIdx.x] = ((s.lw[0] + s.lw[1]) + s.lw[2]) + s.lw[3];
      }
    }
  }
  if (!ok && tid == 0) atomicExch(err, 1);
  if (!ok) {  // products still in flight end before their operands' memory goes
    if (issuer) tc::mma_commit(&s.bar);
    if (warp == 0) tc::mbar_wait_warp(&s.bar, phase, WAIT_ITERS);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tm, ncols);
}
static_assert(NPARAM % 4 == 0 && P_W1 % 4 == 0 && P_W2 % 4 == 0 && MF % 4 == 0, "16-byte gradient stores");

// The BF16 copy of parameter q.
__device__ __forceinline__ void put_weight(int q, float x, uint16_t* w1, uint16_t* w2, uint16_t* w3) {
  if (q < P_B1) w1[q] = f2bf(x);
  else if (q >= P_W2 && q < P_B2) w2[q - P_W2] = f2bf(x);
  else if (q >= P_W3 && q < P_B3) w3[q - P_W3] = f2bf(x);
}
__global__ void mlp_cast_kernel(const float* __restrict__ p, uint16_t* w1, uint16_t* w2, uint16_t* w3) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < NPARAM) put_weight(q, p[q], w1, w2, w3);
}

struct AdamArgs {
  float *p, *m, *v;
  uint16_t *w1, *w2, *w3;
  float lr, b1, b2, eps, c1, c2;
  double rows;
  float* hist;  // the step's mean loss (null: not kept)
};

// grad[q] = sum over the CTAs' slots in CTA order, 16 loads in flight (12 MB
// from L2 for 148 slots); the loss likewise.  ADAM: then the update (Kingma &
// Ba, 2015: m = b1 m + (1-b1) g; v = b2 v + (1-b2) g^2;
// p -= lr * (m / (1-b1^t)) / (sqrt(v / (1-b2^t)) + eps)) and the BF16 copies,
// unless an earlier kernel's wait has run out.
constexpr int STEP_NT = 64;
template <bool ADAM>
__global__ void __launch_bounds__(STEP_NT) mlp_step_kernel(const float* __restrict__ parts, int nparts,
                                                           float* __restrict__ grad,
                                                           const double* __restrict__ lparts, double* loss,
                                                           const int* err, AdamArgs a) {
  if (ADAM && *(const volatile int*)err) return;
  if (blockIdx.x == gridDim.x - 1) {
    if (threadIdx.x == 0) {
      double t = 0.0;
#pragma unroll 16
      for (int c = 0; c < nparts; ++c) t += lparts[c];
      *loss = t;
      if (ADAM && a.hist) *a.hist = float(t / a.rows);
    }
    return;
  }
  const int q = blockIdx.x * STEP_NT + threadIdx.x;
  if (q >= NPARAM) return;
  float t = 0.0f;
#pragma unroll 16
  for (int c = 0; c < nparts; ++c) t += parts[size_t(c) * NPARAM + q];
  grad[q] = t;
  if (ADAM) {
    const float gq = t;
    const float mq = a.b1 * a.m[q] + (1.0f - a.b1) * gq;
    const float vq = a.b2 * a.v[q] + (1.0f - a.b2) * gq * gq;
    a.m[q] = mq;
    a.v[q] = vq;
    const float x = a.p[q] - a.lr * (mq / a.c1) / (sqrtf(vq / a.c2) + a.eps);
    a.p[q] = x;
    put_weight(q, x, a.w1, a.w2, a.w3);
  }
}
constexpr int STEP_GRID = (NPARAM + STEP_NT - 1) / STEP_NT + 1;  // and the loss

}  // namespace

struct e2d_mlp {
  int device = 0;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  float* gpart = nullptr;     // [sms][NPARAM] per-CTA gradient slots
  double* lpart = nullptr;    // [sms] per-CTA loss sums
  uint16_t *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
  double* loss = nullptr;
  float* hist = nullptr;      // [hist_cap] mean losses of a training run
  int hist_cap = 0;
  int* err = nullptr;
  int adam_t = 0;
  int sms = 148;
};

namespace {

int mlp_refresh(e2d_mlp* mm, cudaStream_t st) {
  mlp_cast_kernel<<<(NPARAM + 255) / 256, 256, 0, st>>>(mm->p, mm->w1, mm->w2, mm->w3);
  return cudaGetLastError() == cudaSuccess ? 0 : E2D_ERR_CUDA;
}

MlpDev dev_of(const e2d_mlp* mm) { return MlpDev{mm->w1, mm->w2, mm->w3, mm->p}; }

template <bool TRAIN>
int mlp_launch(e2d_mlp* mm, const float* X, const float* T, int n, float* Y, cudaStream_t st) {
  static bool configured = false;
  const size_t smem = sizeof(MlpSmem<TRAIN>);
  if (!configured) {
    if (cudaFuncSetAttribute(mlp_kernel<TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) !=
        cudaSuccess)
      return E2D_ERR_CUDA;
    configured = true;
  }
  const int ntiles = (n + TILE - 1) / TILE;
  // persistent: one CTA per SM in training (its TMEM and a gradient slot),
  // two in inference (one's products under the other's epilogue)
  const int most = TRAIN ? mm->sms : 2 * mm->sms;
  const int grid = ntiles < most ? ntiles : most;
  const int vec = ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(T) | reinterpret_cast<uintptr_t>(Y)) &
                   15u) == 0;
  mlp_kernel<TRAIN><<<grid, NT, smem, st>>>(dev_of(mm), X, T, n, 1.0f / float(n), Y, mm->gpart, mm->lpart, vec,
                                            mm->err);
  return cudaGetLastError() == cudaSuccess ? 0 : E2D_ERR_CUDA;
}

// CTAs of a training pass: the gradient slots to sum
int mlp_slots(const e2d_mlp* mm, int n) {
  const int ntiles = (n + TILE - 1) / TILE;
  return ntiles < mm->sms ? ntiles : mm->sms;
}

int mlp_check(e2d_mlp* mm, cudaStream_t st) {
  int e = 0;
  if (cudaMemcpyAsync(&e, mm->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return E2D_ERR_CUDA;
  return e ? E2D_ERR_CUDA : 0;
}

// PCG32 (O'Neill, 2014) for the initial weights.
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

}  // namespace

extern "C" {

e2d_mlp* e2d_mlp_create(uint64_t seed, int* err) {
  if (err) *err = 0;
  e2d_mlp* mm = new e2d_mlp;
  cudaGetDevice(&mm->device);
  cudaDeviceGetAttribute(&mm->sms, cudaDevAttrMultiProcessorCount, mm->device);
  bool bad = cudaMalloc(&mm->p, 4 * NPARAM) || cudaMalloc(&mm->g, 4 * NPARAM) || cudaMalloc(&mm->m, 4 * NPARAM) ||
             cudaMalloc(&mm->v, 4 * NPARAM) || cudaMalloc(&mm->w1, 2 * MH * MF) || cudaMalloc(&mm->w2, 2 * MH * MH) ||
             cudaMalloc(&mm->w3, 2 * MO * MH) || cudaMalloc(&mm->loss, sizeof(double)) ||
             cudaMalloc(&mm->gpart, 4 * size_t(NPARAM) * mm->sms) || cudaMalloc(&mm->lpart, sizeof(double) * mm->sms) ||
             cudaMalloc(&mm->err, sizeof(int));
  if (bad) {
    if (err) *err = E2D_ERR_NOMEM;
    e2d_mlp_destroy(mm);
    return nullptr;
  }
  // Glorot-uniform weights, zero biases
  std::vector<float> h(NPARAM, 0.0f);
  Pcg rng{seed * 2 + 1, (seed << 1) | 1};
  auto fill = [&](int off, int rows, int cols) {
    const double a = std::sqrt(6.0 / double(rows + cols));
    for (int q = 0; q < rows * cols; ++q) h[off + q] = float((2.0 * rng.uniform() - 1.0) * a);
  };
  fill(P_W1, MH, MF);
  fill(P_W2, MH, MH);
  fill(P_W3, MO, MH);
  if (cudaMemcpy(mm->p, h.data(), 4 * NPARAM, cudaMemcpyHostToDevice) || cudaMemset(mm->m, 0, 4 * NPARAM) ||
      cudaMemset(mm->v, 0, 4 * NPARAM) || cudaMemset(mm->err, 0, sizeof(int)) || mlp_refresh(mm, 0) ||
      cudaDeviceSynchronize()) {
    if (err) *err = E2D_ERR_CUDA;
    e2d_mlp_destroy(mm);
    return nullptr;
  }
  return mm;
}

void e2d_mlp_destroy(e2d_mlp* mm) {
  if (!mm) return;
  for (void* q : {(void*)mm->gpart, (void*)mm->lpart, (void*)mm->p, (void*)mm->g, (void*)mm->m, (void*)mm->v, (void*)mm->w1, (void*)mm->w2,
                  (void*)mm->w3, (void*)mm->loss, (void*)mm->hist, (void*)mm->err})
    if (q) cudaFree(q);
  delete mm;
}

int e2d_mlp_nparams(void) { return NPARAM; }

int e2d_mlp_params(e2d_mlp* mm, float* out, const float* in) {
  if (!mm) return E2D_ERR_ARG;
  if (in) {
    if (cudaMemcpy(mm->p, in, 4 * NPARAM, cudaMemcpyHostToDevice) != cudaSuccess) return E2D_ERR_CUDA;
    if (mlp_refresh(mm, 0) || cudaDeviceSynchronize() != cudaSuccess) return E2D_ERR_CUDA;
  }
  if (out && cudaMemcpy(out, mm->p, 4 * NPARAM, cudaMemcpyDeviceToHost) != cudaSuccess) return E2D_ERR_CUDA;
  return 0;
}

int e2d_mlp_forward(e2d_mlp* mm, const float* X, int n, float* Y, void* stream) {
  if (!mm || !X || !Y || n < 1) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = mlp_launch<false>(mm, X, nullptr, n, Y, st);
  return rc ? rc : mlp_check(mm, st);
}

int e2d_mlp_gradient(e2d_mlp* mm, const float* X, const float* T, int n, float* grad, double* loss, void* stream) {
  if (!mm || !X || !T || n < 1) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = mlp_launch<true>(mm, X, T, n, nullptr, st);
  if (rc) return rc;
  mlp_step_kernel<false><<<STEP_GRID, STEP_NT, 0, st>>>(mm->gpart, mlp_slots(mm, n), mm->g, mm->lpart, mm->loss,
                                                        mm->err, AdamArgs{});
  if (cudaGetLastError() != cudaSuccess) return E2D_ERR_CUDA;
  if ((rc = mlp_check(mm, st))) return rc;
  if (grad && cudaMemcpy(grad, mm->g, 4 * NPARAM, cudaMemcpyDeviceToHost) != cudaSuccess) return E2D_ERR_CUDA;
  if (loss) {
    double l = 0.0;
    if (cudaMemcpy(&l, mm->loss, sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return E2D_ERR_CUDA;
    *loss = l / double(n);
  }
  return 0;
}

int e2d_mlp_train(e2d_mlp* mm, const float* X, const float* T, int n, int steps, float lr, float* loss_hist,
                  void* stream) {
  if (!mm || !X || !T || n < 1 || steps < 0 || !(lr > 0.0f)) return E2D_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (loss_hist && steps > mm->hist_cap) {
    if (mm->hist && cudaFree(mm->hist) != cudaSuccess) return E2D_ERR_CUDA;
    mm->hist = nullptr;
    mm->hist_cap = 0;
    if (cudaMalloc(&mm->hist, sizeof(float) * size_t(steps)) != cudaSuccess) return E2D_ERR_NOMEM;
    mm->hist_cap = steps;
  }
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int k = 0; k < steps; ++k) {
    int rc = mlp_launch<true>(mm, X, T, n, nullptr, st);
    if (rc) return rc;
    ++mm->adam_t;
    const float c1 = 1.0f - powf(b1, float(mm->adam_t)), c2 = 1.0f - powf(b2, float(mm->adam_t));
    mlp_step_kernel<true><<<STEP_GRID, STEP_NT, 0, st>>>(
        mm->gpart, mlp_slots(mm, n), mm->g, mm->lpart, mm->loss, mm->err,
        AdamArgs{mm->p, mm->m, mm->v, mm->w1, mm->w2, mm->w3, lr, b1, b2, eps, c1, c2, double(n),
                 loss_hist ? mm->hist + k : nullptr});
    if (cudaGetLastError() != cudaSuccess) return E2D_ERR_CUDA;
  }
  if (loss_hist && steps > 0 &&
      cudaMemcpyAsync(loss_hist, mm->hist, sizeof(float) * size_t(steps), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return E2D_ERR_CUDA;
  return mlp_check(mm, st);
}

}  // extern "C"
