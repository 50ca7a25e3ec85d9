// e2d_aux.cuh — ghost fill, time step and residual-norm kernels.
//
//   ghost_fill_kernel   same-resolution exchange between blocks
//                       (Send_All_Messages, src_2D/AMR/AdaptiveBlock2D_MessagePassing.h:7883;
//                        LoadSendBuffer/UnloadReceiveBuffer, src_2D/Euler2D/Euler2DQuad.h:1570-1650)
//                       followed by BCs (src_2D/Euler2D/Euler2DQuadSingleBlock.cc:2354-2995)
//   cfl_kernel          CFL (Euler2DQuadSingleBlock.cc:3019-3080) + the global minimum
//                       (CFFC_Minimum_MPI, Euler2DQuadSolvers.cc:657-660)
//   norm kernels        L1/L2/Max_Norm_Residual (Euler2DQuadSingleBlock.cc:3111-3167,
//                       Euler2DQuadMultiBlock.cc:1017-1190)
// Compiled in the exact (no-FMA) translation unit only.
#pragma once
#include "e2d_device.cuh"
#include "e2d_geom.cuh"
#include "e2d_pdl.cuh"

#include <algorithm>

namespace e2d {

constexpr int AUX_THREADS = 256;
// most threads of a ghost-fill CTA; two such CTAs fit an SM (at most 56
// registers a thread), so a launch over 256 blocks runs in one wave
constexpr int GHOST_THREADS = 576;
constexpr double MILLION = 1000000.0;

// End of a step, by one CTA: the fused epilogue summed r^2 into the next slots'
// L2 entries; with `init` the slots after those are made ready for the next
// step's epilogue (slot_init_kernel's work).
__device__ __forceinline__ void end_step(double* hist, int* step, int fused, int ncase, int init) {
  const int k = *step;
  for (int c = threadIdx.x; c < ncase; c += blockDim.x) {
    if (fused) {
      double* h = hist + 4 * ((k + 1) * ncase + c);
      h[2] = sqrt(h[2]);
    }
    if (init) {
      double* h = hist + 4 * ((k + 2) * ncase + c);
      h[0] = MILLION; h[1] = 0.0; h[2] = 0.0; h[3] = 0.0;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *step = k + 1;
}

// Outward unit normal of the block edge's face at cell m of edge e (W, E, S,
// N): nfaceW/E/S/N of the first interior cell.
__device__ void edge_normal_at(const Blocks& B, int b, int e, int m, double& nx, double& ny) {
  switch (e) {
    case 0: nfaceW(B, b, NG, m, nx, ny); break;
    case 1: nfaceE(B, b, B.nci + NG - 1, m, nx, ny); break;
    case 2: nfaceS(B, b, m, NG, nx, ny); break;
    default: nfaceN(B, b, m, B.ncj + NG - 1, nx, ny); break;
  }
}
// Cells of a block's four edges laid end to end (W, E: NCj each; S, N: NCi).
__device__ __forceinline__ int edge_first(const Blocks& B, int e) {
  return e < 2 ? e * B.NCj : 2 * B.NCj + (e - 2) * B.NCi;
}
__device__ __forceinline__ const int* edge_codes(const Blocks& B, int b, int e) {
  return e < 2 ? (e ? B.bce : B.bcw) + size_t(b) * B.NCj : (e == 2 ? B.bcs : B.bcn) + size_t(b) * B.NCi;
}

// The boundary condition of cell m of edge e of block b: both ghost layers.
// One body for the four edges (the ghosts and the interior cells behind the
// edge lie `st` apart), with the face normal from the handle's table.
__device__ __forceinline__ void bc_edge(const Blocks& B, int b, int e, int m) {
  const bool vert = e < 2, hi = e & 1;
  const int bc = edge_codes(B, b, e)[m];
  const double2 nrm = B.edge_nrm[size_t(b) * 2 * (B.NCj + B.NCi) + edge_first(B, e) + m];
  const size_t plane = size_t(B.NCj) * B.NCi;
  const int nc = vert ? B.nci : B.ncj, in = hi ? nc + NG - 1 : NG;  // interior cells across, the first one
  const long long st = (hi ? 1ll : -1ll) * (vert ? 1 : B.NCi);
  const long long o = (long long)(vert ? cell_var(B, b, 0, m, in) : cell_var(B, b, 0, in, m));
  auto ld = [&](const double* a, long long q, double* v) {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = a[q + (long long)(k * plane)];
  };
  auto st4 = [&](double* a, long long q, const double* v) {
#pragma unroll
    for (int k = 0; k < 4; ++k) a[q + (long long)(k * plane)] = v[k];
  };
  auto set = [&](int g, const PState<double>& w) {  // ghost layer g
    const CState<double> u = U_of_W(w, B.gm1i);
    const double wv[4] = {w.d, w.u, w.v, w.p}, uv[4] = {u.d, u.mx, u.my, u.E};
    st4(B.W, o + g * st, wv);
    st4(B.U, o + g * st, uv);
  };
  double v0[4], v1[4];  // the first two interior cells
  ld(B.W, o, v0);
  ld(B.W, o - st, v1);
  if (bc == E2D_BC_NONE) return;
  const double* wo = vert ? (hi ? B.woe : B.wow) : (hi ? B.won : B.wos);
  const PState<double> w0{v0[0], v0[1], v0[2], v0[3]};
  if (bc == E2D_BC_FIXED) {
    const PState<double> w = wo_at(wo, b, vert ? B.NCj : B.NCi, m);
#pragma unroll
    for (int g = 1; g <= NG; ++g) set(g, w);
  } else if (bc == E2D_BC_REFLECTION) {
    set(1, reflect(w0, nrm.x, nrm.y));
    set(2, reflect(PState<double>{v1[0], v1[1], v1[2], v1[3]}, nrm.x, nrm.y));
  } else if (bc == E2D_BC_CHARACTERISTIC) {
    const PState<double> w =
        bc_char_pressure(w0, wo_at(wo, b, vert ? B.NCj : B.NCi, m), nrm.x, nrm.y, B.g, B.gm1i);
#pragma unroll
    for (int g = 1; g <= NG; ++g) set(g, w);
  } else {
    // copies: the opposite side's interior (periodic), else the first interior
    // cell (constant extrapolation, the reference's default)
#pragma unroll
    for (int g = 1; g <= NG; ++g) {
      const long long q = bc == E2D_BC_PERIODIC ? o - (nc - g) * st : o;
      double wv[4], uv[4];
      ld(B.W, q, wv);
      ld(B.U, q, uv);
      st4(B.W, o + g * st, wv);
      st4(B.U, o + g * st, uv);
    }
  }
}
static_assert(NG == 2, "two ghost layers");

// Ghost cell q of block b's exchange, from its neighbour across k (W, E, S, N,
// then the corners): two layers of an edge, a 2 x 2 patch of a corner.
__device__ __forceinline__ void exchange_cell(const Blocks& B, int b, int q) {
  const int ICl = NG, ICu = B.nci + NG - 1, JCl = NG, JCu = B.ncj + NG - 1;
  const int ne = NG * B.ncj, nn = NG * B.nci, nc = NG * NG;
  int k, r = q;
  if (r < 2 * ne) { k = r / ne; r %= ne; }
  else if ((r -= 2 * ne) < 2 * nn) { k = 2 + r / nn; r %= nn; }
  else { r -= 2 * nn; k = 4 + r / nc; r %= nc; }
  const int s = B.neigh[b * 8 + k];
  if (s < 0) return;
  int i, j, di, dj;
  const bool wi = (k == 0 || k == 4 || k == 6), ei = (k == 1 || k == 5 || k == 7);
  const bool sj = (k == 2 || k == 4 || k == 5), nj = (k == 3 || k == 6 || k == 7);
  int ri, rj;  // position inside the ghost patch
  if (k < 2) { ri = r % NG; rj = r / NG; }
  else if (k < 4) { ri = r % B.nci; rj = r / B.nci; }
  else { ri = r % NG; rj = r / NG; }
  if (wi) { i = ICl - NG + ri; di = (ICu + 1) - ICl; }
  else if (ei) { i = ICu + 1 + ri; di = ICl - (ICu + 1); }
  else { i = ICl + ri; di = 0; }
  if (sj) { j = JCl - NG + rj; dj = (JCu + 1) - JCl; }
  else if (nj) { j = JCu + 1 + rj; dj = JCl - (JCu + 1); }
  else { j = JCl + rj; dj = 0; }
  const CState<double> u = ldU(B, s, i + di, j + dj);
  stU(B, b, i, j, u);
  stW(B, b, i, j, W_of_U(u, B.gm1));
}

// Per block (bc_flag_kernel, once per handle): BCF_ANY, an edge cell has a
// boundary condition; BCF_MIXED, an edge has conditions on some of its cells
// only or on an edge that also exchanges with a neighbour.
constexpr unsigned BCF_ANY = 1, BCF_MIXED = 2;

// One CTA per block: exchange, then W/E BCs, then S/N BCs (the reference's
// order; the S/N pass also fills the corner ghosts).
//
// Off the corners a condition reads interior cells only, so in a block whose
// edges have it on all their cells or on none, and no neighbour where they do,
// everything but the corners is one round of independent items -- exchanged
// cells and edge cells, each its own thread -- and a second round, after a
// barrier, applies to the corners the condition that comes last there: W/E on
// the ghost rows of an S or N edge without one, else S/N on the ghost columns.
// A mixed block takes exchange, W/E and S/N one after another.
//
// Latency bound, by rounds of loads (B200, cold caches): 12 blocks of 32 x 32
// with walls and characteristic ends 9.1 us a fill against 12.6 in passes of two
// edges a thread with the normals from the nodes, 256 periodic blocks of 64 x 64
// 8.9 against 8.6.
//
// With `hist` a CTA of its own ends the step before (end_step), once step[1]
// says that there is one: a kernel less in the chain of a step (100 two-stage
// steps of 16 blocks of 32 x 32 2.30 -> 2.19 ms).
__global__ void __launch_bounds__(GHOST_THREADS, 2) ghost_fill_kernel(Blocks B, double* hist, int* step) {
  const int b = blockIdx.x;
  if (b == B.nblk) {
    pdl_launch_next();
    pdl_wait();
    const bool pending = step[1] != 0;
    __syncthreads();
    if (pending) end_step(hist, step, 1, B.ncase, 1);
    else if (threadIdx.x == 0) step[1] = 1;
    return;
  }
  const unsigned flag = B.bcflag[b];
  pdl_launch_next();
  pdl_wait();
  if (*(volatile int*)B.status) return;  // uniform: an earlier kernel failed
  const int total = 2 * NG * (B.nci + B.ncj) + 4 * NG * NG;
  const bool mixed = flag & BCF_MIXED;
  const int phases = mixed ? 3 : (flag & BCF_ANY ? 2 : 1);
  for (int ph = 0; ph < phases; ++ph) {
    if (ph) __syncthreads();
    const int items = mixed ? (ph == 0 ? total : (ph == 1 ? 2 * B.NCj : 2 * B.NCi))
                            : (ph == 0 ? total + (phases > 1 ? 2 * (B.nci + B.ncj) : 0) : 8 * NG);
    for (int q = threadIdx.x; q < items; q += blockDim.x) {
      if (ph == 0 && q < total) {
        exchange_cell(B, b, q);
        continue;
      }
      int e, m;  // edge and its cell
      if (mixed) {
        const int n = ph == 1 ? B.NCj : B.NCi;
        e = (ph == 1 ? 0 : 2) + q / n;
        m = q % n;
      } else if (ph == 0) {
        const int r = q - total, v = 2 * B.ncj;
        e = r < v ? r / B.ncj : 2 + (r - v) / B.nci;
        m = NG + (r < v ? r % B.ncj : (r - v) % B.nci);
      } else {  // corners: four edges, their 2 NG cells in the ghost rows or columns
        e = q / (2 * NG);
        m = q % (2 * NG);
        if (m >= NG) m += (e < 2 ? B.ncj : B.nci);
      }
      // W and E along ghost rows only where the S or N edge has no condition
      if (e < 2 && (m < NG || m >= B.ncj + NG) &&
          edge_codes(B, b, m < NG ? 2 : 3)[e ? B.nci + NG : NG - 1] != E2D_BC_NONE)
        continue;
      bc_edge(B, b, e, m);
    }
  }
}

// The normals of the edges' faces, for the fills' whole life.
__global__ void edge_normal_kernel(Blocks B, double2* nrm) {
  const int per = 2 * (B.NCj + B.NCi);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)per * B.nblk;
       t += (long long)gridDim.x * blockDim.x) {
    const int b = int(t / per), q = int(t % per);
    const int e = q < 2 * B.NCj ? q / B.NCj : 2 + (q - 2 * B.NCj) / B.NCi;
    double2 n;
    edge_normal_at(B, b, e, q - edge_first(B, e), n.x, n.y);
    nrm[t] = n;
  }
}

// The flags of ghost_fill_kernel, one warp per block.
__global__ void bc_flag_kernel(Blocks B, unsigned char* flags) {
  const int b = blockIdx.x;
  bool any = false, mixed = false;
  for (int e = 0; e < 4; ++e) {
    const int n = e < 2 ? B.NCj : B.NCi;
    const int* code = edge_codes(B, b, e);
    bool some = false, all = true;
    for (int q = threadIdx.x; q < n; q += 32) {
      some |= code[q] != E2D_BC_NONE;
      all &= code[q] != E2D_BC_NONE;
    }
    some = __any_sync(0xffffffffu, some);
    all = __all_sync(0xffffffffu, all);
    any |= some;
    mixed |= some && (!all || B.neigh[b * 8 + e] >= 0);
  }
  if (threadIdx.x == 0) flags[b] = (unsigned char)((any ? BCF_ANY : 0u) | (mixed ? BCF_MIXED : 0u));
}

// Positive doubles order like their int64 bit patterns.
__device__ __forceinline__ void atomic_min_pos(double* addr, double v) {
  atomicMin(reinterpret_cast<unsigned long long*>(addr), __double_as_longlong(v));
}
__device__ __forceinline__ void atomic_max_pos(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr), __double_as_longlong(v));
}

// Local time step of every interior cell and the minimum of each case (into
// its slot of the step history).  One CTA per block.
__global__ void __launch_bounds__(AUX_THREADS) cfl_kernel(Blocks B, double* hist, const int* step) {
  __shared__ double red[AUX_THREADS / 32];
  const int b = blockIdx.x;
  double* dtmin = hist + 4 * ((*step) * B.ncase + case_id(B, b));
  const int per = B.nci * B.ncj;
  double m = MILLION;
  for (int r = threadIdx.x; r < per; r += blockDim.x) {
    const int i = NG + r % B.nci, j = NG + r / B.nci;
    double xc, yc, A;
    quad_centroid(nodeX(B, b, i, j), nodeY(B, b, i, j), nodeX(B, b, i + 1, j), nodeY(B, b, i + 1, j),
                  nodeX(B, b, i + 1, j + 1), nodeY(B, b, i + 1, j + 1), nodeX(B, b, i, j + 1),
                  nodeY(B, b, i, j + 1), xc, yc, A);
    const double lE = glen(B, b, i + 1, j, i + 1, j + 1), lW = glen(B, b, i, j, i, j + 1);
    const double lN = glen(B, b, i, j + 1, i + 1, j + 1), lS = glen(B, b, i, j, i + 1, j);
    const double per_c = lE + lN + lW + lS;
    double nEx, nEy, nWx, nWy, nNx, nNy, nSx, nSy;
    gnormal(B, b, i + 1, j + 1, i + 1, j, lE, per_c, nEx, nEy);
    gnormal(B, b, i, j, i, j + 1, lW, per_c, nWx, nWy);
    gnormal(B, b, i, j + 1, i + 1, j + 1, lN, per_c, nNx, nNy);
    gnormal(B, b, i + 1, j, i, j, lS, per_c, nSx, nSy);
    const PState<double> w = ldW(B, b, i, j);
    const double d_i = 2.0 * (A / (lE + lW));
    const double d_j = 2.0 * (A / (lN + lS));
    const double v_i = HALF * (w.u * (nEx - nWx) + w.v * (nEy - nWy));
    const double v_j = HALF * (w.u * (nNx - nSx) + w.v * (nNy - nSy));
    const double a = a_of(w, B.g);
    const double dt = dmin(d_i / (a + fabs(v_i)), d_j / (a + fabs(v_j)));
    if (B.local_dt) B.dt[cell_sc(B, b, j, i)] = dt;
    m = dmin(m, dt);
  }
  for (int o = 16; o > 0; o >>= 1) m = dmin(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < AUX_THREADS / 32 ? red[threadIdx.x] : MILLION;
    for (int o = 16; o > 0; o >>= 1) m = dmin(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) atomic_min_pos(dtmin, m);
  }
}

// Per-block sums of |r|, r^2 and max |r| of the density residual.
__global__ void __launch_bounds__(AUX_THREADS) norm_partial_kernel(Blocks B, double* part) {
  __shared__ double red[3][AUX_THREADS / 32];
  const int b = blockIdx.x;
  double s1 = 0, s2 = 0, mx = 0;
  for (int r = threadIdx.x; r < B.nci * B.ncj; r += blockDim.x) {
    const int i = NG + r % B.nci, j = NG + r / B.nci;
    const double v = B.dUdt[cell_var(B, b, 0, j, i)];
    s1 += fabs(v);
    s2 += v * v;
    mx = dmax(mx, fabs(v));
  }
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    mx = dmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = s1; red[1][threadIdx.x >> 5] = s2; red[2][threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s1 = 0; s2 = 0; mx = 0;
    for (int w = 0; w < AUX_THREADS / 32; ++w) { s1 += red[0][w]; s2 += red[1][w]; mx = dmax(mx, red[2][w]); }
    part[3 * b] = s1; part[3 * b + 1] = s2; part[3 * b + 2] = mx;
  }
}

// Combines the per-block partials in block order as the multi-block norms
// and the solver loop do; out = (L1, L2, Max) of each case.
// One warp per case: lane l sums the case's blocks l, l+32, ...; the lanes
// are then combined.
__global__ void norm_final_kernel(Blocks B, const double* part, double* hist, const int* step) {
  if (threadIdx.x >= 32) return;
  const int c = blockIdx.x;
  const int b0 = B.case_start ? B.case_start[c] : 0, b1 = B.case_start ? B.case_start[c + 1] : B.nblk;
  double l1 = 0, l2 = 0, mx = 0;
  for (int b = b0 + threadIdx.x; b < b1; b += 32) {
    l1 += part[3 * b];
    l2 += sqr(sqrt(part[3 * b + 1]));
    mx = dmax(mx, part[3 * b + 2]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    l2 += __shfl_xor_sync(0xffffffffu, l2, o);
    mx = dmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (threadIdx.x == 0) {
    double* out = hist + 4 * ((*step) * B.ncase + c) + 1;
    out[0] = l1;
    out[1] = sqrt(sqr(sqrt(l2)));
    out[2] = mx;
  }
}

__global__ void fill_kernel(double* p, long long n, double v) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    p[q] = v;
}

// Explicit-step bookkeeping: the step index lives on the device so that one
// captured step graph replays for every step.
// Slot of step *step + offset: dt = MILLION (min-reduced), norms = 0 (summed).
__global__ void slot_init_kernel(double* hist, const int* step, int offset, int ncase) {
  for (int c = threadIdx.x; c < ncase; c += blockDim.x) {
    double* h = hist + 4 * ((*step + offset) * ncase + c);
    h[0] = MILLION; h[1] = 0.0; h[2] = 0.0; h[3] = 0.0;
  }
}
__global__ void step_end_kernel(double* hist, int* step, int fused, int ncase, int init) {
  pdl_launch_next();
  pdl_wait();
  end_step(hist, step, fused, ncase, init);
}

cudaError_t launch_ghost_fill(const Blocks& B, cudaStream_t st, double* hist, int* step) {
  // one thread per exchanged ghost cell or edge cell where the block allows (a
  // single round of independent loads), at least one CTA of AUX_THREADS
  const int cells = 2 * NG * (B.nci + B.ncj) + 4 * NG * NG;
  const int threads = std::min(GHOST_THREADS, std::max(AUX_THREADS, (cells + 31) / 32 * 32));
  return launch_pdl(ghost_fill_kernel, B.nblk + (hist ? 1 : 0), threads, 0, st, B, hist, step);
}

cudaError_t launch_edge_setup(const Blocks& B, unsigned char* flags, double2* nrm, cudaStream_t st) {
  bc_flag_kernel<<<B.nblk, 32, 0, st>>>(B, flags);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long n = 2ll * (B.NCj + B.NCi) * B.nblk;
  edge_normal_kernel<<<int(std::min<long long>((n + 255) / 256, 1184)), 256, 0, st>>>(B, nrm);
  return cudaGetLastError();
}

cudaError_t launch_cfl(const Blocks& B, double* hist, const int* step, cudaStream_t st) {
  cfl_kernel<<<B.nblk, AUX_THREADS, 0, st>>>(B, hist, step);
  return cudaGetLastError();
}

cudaError_t launch_norms(const Blocks& B, double* part, double* hist, const int* step, cudaStream_t st) {
  norm_partial_kernel<<<B.nblk, AUX_THREADS, 0, st>>>(B, part);
  norm_final_kernel<<<B.ncase, 32, 0, st>>>(B, part, hist, step);
  return cudaGetLastError();
}

cudaError_t launch_slot_init(double* hist, const int* step, int offset, int ncase, cudaStream_t st) {
  slot_init_kernel<<<1, 128, 0, st>>>(hist, step, offset, ncase);
  return cudaGetLastError();
}
cudaError_t launch_step_end(double* hist, int* step, int fused, int ncase, int init, cudaStream_t st) {
  return launch_pdl(step_end_kernel, 1, 128, 0, st, hist, step, fused, ncase, init);
}
cudaError_t launch_fill(double* p, long long n, double v, cudaStream_t st) {
  int grid = int((n + 255) / 256);
  if (grid > 1184) grid = 1184;
  if (grid < 1) grid = 1;
  fill_kernel<<<grid, 256, 0, st>>>(p, n, v);
  return cudaGetLastError();
}

}  // namespace e2d
