// e2d_arnoldi.cuh — one kernel for what lies between two Fréchet products of
// GMRES (included by e2d_nks.cu inside its anonymous namespace): modified
// Gram-Schmidt of the new Krylov vector against all earlier ones, the Givens
// rotation and stop test of the step, the scaling, the next step's
// preconditioner (block Jacobi) with its perturbation size, and the perturbed
// state.  As separate kernels (axpy_dot_kernel and the others of e2d_nks.cu)
// an Arnoldi step j was j + 8 launches of a few microseconds of work each, and
// every update passed the vector through memory.
//
// A team of CTAs holds the new vector w of a case on chip.  A team is a
// cluster of 16 CTAs (CLUSTER: reductions through distributed shared memory),
// or, for larger cases, the case's share of a cooperative launch of one CTA
// per SM (reductions through global memory).
//
// The sums are those of the separate kernels bit for bit: a slot (block,
// chunk) is summed by 256 threads, each its entries in order, then warp
// shuffles and the warps in order (cta_sum), and a case's slots by 32 lanes,
// lane l slots l, l + 32, ... in order, and shuffles (partial_done).  CTA r of a
// cluster holds slots r, r + 16, ...: those of lanes r and r + 16, whose sum is
// the shuffles' first step, so it sends one number to each CTA a reduction (a
// message costs its sender about 30 cycles: with one per slot a reduction took
// 2.6 us).
//
// Bound: the latency of a reduction, j + 2 of them a step one after another:
// about 1.3 us each in a cluster (of 2,350 cycles counted 880 for the update and
// product, 500 the warps' sums, 600 the exchange, 370 the final sum and barriers),
// 3.9 us across the GPU, against 4-5 us for a launch of axpy_dot_kernel.  Measured on
// B200: 5 Newton steps on 12,288 cells, block Jacobi 50.5 -> 28.6 ms; 6 on 98,304
// cells 29.8 -> 21.6 ms.  A counter and fences instead of tagged sums took 5.9
// us a round across the GPU, acquiring polls 6.8.
#pragma once

constexpr int AT = 512, AGROUPS = AT / VT;   // threads of a CTA, groups of 256
constexpr int ATEAM = 16;                    // CTAs of a cluster
constexpr int AREG = 2, APRE = 3;            // slots of a group kept in registers, entries of each a thread
constexpr uint32_t A_WAIT = 1u << 22;

static_assert(AREG == 2, "the shuffles pair two slots");
enum Next { NEXT_NONE = 0, NEXT_JACOBI = 1, NEXT_PERTURB = 2 };

struct ArnoldiArgs {
  Blocks B;
  GmresDev G;
  double *V, *Z;             // Krylov vectors, preconditioned vectors
  const double *Minv, *Uo;
  double *eps;
  int* active;
  int* cnt;                  // [2] cases still iterating, teams done
  const int* cta0;           // grid teams: [ncase + 1] first CTA of each case
  ulonglong2* gpart;         // grid teams: partial sums, each with its round; case c has [2][team_slots] of them
  unsigned long long* ground;  // grid teams: [ncase] rounds of all launches so far
  int maxch;                 // more of ch and chc
  long long n;
  double eps0;
  Norm4 nm;
  int j, mgs;                // Arnoldi step (-1: the start of a cycle); orthogonalise v_{j+1} first
  int next;                  // what follows for step j + 1
  int nper2, ch, len;        // vector entries (double2) per block, chunks, entries per chunk
  int cpb, chc, lenc;        // cells per block, chunks, cells per chunk
  int ctaslots, teamslots;   // most slots of a CTA, of a grid team
};

struct TeamSmem {
  uint64_t bar[2];
  double part[2][ATEAM];  // the cluster's sums of a reduction, by CTA
  double sum[2];
  int flag;
};

// Dynamic shared memory: TeamSmem, the Hessenberg column, cosines and sines
// [3][m + 2], warp sums [ctaslots][8], a grid team's partial sums [2][slots],
// the work area (w, then z).
__host__ __device__ inline size_t arnoldi_head(int ctaslots, int slots, int m) {
  return (sizeof(TeamSmem) + sizeof(double) * (3 * size_t(m + 2) + 8 * size_t(ctaslots) + 2 * size_t(slots)) + 15) / 16 *
         16;
}

// A double to another CTA of the cluster, counted on that CTA's barrier.
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
// A partial sum and the number of its round to and from global memory, as one
// 128-bit access each (single-copy atomic): a reader that finds the round has
// the sum, without a fence between data and flag.
__device__ __forceinline__ void st_tagged(ulonglong2* p, double v, unsigned long long round) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(round)
               : "memory");
}
__device__ __forceinline__ unsigned long long ld_tagged(const ulonglong2* p, double& v) {
  long long x;
  unsigned long long round;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(x), "=l"(round)
               : "l"(p)
               : "memory");
  v = __longlong_as_double(x);
  return round;
}
__device__ __forceinline__ double warp_tree(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Partial sums a grid team keeps: its case's slots, or one per CTA.
__host__ __device__ inline int team_slots(int blocks, int maxch, int ctas) {
  return blocks * maxch > ctas ? blocks * maxch : ctas;
}

template <bool CLUSTER>
struct Team {
  TeamSmem& s;
  double (*red)[VT / 32];  // warp sums of the CTA's slots
  int rank, size, round;
  ulonglong2* part;        // grid: the case's partial sums, [2][slots]
  double* copy;            // grid: the same in shared memory
  int slots;
  unsigned long long tag;  // grid: rounds of all launches so far
  bool ok;           // no wait has run out (once one has, the CTA sends and waits no more)

  // every thread: the team's sum of `count` slots, of which this CTA holds nl
  // (slot base + step * i with its warp sums in red[i]).  The CTA's first warp
  // adds each slot's warp sums in order.  A cluster's CTA adds its slots into
  // the two lanes' sums and sends their sum to every CTA; a grid team's CTA
  // sends its slots to global memory, its threads wait for a slot each and
  // every warp adds all of them.  Every CTA of a team sends something and waits
  // for all the others in every round: the sums alternate between two buffers,
  // and a CTA that nobody waited for could find its round's overwritten.
  // With `fence` the team's earlier writes to global memory are visible to every
  // thread afterwards: the CTA barrier and the sender's fence take the CTA's
  // writes along with the sum, the receivers' fences order them before the
  // threads behind the closing CTA barrier.
  __device__ double total(int count, int nl, int base, bool fence = false) {
    const int lane = threadIdx.x & 31;
    __syncthreads();
    if (CLUSTER) {
      if (threadIdx.x < 32) {
        double t = 0.0;
        for (int q = 0; q < nl; q += 32) {
          const double v = q + lane < nl ? slot_sum(q + lane) : 0.0;
          // even lanes: lane `rank` of the case's sum (slots 0, 2, ... here), odd ones: lane rank + 16
          for (int i = 0; i < min(32, nl - q); i += 2) {
            const double x = __shfl_sync(0xffffffffu, v, i + (lane & 1));
            if (q + i + (lane & 1) < nl) t += x;
          }
        }
        uint64_t* bar = &s.bar[round & 1];
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        if (lane == 0) tc::mbar_expect_tx(bar, ATEAM * 8u);
        if (ok && lane < ATEAM)
          st_async(tc::peer_addr(tc::smem_addr(&s.part[round & 1][base]), lane), t,
                   tc::peer_addr(tc::smem_addr(bar), lane));
        if (ok) ok = tc::mbar_wait_warp(bar, uint32_t(round >> 1) & 1u, A_WAIT);
        t = s.part[round & 1][lane & (ATEAM - 1)];
        for (int o = ATEAM / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s.sum[round & 1] = t;
      }
      ok = __syncthreads_and(ok) != 0;
      return s.sum[round++ & 1];
    }
    ulonglong2* gp = part + size_t(round & 1) * slots;
    double* sp = copy + size_t(round & 1) * slots;
    ++tag;
    if (fence && threadIdx.x < 32) __threadfence();
    if (ok && threadIdx.x < 32)
      for (int q = lane; q < nl; q += 32) st_tagged(gp + base + q, slot_sum(q), tag);
    // the CTAs without a slot (rank - base of them below this one) post an empty one after the slots
    if (ok && threadIdx.x == 0 && nl == 0) st_tagged(gp + count + rank - base, 0.0, tag);
    for (int q = threadIdx.x; q < max(count, size); q += AT) {
      double v;
      for (uint32_t it = 0; ld_tagged(gp + q, v) != tag;) {
        if (!ok || ++it >= A_WAIT) {
          ok = false;
          break;
        }
        if (it > 1024) __nanosleep(64);
      }
      sp[q] = v;
    }
    if (fence) __threadfence();
    ok = __syncthreads_and(ok) != 0;
    ++round;
    double t = 0.0;
    for (int q = lane; q < count; q += 32) t += sp[q];
    return warp_tree(t);
  }
  // the sum of slot i of this CTA: its warps' in order
  __device__ double slot_sum(int i) const {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < VT / 32; ++w) v += red[i][w];
    return v;
  }
  // every thread: the team's writes to global memory are visible to the team
  __device__ void barrier() {
    if (CLUSTER) {
      tc::cluster_sync();  // (a release and an acquire)
    } else {
      if (threadIdx.x < VT / 32) red[0][threadIdx.x] = 0.0;
      total(size, 1, rank, true);  // a round of one empty slot per CTA
    }
  }
};

// The last thing a team does: no CTA of a cluster leaves while another may
// still send to it; a grid team leaves its round count to the next launch.
template <bool CLUSTER>
__device__ void team_exit(const Team<CLUSTER>& t, unsigned long long* ground) {
  if (CLUSTER) tc::cluster_sync();
  else if (t.rank == 0 && threadIdx.x == 0) *ground = t.tag;
}

// One thread per case: `on` = the case still iterates after step j; the last
// case to report writes the step's count for the host.
__device__ void team_progress(const ArnoldiArgs& a, int on) {
  if (on) atomicAdd(&a.cnt[0], 1);
  __threadfence();
  if (atomicAdd(&a.cnt[1], 1) != a.G.ncase - 1) return;
  __threadfence();
  const int n = atomicExch(&a.cnt[0], 0);
  a.cnt[1] = 0;
  *(volatile int*)(a.G.progress + a.j) = n;
  __threadfence_system();
}

// The rotation and stop test of gmres_givens_kernel for case c (its Hessenberg
// column h[0..j+1], earlier rotations cs, sn in shared memory): the same
// operations.  Returns the stop flag; `write` (one CTA of the team) records
// the results.  The running right-hand side entry is read from run[j] and
// written to run[j + 1], so that every CTA of a team may compute this.
__device__ int givens_step(const GmresDev& G, int c, int j, const double* h, const double* cs, const double* sn,
                           bool write) {
  const int m = G.m;
  double* Hj = G.H + (size_t(c) * m + j) * (m + 1);
  double a = h[0];
  for (int k = 0; k < j; ++k) {
    double b = h[k + 1];
    apply_rot(a, b, cs[k], sn[k]);
    if (write) Hj[k] = a;
    a = b;
  }
  double dx = a, dy = h[j + 1], cj, sj;
  if (write && !isfinite(dy)) gm_error(G, E2D_ERR_NAN);
  make_rot(dx, dy, cj, sj);
  apply_rot(dx, dy, cj, sj);
  double r0 = G.run[size_t(c) * (m + 1) + j], r1 = 0.0;
  apply_rot(r0, r1, cj, sj);
  const double rr = fabs(r1) / G.resid0[c];
  const int its = *G.its + j + 1;
  int f = 0;
  if (rr <= G.tol[c]) f = GF_MET;
  else if (its >= G.cfg[1]) f = GF_FAILED;
  else if (j >= G.cfg[0] - 1) f = GF_RESTARTED;
  if (write) {
    Hj[j] = dx;
    Hj[j + 1] = dy;
    G.cs[size_t(c) * m + j] = cj;
    G.sn[size_t(c) * m + j] = sj;
    G.sv[size_t(c) * (m + 1) + j] = r0;
    G.run[size_t(c) * (m + 1) + j + 1] = r1;
    G.relres[c] = rr;
    if (f) {
      G.flags[c] = f;
      G.jstop[c] = j;
      G.iters[c] = its;
    }
  }
  return f;
}

// U = Uo + (eps z) normU and W = W(U) (perturb_kernel) for cell q of a case
// whose blocks start at b0.
__device__ __forceinline__ void perturb_cell(const ArnoldiArgs& a, int b0, int q, double2 za, double2 zb, double eps) {
  const Blocks& B = a.B;
  const int b = b0 + q / a.cpb, r = q % a.cpb, j = r / B.NCi, i = r % B.NCi;
  CState<double> u;
  u.d = a.Uo[cell_var(B, b, 0, j, i)] + (eps * za.x) * a.nm.u[0];
  u.mx = a.Uo[cell_var(B, b, 1, j, i)] + (eps * za.y) * a.nm.u[1];
  u.my = a.Uo[cell_var(B, b, 2, j, i)] + (eps * zb.x) * a.nm.u[2];
  u.E = a.Uo[cell_var(B, b, 3, j, i)] + (eps * zb.y) * a.nm.u[3];
  stU(B, b, i, j, u);
  stW(B, b, i, j, W_of_U(u, B.gm1));
}

template <bool CLUSTER>
__global__ void __launch_bounds__(AT, 1) arnoldi_kernel(const __grid_constant__ ArnoldiArgs a) {
  extern __shared__ __align__(16) unsigned char sraw[];
  const Blocks& B = a.B;
  const int tid = threadIdx.x, lane = tid & 31, g = tid / VT, gt = tid % VT, gw = gt >> 5;
  int c = 0;
  if (CLUSTER) c = int(blockIdx.x) / ATEAM;
  else
    while (c + 1 < a.G.ncase && int(blockIdx.x) >= a.cta0[c + 1]) ++c;
  const int rank = CLUSTER ? int(tc::cluster_rank()) : int(blockIdx.x) - a.cta0[c];
  const int size = CLUSTER ? ATEAM : a.cta0[c + 1] - a.cta0[c];
  const bool mgs = a.mgs;
  if (!a.active[c]) {  // uniform over the team
    if (mgs && rank == 0 && tid == 0) team_progress(a, 0);
    return;
  }
  const int mstride = a.G.m + 2;
  TeamSmem& s = *reinterpret_cast<TeamSmem*>(sraw);
  double* hs = reinterpret_cast<double*>(sraw + sizeof(TeamSmem));  // Hessenberg column
  double* cs = hs + mstride;          // cosines, sines
  double* sn = cs + mstride;
  double (*red)[VT / 32] = reinterpret_cast<double (*)[VT / 32]>(sn + mstride);
  unsigned char* work = sraw + arnoldi_head(a.ctaslots, CLUSTER ? 0 : a.teamslots, a.G.m);
  if (tid == 0) {
    tc::mbar_init(&s.bar[0], 1);
    tc::mbar_init(&s.bar[1], 1);
  }
  if (mgs)
    for (int k = tid; k < a.j; k += AT) {
      cs[k] = a.G.cs[size_t(c) * a.G.m + k];
      sn[k] = a.G.sn[size_t(c) * a.G.m + k];
    }
  __syncthreads();
  if (CLUSTER) tc::cluster_sync();  // the team's barriers are ready
  const int b0 = B.case_start ? B.case_start[c] : 0, b1 = B.case_start ? B.case_start[c + 1] : B.nblk;
  Team<CLUSTER> team{s, red, rank, size, 0, nullptr, reinterpret_cast<double*>(red + a.ctaslots), 0, 0ull, true};
  if (!CLUSTER) {
    team.part = a.gpart + 2 * (size_t(b0) * a.maxch + a.cta0[c]);
    team.slots = team_slots(b1 - b0, a.maxch, size);
    team.tag = *(volatile unsigned long long*)(a.ground + c);
  }
  // this CTA's slots of n: i = 0 .. nl-1 is slot base + step * i (group g
  // takes i = g, g + 2, ...)
  const int step = CLUSTER ? ATEAM : 1;
  auto first = [&](int n) { return CLUSTER ? rank : int((long long)rank * n / size); };
  auto held = [&](int n) {
    return CLUSTER ? (n - rank + ATEAM - 1) / ATEAM : int((long long)(rank + 1) * n / size) - first(n);
  };
  const int ns = (b1 - b0) * a.ch, base = first(ns), nl = held(ns);
  double2* w = reinterpret_cast<double2*>(work);
  auto entry = [&](int i, int& e0, int& e1) {  // first double2 of slot i's block, the slot's range in it
    const int q = base + step * i, blk = b0 + q / a.ch, p = q % a.ch;
    e0 = p * a.len;
    e1 = min(a.nper2, e0 + a.len);
    return size_t(blk) * a.nper2;
  };

  if (mgs) {
    double2* Vn = reinterpret_cast<double2*>(a.V + size_t(a.j + 1) * a.n);
    const double2* V0 = reinterpret_cast<const double2*>(a.V);
    const size_t vstep = size_t(a.n) / 2;
    // the group's first AREG slots stay in registers (w, v_k, v_{k+1}: the
    // latter loaded before the wait for h_k), the others in shared memory
    const bool regs = a.len <= APRE * VT;
    double2 wr[AREG][APRE], pk[AREG][APRE], pn[AREG][APRE];
    size_t ro[AREG];
    int rn[AREG];  // entries of the slot from this thread's first on
#pragma unroll
    for (int u = 0; u < AREG; ++u) {
      int e0 = 0, e1 = 0;
      const int q = g + u * AGROUPS;
      ro[u] = regs && q < nl ? entry(q, e0, e1) : 0;
      ro[u] += size_t(e0 + gt);
      rn[u] = e1 - e0 - gt;
#pragma unroll
      for (int i = 0; i < APRE; ++i) {
        wr[u][i] = pk[u][i] = pn[u][i] = make_double2(0.0, 0.0);
        if (i * VT < rn[u]) {
          wr[u][i] = Vn[ro[u] + i * VT];
          pn[u][i] = __ldg(V0 + ro[u] + i * VT);
        }
      }
    }
    const int q1 = regs ? g + AREG * AGROUPS : g;  // the first slot in shared memory
    for (int q = q1; q < nl; q += AGROUPS) {
      int e0, e1;
      const size_t o = entry(q, e0, e1);
      for (int e = e0 + gt; e < e1; e += VT) w[q * a.len + e - e0] = Vn[o + e];
    }
    double h = 0.0;
    for (int k = -1; k <= a.j; ++k) {
      // w -= h_k v_k (k >= 0), then its product with v_{k+1} (with itself at the end)
      const bool last = k == a.j;
      const double alpha = -1.0 * h;
      const double2* vk = V0 + size_t(k < 0 ? 0 : k) * vstep;
      const double2* vn = V0 + size_t(k + 1) * vstep;  // (not read when last)
      auto one = [&](double2& v, const double2& u, const double2& b, double& sum) {
        if (k >= 0) {
          v.x = v.x + alpha * u.x;
          v.y = v.y + alpha * u.y;
        }
        const double2 m = last ? v : b;
        sum += v.x * m.x;
        sum += v.y * m.y;
      };
      double rs[AREG];
#pragma unroll
      for (int u = 0; u < AREG; ++u) {
        rs[u] = 0.0;
#pragma unroll
        for (int i = 0; i < APRE; ++i)
          if (i * VT < rn[u]) one(wr[u][i], pk[u][i], pn[u][i], rs[u]);
      }
      // two slots' shuffle sums at once: the lower lanes end with the first's
      // (lane l's steps pair it with l ^ 16, ^ 8, ... as warp_tree does)
      {
        const bool up = lane >= 16;
        double t = (up ? rs[1] : rs[0]) + __shfl_xor_sync(0xffffffffu, up ? rs[0] : rs[1], 16);
        for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const int q = g + (up ? AGROUPS : 0);
        if (regs && (lane & 15) == 0 && q < nl) red[q][gw] = t;
      }
      for (int q = q1; q < nl; q += AGROUPS) {
        int e0, e1;
        const size_t o = entry(q, e0, e1);
        double sum = 0.0;
        for (int e = e0 + gt; e < e1; e += VT) {
          double2& v = w[q * a.len + e - e0];
          const double2 u = k >= 0 ? __ldg(vk + o + e) : make_double2(0.0, 0.0);
          const double2 b = last ? u : __ldg(vn + o + e);
          double2 x = v;
          one(x, u, b, sum);
          if (k >= 0) v = x;
        }
        sum = warp_tree(sum);
        if (lane == 0) red[q][gw] = sum;
      }
#pragma unroll
      for (int u = 0; u < AREG; ++u)
#pragma unroll
        for (int i = 0; i < APRE; ++i) {
          pk[u][i] = pn[u][i];
          if (k + 1 < a.j && i * VT < rn[u]) pn[u][i] = __ldg(vn + vstep + ro[u] + i * VT);
        }
      h = team.total(ns, nl, base);
      if (tid == 0) hs[k + 1] = h;
    }
    h = sqrt(h);  // ||w||
    if (tid == 0) hs[a.j + 1] = h;
    if (tid == 0) s.flag = givens_step(a.G, c, a.j, hs, cs, sn, rank == 0);
    if (!__syncthreads_and(team.ok) && tid == 0) {
      gm_error(a.G, E2D_ERR_CUDA);
      s.flag = GF_DONE;
    }
    __syncthreads();
    const int f = s.flag;
    if (rank == 0 && tid == 0) {
      if (f) a.active[c] = 0;
      team_progress(a, f ? 0 : 1);
    }
    if (f) {  // uniform over the team's CTAs whose waits have not run out
      // one whose wait has stays until the others, which may go on to the next
      // step's head, have sent to it for the last time
      if (CLUSTER && !team.ok && a.next == NEXT_JACOBI) tc::cluster_sync();  // their barrier()
      team_exit(team, a.ground + c);
      return;
    }
    // v_{j+1} = w / ||w||
    const double sc = 1.0 / h;
#pragma unroll
    for (int u = 0; u < AREG; ++u)
#pragma unroll
      for (int i = 0; i < APRE; ++i)
        if (i * VT < rn[u]) Vn[ro[u] + i * VT] = make_double2(sc * wr[u][i].x, sc * wr[u][i].y);
    for (int q = q1; q < nl; q += AGROUPS) {
      int e0, e1;
      const size_t o = entry(q, e0, e1);
      for (int e = e0 + gt; e < e1; e += VT) {
        double2 v = w[q * a.len + e - e0];
        v.x = sc * v.x;
        v.y = sc * v.y;
        Vn[o + e] = v;
      }
    }
  }
  if (a.next == NEXT_NONE) {
    team_exit(team, a.ground + c);
    return;
  }
  double2* Zn = reinterpret_cast<double2*>(a.Z + size_t(a.j + 1) * a.n);
  if (a.next == NEXT_JACOBI) {
    // z = M^-1 v per cell, the cells by slots of lenc
    if (mgs) team.barrier();  // v_{j+1} is written by other CTAs' slots too
    const double2* Vn = reinterpret_cast<const double2*>(a.V + size_t(a.j + 1) * a.n);
    const int nsc = (b1 - b0) * a.chc, basec = first(nsc), nlc = held(nsc);
    // cell k of this CTA (slot k / lenc, its k % lenc-th): its index in the case, or -1
    auto cell = [&](int k) {
      const int q = basec + step * (k / a.lenc), r = q % a.chc * a.lenc + k % a.lenc;
      return r < a.cpb ? q / a.chc * a.cpb + r : -1;
    };
    double2* zs = reinterpret_cast<double2*>(work);
    __syncthreads();  // w is read no more
    for (int k = tid; k < nlc * a.lenc; k += AT) {
      const int q = cell(k);
      if (q < 0) continue;
      const size_t o = size_t(b0) * a.cpb + q;
      const double2 va = __ldcg(Vn + 2 * o), vb = __ldcg(Vn + 2 * o + 1);
      const double2* M = reinterpret_cast<const double2*>(a.Minv + 16 * o);
      double z[4];
#pragma unroll
      for (int row = 0; row < 4; ++row) {
        const double2 m0 = __ldg(M + 2 * row), m1 = __ldg(M + 2 * row + 1);
        double t = 0.0;
        t = t + va.x * m0.x;
        t = t + va.y * m0.y;
        t = t + vb.x * m1.x;
        t = t + vb.y * m1.y;
        z[row] = t;
      }
      zs[2 * k] = Zn[2 * o] = make_double2(z[0], z[1]);
      zs[2 * k + 1] = Zn[2 * o + 1] = make_double2(z[2], z[3]);
    }
    __syncthreads();
    for (int i = g; i < nlc; i += AGROUPS) {
      double sum = 0.0;
      const int n = min(a.lenc, a.cpb - (basec + step * i) % a.chc * a.lenc);
      for (int r = gt; r < n; r += VT) {
        const double2 x = zs[2 * (i * a.lenc + r)], y = zs[2 * (i * a.lenc + r) + 1];
        sum += x.x * x.x;
        sum += x.y * x.y;
        sum += y.x * y.x;
        sum += y.y * y.y;
      }
      sum = warp_tree(sum);
      if (lane == 0) red[i][gw] = sum;
    }
    const double eps = a.eps0 / sqrt(team.total(nsc, nlc, basec));
    if (rank == 0 && tid == 0) a.eps[c] = eps;
    for (int k = tid; k < nlc * a.lenc; k += AT) {
      const int q = cell(k);
      if (q >= 0) perturb_cell(a, b0, q, zs[2 * k], zs[2 * k + 1], eps);
    }
  } else {
    // z is there: its norm by the vectors' slots
    for (int q = g; q < nl; q += AGROUPS) {
      int e0, e1;
      const size_t o = entry(q, e0, e1);
      double sum = 0.0;
      for (int e = e0 + gt; e < e1; e += VT) {
        const double2 x = __ldg(Zn + o + e);
        sum += x.x * x.x;
        sum += x.y * x.y;
      }
      sum = warp_tree(sum);
      if (lane == 0) red[q][gw] = sum;
    }
    const double eps = a.eps0 / sqrt(team.total(ns, nl, base));
    if (rank == 0 && tid == 0) a.eps[c] = eps;
    const int cells = (b1 - b0) * a.cpb;
    const int c0 = int((long long)rank * cells / size), c1 = int((long long)(rank + 1) * cells / size);
    const double2* zc = Zn + 2 * size_t(b0) * a.cpb;
    for (int q = c0 + tid; q < c1; q += AT) perturb_cell(a, b0, q, __ldg(zc + 2 * q), __ldg(zc + 2 * q + 1), eps);
  }
  if (!__syncthreads_and(team.ok) && tid == 0) gm_error(a.G, E2D_ERR_CUDA);
  team_exit(team, a.ground + c);
}
