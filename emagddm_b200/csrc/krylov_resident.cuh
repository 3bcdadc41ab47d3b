// krylov_resident.cuh -- CG and BiCGSTAB as one persistent cooperative kernel
// for matrices whose rows fit the GPU's threads (included by krylov.cu).
//
// A solve of a few ten thousand unknowns is bound by latency, not by bytes:
// the loop graph runs two (CG) or five (BiCGSTAB) dependent launches an
// iteration, 17 us for the 22,320 rows of the 16^3 problem whose 3.4 MB matrix
// the SMs could read in one (8 us here; BiCGSTAB on 67,712 rows of 33^3
// hexahedra 33 -> 14 us).  Here one block per SM owns a contiguous run of
// slices for the whole solve: its part of the matrix is staged in shared
// memory once (as many slices as fit; the rest is read through L2), a lane
// keeps its rows' entries of every vector in registers, and only what other
// blocks gather (z and p) goes through global memory.  The two reductions of
// a CG iteration are its only grid-wide waits: every block publishes its
// partial sums in a slot of its own and reads all blocks' slots, so a
// reduction and the barrier are one trip through L2, and every block forms the
// same scalars in the same order.  p = z + beta p is formed by the reader of a
// gathered entry as well as by its owner, from the pair (z, old p) of one
// 16-byte load, which saves the third wait.  Only the reduction after the pairs
// are written carries a release / acquire fence (1.3 and 0.5 us); the one of
// p.q moves the sums alone.
#pragma once

namespace emg {
namespace {

constexpr int kResVals = 2;      // values of one reduction at most
constexpr int kResBuffers = 5;   // reductions before a slot is used again (GridSums)
constexpr int kResMaxGrid = 256; // a thread polls one block's slots
constexpr unsigned long long kResEmpty = ~0ull;  // an unpublished slot (a NaN no sum produces)

struct ResidentArgs {
  Sell A;
  const double* b;
  double* x;
  const int32_t *rp, *ccol;   // CSR, for the diagonal
  const double* cval;
  int32_t precond;
  double2* zp;                // CG: (z, old p) of every row; what other blocks gather, permuted numbering
  double *z, *p;              // BiCGSTAB: z and p, likewise
  unsigned long long* slots;  // kResBuffers x grid x kResVals, all kResEmpty at launch
  SolverState* st;
  double* hist;
  int32_t hist_cap;
  int32_t stage_slots;        // matrix slots a block can stage in shared memory
};

// Grid-wide sums of K values per thread, every thread of every block gets the
// same totals.  kFence: also the barrier that makes the blocks' earlier writes
// to global memory visible to each other (the block's slot is published with
// release semantics after its barrier).  Without it a block's sums still depend on
// all it has read, so what it read may be overwritten afterwards.  Five slot
// buffers in turn: reduction k resets the block's slots of reduction k + 3.
// Every block has read what they held, the sums of k - 2, since it has
// published to k - 1; and the reset is seen before anything is polled there,
// since one of the reductions k .. k + 2 carries the fence in every sequence
// the kernels run (CG alternates, BiCGSTAB has two without in a row at most).
// False when a wait ran out: the block raises st->copy_err at its end and the solve
// counts as timed out, whatever the other blocks had seen by then.
template <int T>
struct GridSums {
  unsigned long long* slots;
  int32_t k;
  int32_t spins;
  double (*part)[T / 32];      // [kResVals]
  double (*all)[kResMaxGrid];  // [kResVals]
  double* tot;                 // [kResVals]
  int* bad;

  template <int K, bool kFence>
  __device__ __forceinline__ bool sum(double (&v)[K]) {
    static_assert(T >= kResMaxGrid && kResVals == 2, "a thread polls the pair of slots of one block");
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, G = gridDim.x;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const double s = warp_sum(v[i]);
      if (lane == 0) part[i][w] = s;
    }
    __syncthreads();
    unsigned long long* now = slots + static_cast<int64_t>(k % kResBuffers) * (kResVals * G);
    unsigned long long* next = slots + static_cast<int64_t>((k + 3) % kResBuffers) * (kResVals * G);
    if (w < K) {
      const double s = warp_sum(lane < T / 32 ? part[w][lane] : 0.0);
      if (lane == 0) {
        unsigned long long u = __double_as_longlong(s);
        if (u == kResEmpty) u = 0x7ff8000000000000ull;
        const int64_t at = kResVals * blockIdx.x + w;
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(next + at), "l"(kResEmpty) : "memory");
        if (kFence) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(now + at), "l"(u) : "memory");
        else asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(now + at), "l"(u) : "memory");
      }
    } else if (K == 1 && w == 1 && lane == 0) {  // a slot that this reduction does not publish
      asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(next + kResVals * blockIdx.x + 1), "l"(kResEmpty)
                   : "memory");
    }
    if (t < G) {
      const unsigned long long* at = now + kResVals * t;
      unsigned long long u0 = kResEmpty, u1 = kResEmpty;
      bool got = false;
      for (int32_t i = 0; i < spins && !got; ++i) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u0), "=l"(u1) : "l"(at) : "memory");
        got = u0 != kResEmpty && (K == 1 || u1 != kResEmpty);
      }
      if (kFence) asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (!got) *bad = 1;
      all[0][t] = __longlong_as_double(u0);
      if (K > 1) all[1][t] = __longlong_as_double(u1);
    }
    __syncthreads();
    if (w < K) {
      double a[kResMaxGrid / 32], s = 0.0;
#pragma unroll
      for (int j = 0; j < kResMaxGrid / 32; ++j) a[j] = lane + 32 * j < G ? all[w][lane + 32 * j] : 0.0;
#pragma unroll
      for (int j = 0; j < kResMaxGrid / 32; ++j) s += a[j];
      s = warp_sum(s);
      if (lane == 0) tot[w] = s;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = tot[i];
    ++k;
    return *bad == 0;
  }
};

// What a block owns: slices s0 .. s0 + ns, staged into shared memory as far as
// they fit; a thread's rows are lane `lane` of the local slices w, w + 32, ...
template <int R>
struct ResidentRows {
  int32_t row[R];
  bool live[R];
  int32_t base[R];  // first slot, in shared memory or (negative: ~slot) in global memory
  int32_t len[R];
};

// sum_j v0[32 j] * get(c0[32 j]) over a row's len entries, U gathers in flight
// (masked entries multiply column 0 by 0)
template <int U, class Get>
__device__ __forceinline__ double resident_dot(const double* v0, const int32_t* c0, int len, Get get) {
  double sum[2] = {0.0, 0.0};
  for (int j = 0; j < len; j += U) {
    int c[U];
    double v[U], g[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = j + u < len ? c0[32 * (j + u)] : 0;
#pragma unroll
    for (int u = 0; u < U; ++u) g[u] = get(c[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = j + u < len ? v0[32 * (j + u)] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) sum[u & 1] += v[u] * g[u];
  }
  return sum[0] + sum[1];
}

template <int U, int NR, class Get>
__device__ __forceinline__ double resident_row(const ResidentRows<NR>& R, int q, const double* sval,
                                               const int32_t* scol, const Sell& A, Get get) {
  const int32_t b = R.base[q];
  if (b >= 0) return resident_dot<U>(sval + b, scol + b, R.len[q], get);
  return resident_dot<U < 8 ? U : 8>(A.val + ~b, A.col + ~b, R.len[q], get);
}

template <int T, int NR>
__device__ __forceinline__ void resident_stage(const ResidentArgs& P, double* sval, int32_t* scol,
                                               ResidentRows<NR>& R) {
  const Sell& A = P.A;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int64_t s0 = A.nslices * blockIdx.x / gridDim.x, s1 = A.nslices * (blockIdx.x + 1) / gridDim.x;
  const int64_t k0 = s1 > s0 ? A.slice_ptr[s0] : 0;
  const int64_t k1 = s1 > s0 ? min(A.slice_ptr[s1], k0 + P.stage_slots) : 0;
  for (int64_t k = k0 + t; k < k1; k += T) {
    sval[k - k0] = A.val[k];
    scol[k - k0] = A.col[k];
  }
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const int64_t s = s0 + w + T / 32 * q;
    R.row[q] = static_cast<int32_t>(s * kSliceRows + lane);
    R.live[q] = s < s1 && R.row[q] < A.n;
    R.base[q] = 0;
    R.len[q] = 0;
    if (s < s1) {
      const int64_t a = A.slice_ptr[s], b = A.slice_ptr[s + 1];
      R.len[q] = static_cast<int32_t>((b - a) >> 5);
      R.base[q] = b - k0 <= P.stage_slots ? static_cast<int32_t>(a - k0) + lane : ~static_cast<int32_t>(a + lane);
    }
  }
  __syncthreads();
}

// 1 / A(o, o), or 1 where |A(o, o)| <= 1e-15 (k_jacobi)
__device__ __forceinline__ double resident_dinv(const ResidentArgs& P, int32_t o) {
  if (!P.precond) return 1.0;
  int32_t lo = P.rp[o], hi = P.rp[o + 1];
  const int32_t end = hi;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (P.ccol[mid] < o) lo = mid + 1; else hi = mid;
  }
  const double a = lo < end && P.ccol[lo] == o ? P.cval[lo] : 0.0;
  return fabs(a) > 1e-15 ? 1.0 / a : 1.0;
}

#define EMG_RESIDENT_SHARED()                                                                      \
  extern __shared__ __align__(16) double res_dyn[];                                                \
  __shared__ double sh_part[kResVals][T / 32], sh_all[kResVals][kResMaxGrid], sh_tot[kResVals];     \
  __shared__ int sh_bad;                                                                           \
  double* sval = res_dyn;                                                                          \
  int32_t* scol = reinterpret_cast<int32_t*>(res_dyn + P.stage_slots);                             \
  if (threadIdx.x == 0) sh_bad = 0;                                                                \
  ResidentRows<NR> R;                                                                              \
  resident_stage<T>(P, sval, scol, R);                                                             \
  GridSums<T> sums{P.slots, 0, g_barrier_spins, sh_part, sh_all, sh_tot, &sh_bad};                 \
  constexpr int U = T == 256 ? 20 : T == 512 ? 10 : 4; /* gathers in flight a thread */            \
  const bool writer = blockIdx.x == 0 && threadIdx.x == 0;                                         \
  const double tol = P.st->tol;                                                                    \
  const int32_t max_iter = P.st->max_iter

// CG: the same recurrences, stopping and failure rules as k_cg_init,
// k_cg_spmv_dot and k_cg_update_dir.
template <int T, int NR>
__global__ void __launch_bounds__(T, 1) k_cg_resident(ResidentArgs P) {
  EMG_RESIDENT_SHARED();
  double x[NR], r[NR], d[NR], p[NR], zo[NR];
  double acc2[2] = {0.0, 0.0};
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    x[q] = r[q] = d[q] = p[q] = zo[q] = 0.0;
    if (!R.live[q]) continue;
    const int32_t o = P.A.perm[R.row[q]];
    r[q] = P.b[o];
    d[q] = resident_dinv(P, o);
    zo[q] = d[q] * r[q];
    P.zp[R.row[q]] = make_double2(zo[q], 0.0);
    acc2[0] += r[q] * r[q];
    acc2[1] += r[q] * zo[q];
  }
  bool ok = sums.template sum<2, true>(acc2);
  const double bnorm = sqrt(acc2[0]);
  double rz = acc2[1], beta = 0.0, res = bnorm / bnorm, prev = res;
  int32_t it = 1, status = EMG_MAX_ITER_REACHED;
  bool done = false;
  if (!ok) { status = EMG_ERR_TIMEOUT; done = true; }
  else if (bnorm < 1e-15) { status = EMG_SUCCESS; it = 0; res = 0.0; done = true; }  // iterative_solvers.cpp:440-446
  else if (max_iter < 1) { it = max_iter; done = true; }
  while (!done) {
    double acc1[1] = {0.0}, qv[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      p[q] = fma(beta, p[q], zo[q]);
      qv[q] = resident_row<U>(R, q, sval, scol, P.A, [&](int c) {
        const double2 zp = P.zp[c];
        return fma(beta, zp.y, zp.x);
      });
      if (R.live[q]) acc1[0] += p[q] * qv[q];
    }
    if (!sums.template sum<1, false>(acc1)) { status = EMG_ERR_TIMEOUT; break; }
    if (fabs(acc1[0]) < 1e-30) { status = EMG_NUMERICAL_ERROR; break; }  // :453-457
    const double alpha = rz / acc1[0];
    acc2[0] = acc2[1] = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      x[q] += alpha * p[q];
      r[q] -= alpha * qv[q];
      zo[q] = d[q] * r[q];
      if (!R.live[q]) continue;
      P.zp[R.row[q]] = make_double2(zo[q], p[q]);
      acc2[0] += r[q] * zo[q];
      acc2[1] += r[q] * r[q];
    }
    if (!sums.template sum<2, true>(acc2)) { status = EMG_ERR_TIMEOUT; break; }
    res = sqrt(acc2[1]) / bnorm;
    if (writer && it - 1 < P.hist_cap) P.hist[it - 1] = res;
    if (res < tol) { status = EMG_SUCCESS; break; }
    if (it > 10 && res > prev * 1000.0) { status = EMG_DIVERGED; break; }  // :477-483
    beta = acc2[0] / rz;
    rz = acc2[0];
    prev = res;
    if (it >= max_iter) break;
    ++it;
  }
#pragma unroll
  for (int q = 0; q < NR; ++q)
    if (R.live[q]) P.x[P.A.perm[R.row[q]]] = x[q];
  if (threadIdx.x == 0 && status == EMG_ERR_TIMEOUT) atomicOr(&P.st->copy_err, 1);
  if (writer) {
    P.st->status = status;
    P.st->iter = it;
    P.st->res = res;
    P.st->bnorm = bnorm;
    P.st->done = 1;
  }
}

// BiCGSTAB: as k_bi_init .. k_bi_x (the reference's variant: s preconditioned,
// p not), four reductions an iteration and one more wait for p.
template <int T, int NR>
__global__ void __launch_bounds__(T, 1) k_bi_resident(ResidentArgs P) {
  EMG_RESIDENT_SHARED();
  double x[NR], r[NR], rh[NR], d[NR], p[NR], v[NR];
  double acc1[1] = {0.0}, acc2[2];
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    x[q] = r[q] = rh[q] = d[q] = p[q] = v[q] = 0.0;
    if (!R.live[q]) continue;
    const int32_t o = P.A.perm[R.row[q]];
    r[q] = rh[q] = p[q] = P.b[o];
    d[q] = resident_dinv(P, o);
    acc1[0] += r[q] * r[q];
  }
  bool ok = sums.template sum<1, false>(acc1);
  const double bnorm = sqrt(acc1[0]);
  double rho = acc1[0], alpha = 1.0, omega = 1.0, beta = 0.0, res = bnorm / bnorm, prev = res;
  int32_t it = 1, status = EMG_MAX_ITER_REACHED, dcount = 0;
  bool done = false;
  // start of iteration `next` from rho_n = r.r_hat (bi_next_iteration)
  auto next_iteration = [&](int32_t next, double rho_n) {
    if (next > max_iter) { it = max_iter; done = true; }
    else if (fabs(rho_n) < 1e-30) { status = EMG_NUMERICAL_ERROR; it = next; done = true; }  // :1031-1035
    else { beta = (rho_n / rho) * (alpha / omega); rho = rho_n; it = next; }
  };
  if (!ok) { status = EMG_ERR_TIMEOUT; done = true; }
  else if (bnorm < 1e-15) { status = EMG_SUCCESS; it = 0; res = 0.0; done = true; }
  else next_iteration(1, rho);
  while (!done) {
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      p[q] = r[q] + beta * (p[q] - omega * v[q]);
      if (R.live[q]) P.p[R.row[q]] = p[q];
    }
    acc1[0] = 0.0;
    if (!sums.template sum<1, true>(acc1)) { status = EMG_ERR_TIMEOUT; break; }
    acc1[0] = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      v[q] = resident_row<U>(R, q, sval, scol, P.A, [&](int c) { return P.p[c]; });
      if (R.live[q]) acc1[0] += rh[q] * v[q];
    }
    if (!sums.template sum<1, false>(acc1)) { status = EMG_ERR_TIMEOUT; break; }
    if (fabs(acc1[0]) < 1e-30) { status = EMG_NUMERICAL_ERROR; break; }  // :1043-1047
    alpha = rho / acc1[0];
    acc1[0] = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      r[q] -= alpha * v[q];  // s
      if (!R.live[q]) continue;
      P.z[R.row[q]] = d[q] * r[q];
      acc1[0] += r[q] * r[q];
    }
    if (!sums.template sum<1, true>(acc1)) { status = EMG_ERR_TIMEOUT; break; }
    const double rs = sqrt(acc1[0]) / bnorm;
    if (rs < tol) {  // :1050-1058
      res = rs;
      status = EMG_SUCCESS;
      if (writer && it - 1 < P.hist_cap) P.hist[it - 1] = res;
#pragma unroll
      for (int q = 0; q < NR; ++q) x[q] += alpha * p[q];
      break;
    }
    acc2[0] = acc2[1] = 0.0;
    double tv[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      tv[q] = resident_row<U>(R, q, sval, scol, P.A, [&](int c) { return P.z[c]; });
      if (!R.live[q]) continue;
      acc2[0] += tv[q] * tv[q];
      acc2[1] += d[q] * r[q] * tv[q];
    }
    if (!sums.template sum<2, false>(acc2)) { status = EMG_ERR_TIMEOUT; break; }
    omega = fabs(acc2[0]) < 1e-30 ? 0.0 : acc2[1] / acc2[0];
    acc2[0] = acc2[1] = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      x[q] += alpha * p[q] + omega * (d[q] * r[q]);
      r[q] -= omega * tv[q];
      acc2[0] += r[q] * r[q];
      acc2[1] += r[q] * rh[q];
    }
    if (!sums.template sum<2, false>(acc2)) { status = EMG_ERR_TIMEOUT; break; }
    res = sqrt(acc2[0]) / bnorm;
    if (writer && it - 1 < P.hist_cap) P.hist[it - 1] = res;
    if (res < tol) { status = EMG_SUCCESS; break; }
    if (res > prev * 1.5 && it > 20) {  // :1083-1093
      if (++dcount >= 3) { status = EMG_DIVERGED; break; }
    } else {
      dcount = 0;
    }
    if (it > 10 && res > prev * 1000.0) { status = EMG_DIVERGED; break; }
    prev = res;
    next_iteration(it + 1, acc2[1]);
  }
#pragma unroll
  for (int q = 0; q < NR; ++q)
    if (R.live[q]) P.x[P.A.perm[R.row[q]]] = x[q];
  if (threadIdx.x == 0 && status == EMG_ERR_TIMEOUT) atomicOr(&P.st->copy_err, 1);
  if (writer) {
    P.st->status = status;
    P.st->iter = it;
    P.st->res = res;
    P.st->bnorm = bnorm;
    P.st->done = 1;
  }
}

}  // namespace
}  // namespace emg
