// ilu.cu -- the ILU0 preconditioner option of CGSolver / BiCGSTABSolver on
// the device (CGConfig / BiCGSTABConfig::PreconditionerType::ILU0,
// iterative_solvers.h:59-76).
//
// The reference computes Eigen::IncompleteLUT (iterative_solvers.cpp:277-286)
// in set_matrix and, if that fails, drops to no preconditioner
// (:279-282, :805-810).  Here the preconditioner is ILU(0): L (unit, strictly
// lower) and U (upper with the diagonal) on A's own sparsity pattern, the
// classic row-by-row (IKJ) elimination restricted to that pattern.  Rows are
// grouped into levels (a row's level is one more than the highest level of
// the rows its lower part depends on), so the factorization runs as one kernel
// launch per level, a warp per row, and the two triangular solves level by
// level in one block (k_ilu_sweeps) or, for levels of many rows, as one launch
// per level, 8 lanes per row; a zero or non-finite pivot counts as a failed
// factorization and, as in the reference, the solve then runs without a
// preconditioner.  Different fill than IncompleteLUT's gives different
// iteration counts; the converged solution is the same.
//
// The Krylov iterations follow the reference's solve_with_ilu0 text step by
// step (CG :505-585; BiCGSTAB :1121-1243, whose omega is z.t / t.t with
// z = M^-1 s and whose p is not preconditioned), every scalar through a
// device state, and run as one CUDA graph: a conditional while-node whose
// body is one iteration (SpMV, dots, the level kernels of M^-1) and a control
// kernel.  Where conditional nodes are unavailable the same body runs from a
// host loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "device.h"

namespace emg {

namespace {

constexpr int kIlThreads = 256;
constexpr int kIlGrid = 592;   // vector kernels: 4 blocks of 256 threads per SM of a 148-SM B200
constexpr int kIlLanes = 8;    // lanes per row in the SpMV and the triangular solves

struct IlState {
  double bnorm, rz, rho, alpha, beta, omega, res, prev;
  double tol;
  int32_t iter, max_iter, status, done, early, div_count, loops, loop_limit;
  uint32_t ticket;  // blocks of the running kernel that have published their partial sums
};

enum Step : int32_t {
  kCgPq = 0,     // alpha = rz / p.q, breakdown test
  kCgRr = 1,     // residual of x, r
  kCgRz = 2,     // convergence, divergence, beta
  kBiRho = 3,    // rho, breakdown, beta
  kBiRv = 4,     // alpha = rho / r_hat.v
  kBiSs = 5,     // ||s||: early exit
  kBiTt = 6,     // omega = z.t / t.t
  kBiRr = 7,     // ||r||: convergence, divergence tests, next iteration
  kInitB = 8,    // ||b||
  kInitCg = 9,   // r.z of the start
  kInitBi = 10,  // rho of the start
};

__device__ __forceinline__ int64_t gtid() { return static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t gsize() { return static_cast<int64_t>(gridDim.x) * blockDim.x; }

// One step of the scalar recurrence from the totals s0, s1 (one thread).
__device__ void il_step(IlState* st, int32_t step, double s0, double s1) {
  const int32_t it = st->iter;
  switch (step) {
    case kInitB: st->bnorm = sqrt(s0); break;
    case kInitCg: st->rz = s0; break;
    case kInitBi: st->rho = s0; break;
    case kCgPq:
      if (fabs(s0) < 1e-30) { st->status = EMG_NUMERICAL_ERROR; st->done = 1; }
      else st->alpha = st->rz / s0;
      break;
    case kCgRr: st->res = sqrt(s0) / st->bnorm; break;
    case kCgRz: {
      const double res = st->res;
      if (res < st->tol) { st->status = EMG_SUCCESS; st->done = 1; break; }
      if (it > 10 && res > st->prev * 1000.0) { st->status = EMG_DIVERGED; st->done = 1; break; }
      st->beta = s0 / st->rz;
      st->rz = s0;
      st->prev = res;
      if (it >= st->max_iter) { st->status = EMG_MAX_ITER_REACHED; st->done = 1; }
      else st->iter = it + 1;
      break;
    }
    case kBiRho: {
      const double rho_old = st->rho;
      st->rho = s0;
      if (fabs(s0) < 1e-30) { st->status = EMG_NUMERICAL_ERROR; st->done = 1; break; }
      st->beta = (s0 / rho_old) * (st->alpha / st->omega);
      break;
    }
    case kBiRv:
      if (fabs(s0) < 1e-30) { st->status = EMG_NUMERICAL_ERROR; st->done = 1; }
      else st->alpha = st->rho / s0;
      break;
    case kBiSs: {
      const double res = sqrt(s0) / st->bnorm;
      st->res = res;
      if (res < st->tol) { st->status = EMG_SUCCESS; st->done = 1; st->early = 1; }
      break;
    }
    case kBiTt: st->omega = fabs(s0) < 1e-30 ? 0.0 : s1 / s0; break;
    case kBiRr: {
      const double res = sqrt(s0) / st->bnorm;
      st->res = res;
      if (res < st->tol) { st->status = EMG_SUCCESS; st->done = 1; break; }
      if (res > st->prev * 1.5 && it > 20) {
        if (++st->div_count >= 3) { st->status = EMG_DIVERGED; st->done = 1; break; }
      } else {
        st->div_count = 0;
      }
      if (it > 10 && res > st->prev * 1000.0) { st->status = EMG_DIVERGED; st->done = 1; break; }
      st->prev = res;
      if (it >= st->max_iter) { st->status = EMG_MAX_ITER_REACHED; st->done = 1; }
      else st->iter = it + 1;
      break;
    }
    default: break;
  }
}

// The block's share of up to two sums; the last block to arrive adds all
// blocks' shares in block order and takes the step.
__device__ __forceinline__ void il_finish(double a0, double a1, double* partial, IlState* st, int32_t step) {
  __shared__ double red[kIlThreads / 32];
  __shared__ bool last;
  const double b0 = block_sum(a0, red);
  const double b1 = block_sum(a1, red);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = b0;
    partial[gridDim.x + blockIdx.x] = b1;
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double c0 = 0.0, c1 = 0.0;
  for (int i = threadIdx.x; i < static_cast<int>(gridDim.x); i += blockDim.x) {
    c0 += ld_l2(partial + i);
    c1 += ld_l2(partial + gridDim.x + i);
  }
  const double s0 = block_sum(c0, red);
  const double s1 = block_sum(c1, red);
  if (threadIdx.x != 0) return;
  st->ticket = 0;
  il_step(st, step, s0, s1);
}

// ----------------------------------------------------------- factorization

// One level of the IKJ elimination, a warp per row i:
//   for k in row i with k < i (ascending): a_ik /= a_kk;
//     for j in row k with j > k and j in row i: a_ij -= a_ik a_kj.
__global__ void __launch_bounds__(kIlThreads) k_ilu_factor(const int32_t* __restrict__ rows, int32_t nrows,
                                                           const int32_t* __restrict__ rp,
                                                           const int32_t* __restrict__ col,
                                                           const int32_t* __restrict__ diag, double* lu,
                                                           int32_t* __restrict__ fail) {
  const int64_t w = gtid() >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= nrows) return;
  const int32_t i = rows[w];
  const int32_t b = rp[i + 1], d = diag[i];
  for (int32_t p = rp[i]; p < d; ++p) {
    const int32_t k = col[p];
    const double l = lu[p] / lu[diag[k]];
    __syncwarp();
    if (lane == 0) lu[p] = l;
    for (int32_t q = diag[k] + 1 + lane; q < rp[k + 1]; q += 32) {
      const int32_t j = col[q];
      int32_t lo = p + 1, hi = b;  // row i's columns after k
      while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (col[mid] < j) lo = mid + 1;
        else hi = mid;
      }
      if (lo < b && col[lo] == j) lu[lo] -= l * lu[q];
    }
    __syncwarp();
  }
  if (lane == 0) {
    const double u = lu[d];
    if (!(fabs(u) > 0.0) || !isfinite(u)) atomicOr(fail, 1);
  }
}

// ------------------------------------------------------ triangular solves

// y_i = r_i - sum_{k<i} l_ik y_k for the rows of one level (unit lower L).
__global__ void __launch_bounds__(kIlThreads) k_ilu_lower(const int32_t* __restrict__ rows, int32_t nrows,
                                                          const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ col,
                                                          const int32_t* __restrict__ diag,
                                                          const double* __restrict__ lu, const double* __restrict__ r,
                                                          double* y, const IlState* __restrict__ st) {
  if (st->done) return;
  const int64_t g = gtid() / kIlLanes;
  const int sub = threadIdx.x & (kIlLanes - 1);
  double s = 0.0;
  int32_t i = -1;
  if (g < nrows) {
    i = rows[g];
    for (int32_t p = rp[i] + sub; p < diag[i]; p += kIlLanes) s += lu[p] * y[col[p]];
  }
#pragma unroll
  for (int o = kIlLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (i >= 0 && sub == 0) y[i] = r[i] - s;
}

// z_i = (y_i - sum_{j>i} u_ij z_j) / u_ii for the rows of one level.
__global__ void __launch_bounds__(kIlThreads) k_ilu_upper(const int32_t* __restrict__ rows, int32_t nrows,
                                                          const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ col,
                                                          const int32_t* __restrict__ diag,
                                                          const double* __restrict__ lu, const double* __restrict__ y,
                                                          double* z, const IlState* __restrict__ st) {
  if (st->done) return;
  const int64_t g = gtid() / kIlLanes;
  const int sub = threadIdx.x & (kIlLanes - 1);
  double s = 0.0;
  int32_t i = -1;
  if (g < nrows) {
    i = rows[g];
    for (int32_t p = diag[i] + 1 + sub; p < rp[i + 1]; p += kIlLanes) s += lu[p] * z[col[p]];
  }
#pragma unroll
  for (int o = kIlLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (i >= 0 && sub == 0) z[i] = (y[i] - s) / lu[diag[i]];
}

// Both triangular solves in one launch of one block, for matrices whose levels
// are too small to fill more.  The solves are a chain of levels (178 of about
// 125 rows each for the 16^3 system), so what counts is the step from level
// to level: with a launch per level 2.8 us, here a block barrier, a gather
// from shared memory and a row's few multiply-adds, 0.4 us (16^3 solve 140 ->
// 28 ms).
//   Rows are stored in level order in chunks of 32 (padded), a lane a row, its
// entries in groups of four for 16-byte loads; chunk c belongs to warp c mod 16, so that with a few chunks a level a
// warp has several levels' time between its chunks: right after the barrier
// that ends its level it loads the next chunk's entries and right-hand side
// into registers (its offsets and indices came one chunk earlier still), off
// the path of the warps that work on the level now.  The last kIlRing solved
// values lie in a ring in shared memory; older ones are read back from global
// memory (which is which is known when the rows are laid out).
constexpr int kIlWarps = 16;
constexpr int kIlRing = 12288;  // values (96 KB; a multiple of 32)
constexpr int kIlZero = kIlRing;  // a slot behind the ring that stays 0: what padding entries read
constexpr int kIlRingSize = kIlRing + 2;
constexpr int kIlGroups = 2;  // groups of four entries of a row held in registers; the rest are loaded when used

struct IlSweep {
  int32_t nlev = 0, nchunk = 0;
  int64_t groups = 0;       // entry groups of all chunks (32 rows x 4 entries each)
  int32_t* lev = nullptr;   // nlev + 1: first chunk of every level
  int32_t* off = nullptr;   // nchunk + 1: first entry group of every chunk
  int32_t* in = nullptr;    // 32 nchunk: index of the row's right-hand side, -1 = padding
  int32_t* row = nullptr;   // 32 nchunk: matrix row, -1 = padding
  int4* pos = nullptr;      // [group][lane]: four entries' columns: the ring slot, or ~position once it has left the
                            // ring; padding: kIlZero
  int32_t* src = nullptr;   // [group][lane][4]: their index in the factor, -1 = padding
  double2* val = nullptr;   // [group][2][lane]: their values, refreshed with every factorization
  double* dinv = nullptr;   // 32 nchunk: 1 / u_ii (null: unit diagonal)
};

__device__ __forceinline__ void il_sweep(const IlSweep& S, const double* in, double* out, double* z, double* ring,
                                         const int32_t* lev) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  constexpr int E = 4 * kIlGroups;
  int32_t c = w;  // this warp's next chunk; its data below
  int32_t slot = 32 * w + lane;  // its ring slot: 32 c + lane modulo the ring
  int32_t pp[E], len = 0, off = 0, row = -1;
  double pv[E], rhs = 0.0, di = 1.0;
  int32_t off1 = 0, len1 = 0, idx1 = -1, row1 = -1;  // offsets and indices of the chunk after it
  auto meta = [&](int32_t k) {
    idx1 = row1 = -1;
    len1 = 0;
    if (k < S.nchunk) {
      off1 = S.off[k];
      len1 = S.off[k + 1] - off1;
      idx1 = S.in[32 * k + lane];
      if (z) row1 = S.row[32 * k + lane];
    }
  };
  auto load = [&](int32_t g, int32_t* p, double* v) {
    const int4 a = S.pos[32 * g + lane];
    const double2 x = S.val[64 * g + lane], y = S.val[64 * g + 32 + lane];
    p[0] = a.x; p[1] = a.y; p[2] = a.z; p[3] = a.w;
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
  };
  auto fetch = [&](int32_t k) {  // the chunk whose offsets are in off1 / len1 / idx1
    off = off1;
    len = len1;
#pragma unroll
    for (int g = 0; g < kIlGroups; ++g) {
      if (g < len) {
        load(off + g, pp + 4 * g, pv + 4 * g);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) { pp[4 * g + j] = kIlZero; pv[4 * g + j] = 0.0; }
      }
    }
    rhs = idx1 >= 0 ? in[idx1] : 0.0;
    di = S.dinv && idx1 >= 0 ? S.dinv[32 * k + lane] : 1.0;
    row = row1;
    meta(k + kIlWarps);
  };
  meta(c);
  fetch(c);
  for (int32_t l = 1; l <= S.nlev; ++l) {
    const int32_t e1 = lev[l];
    bool pending = false;
    while (c < e1) {
      if (pending) fetch(c);
      double g[E], s = 0.0, s1 = 0.0;
      bool far = false;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        g[j] = ring[max(pp[j], 0)];
        far |= pp[j] < 0;
      }
      if (__any_sync(0xffffffffu, far)) {
#pragma unroll
        for (int j = 0; j < E; ++j)
          if (pp[j] < 0) g[j] = out[~pp[j]];
      }
#pragma unroll
      for (int j = 0; j < E; j += 2) {
        s = fma(pv[j], g[j], s);
        s1 = fma(pv[j + 1], g[j + 1], s1);
      }
      for (int q = kIlGroups; q < len; ++q) {
        int32_t p[4];
        double v[4];
        load(off + q, p, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) s = fma(v[j], p[j] < 0 ? out[~p[j]] : ring[p[j]], s);
      }
      const double v = (rhs - (s + s1)) * di;
      const int32_t p = 32 * c + lane;
      ring[slot] = v;
      out[p] = v;
      if (row >= 0) z[row] = v;
      c += kIlWarps;
      slot += 32 * kIlWarps;
      if (slot >= kIlRing) slot -= kIlRing;
      pending = true;
    }
    __syncthreads();
    if (pending) fetch(c);
  }
}

// The line between one block and a launch per level lies at this many rows a
// level on average: 507 (32^3) 333 ms a solve against 593, 1,144 (48^3) 1.97 s
// against 1.86 (the one SM's bandwidth, about 55 GB/s here, is what bounds it).
constexpr int64_t kIlMaxRows = 1000;
// And, since the groups past those in registers are loaded one after another, at
// this many of them in a level's longest row on average. A level of band matrices
// with 8 / 12 / 20 / 24 / 28 / 100 entries a row takes 0.26 / 0.67 / 1.9 / 3.3 /
// 4.2 / 23.6 us here and 3.1 to 3.6 us as a launch.
constexpr int64_t kIlMaxTail = 4;
constexpr int kIlMaxLevels = 8000;  // of a sweep: the level offsets of both lie beside the ring
size_t ilu_sweep_smem(int32_t nl, int32_t nu) { return sizeof(double) * kIlRingSize + sizeof(int32_t) * (nl + nu + 2); }

// z = U^-1 L^-1 r
__global__ void __launch_bounds__(32 * kIlWarps) k_ilu_sweeps(IlSweep L, IlSweep U, const double* r, double* ypos,
                                                              double* zpos, double* z,
                                                              const IlState* __restrict__ st) {
  extern __shared__ __align__(16) double il_ring[];
  if (st->done) return;
  int32_t* lev = reinterpret_cast<int32_t*>(il_ring + kIlRingSize);  // both sweeps' level offsets
  for (int i = threadIdx.x; i < kIlRingSize; i += blockDim.x) il_ring[i] = 0.0;
  for (int i = threadIdx.x; i <= L.nlev; i += blockDim.x) lev[i] = L.lev[i];
  for (int i = threadIdx.x; i <= U.nlev; i += blockDim.x) lev[L.nlev + 1 + i] = U.lev[i];
  __syncthreads();
  il_sweep(L, r, ypos, nullptr, il_ring, lev);
  il_sweep(U, ypos, zpos, z, il_ring, lev + L.nlev + 1);
}

// Values of a sweep's entries (and 1 / u_ii) from the factor.
__global__ void k_ilu_pack(IlSweep S, const double* __restrict__ lu,
                           const int32_t* __restrict__ diag) {
  for (int64_t i = gtid(); i < 64 * S.groups; i += gsize()) {  // [group][half][lane]
    const int64_t g = i >> 6, lane = i & 31, half = (i >> 5) & 1;
    const int32_t* e = S.src + (32 * g + lane) * 4 + 2 * half;
    S.val[i] = make_double2(e[0] >= 0 ? lu[e[0]] : 0.0, e[1] >= 0 ? lu[e[1]] : 0.0);
  }
  if (S.dinv)
    for (int64_t i = gtid(); i < 32 * static_cast<int64_t>(S.nchunk); i += gsize())
      S.dinv[i] = S.row[i] >= 0 ? 1.0 / lu[diag[S.row[i]]] : 1.0;
}

// ------------------------------------------------------- vector kernels

// y = A x (CSR, kIlLanes lanes a row); partials w0.y (w0 null: y.y) and w1.y.
__global__ void __launch_bounds__(kIlThreads) k_il_spmv(int64_t n, const int32_t* __restrict__ rp,
                                                        const int32_t* __restrict__ col,
                                                        const double* __restrict__ val,
                                                        const double* __restrict__ x, double* __restrict__ y,
                                                        const double* __restrict__ w0, const double* __restrict__ w1,
                                                        double* partial, IlState* st, int32_t step) {
  if (st->done) return;
  const int sub = threadIdx.x & (kIlLanes - 1);
  double a0 = 0.0, a1 = 0.0;
  const int64_t groups = gsize() / kIlLanes;
  const int64_t rounds = (n + groups - 1) / groups;  // the same for every lane: the shuffles stay converged
  for (int64_t k = 0; k < rounds; ++k) {
    const int64_t row = gtid() / kIlLanes + k * groups;
    double s = 0.0;
    if (row < n)
      for (int32_t k = rp[row] + sub; k < rp[row + 1]; k += kIlLanes) s += val[k] * x[col[k]];
#pragma unroll
    for (int o = kIlLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (row < n && sub == 0) {
      y[row] = s;
      a0 += (w0 ? w0[row] : s) * s;
      if (w1) a1 += w1[row] * s;
    }
  }
  il_finish(a0, a1, partial, st, step);
}

// partials of a.b
__global__ void __launch_bounds__(kIlThreads) k_il_dot(int64_t n, const double* __restrict__ a,
                                                       const double* __restrict__ b, double* partial,
                                                       IlState* st, int32_t step) {
  if (st->done) return;
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gsize()) acc += a[i] * b[i];
  il_finish(acc, 0.0, partial, st, step);
}

// CG: x += alpha p, r -= alpha q; partials r.r
__global__ void __launch_bounds__(kIlThreads) k_il_cg_xr(int64_t n, double* __restrict__ x, double* __restrict__ r,
                                                         const double* __restrict__ p, const double* __restrict__ q,
                                                         double* partial, IlState* st, int32_t step) {
  if (st->done) return;
  const double a = st->alpha;
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gsize()) {
    x[i] += a * p[i];
    const double ri = r[i] - a * q[i];
    r[i] = ri;
    acc += ri * ri;
  }
  il_finish(acc, 0.0, partial, st, step);
}

// CG: p = z + beta p
__global__ void k_il_cg_dir(int64_t n, double* __restrict__ p, const double* __restrict__ z,
                            const IlState* __restrict__ st) {
  if (st->done) return;
  const double b = st->beta;
  for (int64_t i = gtid(); i < n; i += gsize()) p[i] = z[i] + b * p[i];
}

// BiCGSTAB: p = r + beta (p - omega v)
__global__ void k_il_bi_p(int64_t n, double* __restrict__ p, const double* __restrict__ r,
                          const double* __restrict__ v, const IlState* __restrict__ st) {
  if (st->done) return;
  const double b = st->beta, w = st->omega;
  for (int64_t i = gtid(); i < n; i += gsize()) p[i] = r[i] + b * (p[i] - w * v[i]);
}

// BiCGSTAB: s = r - alpha v; partials s.s
__global__ void __launch_bounds__(kIlThreads) k_il_bi_s(int64_t n, double* __restrict__ s,
                                                        const double* __restrict__ r, const double* __restrict__ v,
                                                        double* partial, IlState* st, int32_t step) {
  if (st->done) return;
  const double a = st->alpha;
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gsize()) {
    const double si = r[i] - a * v[i];
    s[i] = si;
    acc += si * si;
  }
  il_finish(acc, 0.0, partial, st, step);
}

// BiCGSTAB early exit on ||s||: x += alpha p (:1174-1182)
__global__ void k_il_bi_early(int64_t n, double* __restrict__ x, const double* __restrict__ p,
                              const IlState* __restrict__ st) {
  if (st->early != 1) return;
  const double a = st->alpha;
  for (int64_t i = gtid(); i < n; i += gsize()) x[i] += a * p[i];
}

// BiCGSTAB: x += alpha p + omega z, r = s - omega t; partials r.r
__global__ void __launch_bounds__(kIlThreads) k_il_bi_xr(int64_t n, double* __restrict__ x, double* __restrict__ r,
                                                         const double* __restrict__ p, const double* __restrict__ z,
                                                         const double* __restrict__ s, const double* __restrict__ t,
                                                         double* partial, IlState* st, int32_t step) {
  if (st->done) return;
  const double a = st->alpha, w = st->omega;
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gsize()) {
    x[i] += a * p[i] + w * z[i];
    const double ri = s[i] - w * t[i];
    r[i] = ri;
    acc += ri * ri;
  }
  il_finish(acc, 0.0, partial, st, step);
}

// Last node of the loop body: keep looping while not done and below the
// body-count bound (independent of the scalars, so the loop always ends).
__global__ void k_il_control(IlState* st, cudaGraphConditionalHandle handle) {
  if (threadIdx.x != 0) return;
  st->early = 0;
  const int32_t loops = st->loops + 1;
  st->loops = loops;
  cudaGraphSetConditional(handle, (!st->done && loops < st->loop_limit) ? 1u : 0u);
}

__global__ void k_il_host_control(IlState* st) {
  if (threadIdx.x != 0) return;
  st->early = 0;
  st->loops = st->loops + 1;
}

__global__ void __launch_bounds__(kIlThreads) k_il_start(int64_t n, const double* __restrict__ b, double* __restrict__ x, double* __restrict__ r,
                           double* __restrict__ rh, double* __restrict__ p, double* __restrict__ v, double* partial,
                           IlState* st, int bicg) {
  double acc = 0.0;
  for (int64_t i = gtid(); i < n; i += gsize()) {
    const double bi = b[i];
    x[i] = 0.0;
    r[i] = bi;
    if (bicg) { rh[i] = bi; p[i] = bi; v[i] = 0.0; }
    acc += bi * bi;
  }
  il_finish(acc, 0.0, partial, st, kInitB);
}

__global__ void k_il_copy(int64_t n, const double* __restrict__ a, double* __restrict__ b) {
  for (int64_t i = gtid(); i < n; i += gsize()) b[i] = a[i];
}

unsigned level_grid(int32_t rows, int lanes) {
  const int64_t threads = static_cast<int64_t>(rows) * lanes;
  return static_cast<unsigned>(std::max<int64_t>(1, (threads + kIlThreads - 1) / kIlThreads));
}

}  // namespace

struct IluState {
  int64_t n = 0, nnz = 0;
  uint64_t version = ~0ull;  // A.version the factor was computed from
  bool failed = false;       // no diagonal, or a zero / non-finite pivot
  double* lu = nullptr;
  int32_t *diag = nullptr, *lrows = nullptr, *urows = nullptr, *flag = nullptr;
  std::vector<int32_t> lptr, uptr;  // level offsets into lrows / urows
  double *x = nullptr, *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr, *y = nullptr;
  double *rh = nullptr, *v = nullptr, *s = nullptr, *t = nullptr, *part = nullptr;
  IlSweep lsw, usw;                  // level-order copies for the one-block solves (nchunk 0: not used)
  double *ypos = nullptr, *zpos = nullptr;
  IlState* st = nullptr;
  cudaStream_t cap = nullptr;
  cudaGraphExec_t loop[2] = {nullptr, nullptr};  // CG, BiCGSTAB
  bool loop_failed = false;
  std::vector<void*> mem;
};

void free_ilu(IluState* s) {
  if (!s) return;
  cudaDeviceSynchronize();
  for (cudaGraphExec_t g : s->loop)
    if (g) cudaGraphExecDestroy(g);
  if (s->cap) cudaStreamDestroy(s->cap);
  for (void* m : s->mem) cudaFree(m);
  delete s;
}

namespace {

template <class T>
int ilu_alloc(IluState& s, T** p, int64_t count) {
  void* m = nullptr;
  EMG_CK(cudaMalloc(&m, sizeof(T) * static_cast<size_t>(std::max<int64_t>(count, 1))));
  s.mem.push_back(m);
  *p = static_cast<T*>(m);
  return EMG_SUCCESS;
}

template <class T>
int ilu_upload(IluState& s, T** dst, const std::vector<T>& v, cudaStream_t st) {
  int rc = ilu_alloc(s, dst, static_cast<int64_t>(v.size()));
  if (rc) return rc;
  if (!v.empty()) EMG_CK(cudaMemcpyAsync(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st));
  EMG_CK(cudaStreamSynchronize(st));
  return EMG_SUCCESS;
}

// The level-order copies of the two triangles for k_ilu_sweeps.
int ilu_sweeps(IluState& s, const std::vector<int32_t>& rp, const std::vector<int32_t>& col,
               const std::vector<int32_t>& diag, std::vector<int32_t>& lrows, std::vector<int32_t>& urows,
               cudaStream_t st) {
  const int64_t n = s.n;
  if (n > kIlMaxRows * static_cast<int64_t>(s.lptr.size() - 1) ||
      std::max(s.lptr.size(), s.uptr.size()) > static_cast<size_t>(kIlMaxLevels))
    return EMG_SUCCESS;
  bool up = false;
  auto count = [&](int32_t i) { return up ? rp[i + 1] - diag[i] - 1 : diag[i] - rp[i]; };
  for (bool u : {false, true}) {
    up = u;
    const std::vector<int32_t>&ptr = up ? s.uptr : s.lptr, &rows = up ? urows : lrows;
    int64_t tail = 0;
    for (size_t l = 0; l + 1 < ptr.size(); ++l) {
      int32_t longest = 0;
      for (int32_t k = ptr[l]; k < ptr[l + 1]; ++k) longest = std::max(longest, count(rows[k]));
      tail += std::max((longest + 3) / 4 - kIlGroups, 0);
    }
    if (tail > kIlMaxTail * static_cast<int64_t>(ptr.size() - 1)) return EMG_SUCCESS;
  }
  std::vector<int32_t> lpos(n);
  int rc = EMG_SUCCESS;
  for (bool u : {false, true}) {
    up = u;
    const std::vector<int32_t>& ptr = up ? s.uptr : s.lptr;
    std::vector<int32_t>& rows = up ? urows : lrows;
    IlSweep& S = up ? s.usw : s.lsw;
    std::vector<int32_t> at(n), lev(1, 0), off(1, 0), in, row, pos, src;
    S.nlev = static_cast<int32_t>(ptr.size()) - 1;
    for (int32_t l = 0; l < S.nlev; ++l) {  // a level's longest rows first: chunks of even rows
      std::stable_sort(rows.begin() + ptr[l], rows.begin() + ptr[l + 1],
                       [&](int32_t a, int32_t b) { return count(a) > count(b); });
      for (int32_t k = ptr[l]; k < ptr[l + 1]; ++k) {
        if ((k - ptr[l]) % 32 == 0) row.resize((row.size() + 31) / 32 * 32, -1);
        at[rows[k]] = static_cast<int32_t>(row.size());
        row.push_back(rows[k]);
      }
      row.resize((row.size() + 31) / 32 * 32, -1);
      lev.push_back(static_cast<int32_t>(row.size() / 32));
    }
    S.nchunk = static_cast<int32_t>(row.size() / 32);
    in.assign(row.size(), -1);
    std::vector<int32_t> level_end(S.nchunk);  // first chunk past the chunk's level
    for (int32_t l = 0; l < S.nlev; ++l)
      for (int32_t c = lev[l]; c < lev[l + 1]; ++c) level_end[c] = lev[l + 1];
    for (int32_t c = 0; c < S.nchunk; ++c) {
      int32_t len = 0;
      for (int q = 0; q < 32; ++q) {
        const int32_t i = row[32 * c + q];
        if (i < 0) continue;
        len = std::max(len, count(i));
        in[32 * c + q] = up ? lpos[i] : i;
      }
      len = (len + 3) / 4;
      const size_t base = pos.size();  // [group][lane][4]
      pos.resize(base + 128 * static_cast<size_t>(len));
      src.resize(pos.size(), -1);
      for (int q = 0; q < 32; ++q) {
        const int32_t i = row[32 * c + q];
        const int32_t b = i < 0 ? 0 : up ? diag[i] + 1 : rp[i], e = i < 0 ? 0 : up ? rp[i + 1] : diag[i];
        for (int32_t j = 0; j < 4 * len; ++j) {
          const size_t k = base + 128 * static_cast<size_t>(j / 4) + 4 * q + j % 4;
          if (b + j >= e) {
            pos[k] = kIlZero;
            continue;
          }
          const int32_t p = at[col[b + j]];
          pos[k] = p >= 32 * level_end[c] - kIlRing ? p % kIlRing : ~p;
          src[k] = b + j;
        }
      }
      off.push_back(static_cast<int32_t>(pos.size() / 128));
    }
    if (!up) lpos = at;
    if ((rc = ilu_upload(s, &S.lev, lev, st)) || (rc = ilu_upload(s, &S.off, off, st)) ||
        (rc = ilu_upload(s, &S.in, in, st)) || (rc = ilu_upload(s, &S.row, row, st)) ||
        (rc = ilu_upload(s, reinterpret_cast<int32_t**>(&S.pos), pos, st)) || (rc = ilu_upload(s, &S.src, src, st)) ||
        (rc = ilu_alloc(s, &S.val, static_cast<int64_t>(pos.size()) / 2)) ||
        (rc = ilu_alloc(s, up ? &s.zpos : &s.ypos, 32 * static_cast<int64_t>(S.nchunk))))
      return rc;
    if (up && (rc = ilu_alloc(s, &S.dinv, 32 * static_cast<int64_t>(S.nchunk)))) return rc;
    S.groups = static_cast<int64_t>(pos.size()) / 128;
  }
  EMG_CK(cudaFuncSetAttribute(k_ilu_sweeps, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(ilu_sweep_smem(kIlMaxLevels, kIlMaxLevels))));
  return EMG_SUCCESS;
}

// Symbolic phase (host integer work on the pattern): diagonal positions and
// the forward / backward level schedules.
int ilu_symbolic(DevCsr& A, IluState& s, cudaStream_t st) {
  const int64_t n = A.n, nnz = A.nnz;
  std::vector<int32_t> rp(n + 1), col(std::max<int64_t>(nnz, 1));
  EMG_CK(cudaMemcpyAsync(rp.data(), A.row_ptr, sizeof(int32_t) * (n + 1), cudaMemcpyDeviceToHost, st));
  if (nnz > 0) EMG_CK(cudaMemcpyAsync(col.data(), A.col, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost, st));
  EMG_CK(cudaStreamSynchronize(st));
  std::vector<int32_t> diag(n, -1), lo(n), up(n);
  int32_t nl = 0, nu = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int32_t* b = col.data() + rp[i];
    const int32_t* e = col.data() + rp[i + 1];
    const int32_t* d = std::lower_bound(b, e, static_cast<int32_t>(i));
    if (d == e || *d != i) { s.failed = true; continue; }
    diag[i] = static_cast<int32_t>(d - col.data());
    int32_t m = -1;
    for (const int32_t* c = b; c < d; ++c) m = std::max(m, lo[*c]);
    lo[i] = m + 1;
    nl = std::max(nl, lo[i] + 1);
  }
  if (s.failed) return EMG_SUCCESS;
  for (int64_t i = n - 1; i >= 0; --i) {
    int32_t m = -1;
    for (int32_t q = diag[i] + 1; q < rp[i + 1]; ++q) m = std::max(m, up[col[q]]);
    up[i] = m + 1;
    nu = std::max(nu, up[i] + 1);
  }
  auto group = [&](const std::vector<int32_t>& lev, int32_t nlev, std::vector<int32_t>& ptr,
                   std::vector<int32_t>& rows) {
    ptr.assign(nlev + 1, 0);
    for (int64_t i = 0; i < n; ++i) ++ptr[lev[i] + 1];
    for (int32_t k = 0; k < nlev; ++k) ptr[k + 1] += ptr[k];
    rows.resize(n);
    std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
    for (int64_t i = 0; i < n; ++i) rows[fill[lev[i]]++] = static_cast<int32_t>(i);
  };
  std::vector<int32_t> lrows, urows;
  group(lo, nl, s.lptr, lrows);
  group(up, nu, s.uptr, urows);
  int rc = EMG_SUCCESS;
  if ((rc = ilu_alloc(s, &s.diag, n)) || (rc = ilu_alloc(s, &s.lrows, n)) || (rc = ilu_alloc(s, &s.urows, n)) ||
      (rc = ilu_alloc(s, &s.lu, nnz)) || (rc = ilu_alloc(s, &s.flag, 1)))
    return rc;
  EMG_CK(cudaMemcpyAsync(s.diag, diag.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
  EMG_CK(cudaMemcpyAsync(s.lrows, lrows.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
  EMG_CK(cudaMemcpyAsync(s.urows, urows.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
  EMG_CK(cudaStreamSynchronize(st));
  return ilu_sweeps(s, rp, col, diag, lrows, urows, st);
}

int ilu_numeric(DevCsr& A, IluState& s, cudaStream_t st) {
  EMG_CK(cudaMemcpyAsync(s.lu, A.val, sizeof(double) * std::max<int64_t>(A.nnz, 1), cudaMemcpyDeviceToDevice, st));
  EMG_CK(cudaMemsetAsync(s.flag, 0, sizeof(int32_t), st));
  for (size_t k = 0; k + 1 < s.lptr.size(); ++k) {
    const int32_t cnt = s.lptr[k + 1] - s.lptr[k];
    k_ilu_factor<<<level_grid(cnt, 32), kIlThreads, 0, st>>>(s.lrows + s.lptr[k], cnt, A.row_ptr, A.col, s.diag,
                                                              s.lu, s.flag);
  }
  EMG_CK(cudaGetLastError());
  int32_t f = 0;
  EMG_CK(cudaMemcpyAsync(&f, s.flag, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  EMG_CK(cudaStreamSynchronize(st));
  s.failed = f != 0;
  if (!s.failed && s.lsw.nchunk > 0) {
    k_ilu_pack<<<kIlGrid, kIlThreads, 0, st>>>(s.lsw, s.lu, s.diag);
    k_ilu_pack<<<kIlGrid, kIlThreads, 0, st>>>(s.usw, s.lu, s.diag);
    EMG_CK(cudaGetLastError());
  }
  return EMG_SUCCESS;
}

// out = U^-1 L^-1 in (out and s.y are work vectors; in is left unchanged)
void ilu_apply(DevCsr& A, IluState& s, const double* in, double* out, cudaStream_t st) {
  if (s.lsw.nchunk > 0) {
    k_ilu_sweeps<<<1, 32 * kIlWarps, ilu_sweep_smem(s.lsw.nlev, s.usw.nlev), st>>>(s.lsw, s.usw, in, s.ypos, s.zpos,
                                                                                   out, s.st);
    return;
  }
  for (size_t k = 0; k + 1 < s.lptr.size(); ++k) {
    const int32_t cnt = s.lptr[k + 1] - s.lptr[k];
    k_ilu_lower<<<level_grid(cnt, kIlLanes), kIlThreads, 0, st>>>(s.lrows + s.lptr[k], cnt, A.row_ptr, A.col, s.diag,
                                                                   s.lu, in, s.y, s.st);
  }
  for (size_t k = 0; k + 1 < s.uptr.size(); ++k) {
    const int32_t cnt = s.uptr[k + 1] - s.uptr[k];
    k_ilu_upper<<<level_grid(cnt, kIlLanes), kIlThreads, 0, st>>>(s.urows + s.uptr[k], cnt, A.row_ptr, A.col, s.diag,
                                                                   s.lu, s.y, out, s.st);
  }
}

// One iteration of the reference's solve_with_ilu0 (CG or BiCGSTAB).
void ilu_body(DevCsr& A, IluState& s, bool bicg, cudaStream_t st) {
  const int64_t n = A.n;
  if (!bicg) {
    k_il_spmv<<<kIlGrid, kIlThreads, 0, st>>>(n, A.row_ptr, A.col, A.val, s.p, s.q, s.p, nullptr, s.part, s.st, kCgPq);
    k_il_cg_xr<<<kIlGrid, kIlThreads, 0, st>>>(n, s.x, s.r, s.p, s.q, s.part, s.st, kCgRr);
    ilu_apply(A, s, s.r, s.z, st);
    k_il_dot<<<kIlGrid, kIlThreads, 0, st>>>(n, s.r, s.z, s.part, s.st, kCgRz);
    k_il_cg_dir<<<kIlGrid, kIlThreads, 0, st>>>(n, s.p, s.z, s.st);
  } else {
    k_il_dot<<<kIlGrid, kIlThreads, 0, st>>>(n, s.r, s.rh, s.part, s.st, kBiRho);
    k_il_bi_p<<<kIlGrid, kIlThreads, 0, st>>>(n, s.p, s.r, s.v, s.st);
    k_il_spmv<<<kIlGrid, kIlThreads, 0, st>>>(n, A.row_ptr, A.col, A.val, s.p, s.v, s.rh, nullptr, s.part, s.st,
                                              kBiRv);
    k_il_bi_s<<<kIlGrid, kIlThreads, 0, st>>>(n, s.s, s.r, s.v, s.part, s.st, kBiSs);
    k_il_bi_early<<<kIlGrid, kIlThreads, 0, st>>>(n, s.x, s.p, s.st);
    ilu_apply(A, s, s.s, s.z, st);
    k_il_spmv<<<kIlGrid, kIlThreads, 0, st>>>(n, A.row_ptr, A.col, A.val, s.z, s.t, nullptr, s.z, s.part, s.st,
                                              kBiTt);
    k_il_bi_xr<<<kIlGrid, kIlThreads, 0, st>>>(n, s.x, s.r, s.p, s.z, s.s, s.t, s.part, s.st, kBiRr);
  }
}

cudaGraphExec_t ilu_loop_graph(DevCsr& A, IluState& s, bool bicg) {
  if (s.loop[bicg]) return s.loop[bicg];
  if (s.loop_failed) return nullptr;
  if (!s.cap && cudaStreamCreateWithFlags(&s.cap, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    s.loop_failed = true;
    return nullptr;
  }
  cudaGraph_t graph = nullptr;
  if (cudaGraphCreate(&graph, 0) != cudaSuccess) { cudaGetLastError(); s.loop_failed = true; return nullptr; }
  cudaGraphConditionalHandle handle;
  cudaError_t e = cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault);
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = handle;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  if (e == cudaSuccess) e = cudaGraphAddNode(&node, graph, nullptr, 0, &cp);
  if (e == cudaSuccess) {
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph(s.cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      ilu_body(A, s, bicg, s.cap);
      k_il_control<<<1, 32, 0, s.cap>>>(s.st, handle);
      e = cudaStreamEndCapture(s.cap, &body);
    }
  }
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    cudaGetLastError();
    s.loop_failed = true;
    return nullptr;
  }
  s.loop[bicg] = exec;
  return exec;
}

int ilu_setup(DevCsr& A, IluState& s, cudaStream_t st) {
  s.n = A.n;
  s.nnz = A.nnz;
  int rc = ilu_symbolic(A, s, st);
  if (rc || s.failed) return rc;
  for (double** v : {&s.x, &s.r, &s.z, &s.p, &s.q, &s.y, &s.rh, &s.v, &s.s, &s.t})
    if ((rc = ilu_alloc(s, v, A.n))) return rc;
  if ((rc = ilu_alloc(s, &s.part, 2 * kIlGrid)) || (rc = ilu_alloc(s, &s.st, 1))) return rc;
  return EMG_SUCCESS;
}

int ilu_prepare(DevCsr& A, cudaStream_t st) {
  if (!A.ilu) {
    A.ilu = new IluState();
    if (const int rc = ilu_setup(A, *A.ilu, st)) {  // nothing half prepared stays
      free_ilu(A.ilu);
      A.ilu = nullptr;
      cudaGetLastError();
      return rc;
    }
  }
  IluState& s = *A.ilu;
  if (s.lu && s.version != A.version) {
    int rc = ilu_numeric(A, s, st);
    if (rc) return rc;
    s.version = A.version;
  }
  return EMG_SUCCESS;
}

}  // namespace

int ilu_solve(DevCsr& A, const double* b, double* x, const emg_krylov_config& cfg, cudaStream_t st,
              emg_result* res, bool bicg) {
  std::memset(res, 0, sizeof(*res));
  res->status = EMG_INVALID_INPUT;
  if (!b || !x) { set_error("null vector"); return EMG_INVALID_INPUT; }
  if (A.n <= 0) { set_error("empty matrix"); return EMG_INVALID_INPUT; }
  const auto t0 = std::chrono::steady_clock::now();
  int rc = ilu_prepare(A, st);
  if (rc) { res->status = rc; return rc; }
  IluState& s = *A.ilu;
  if (s.failed) {
    // as the reference's setup_preconditioner: a failed factorization leaves
    // the solver without a preconditioner
    emg_krylov_config none = cfg;
    none.preconditioner = EMG_PRECOND_NONE;
    return bicg ? bicgstab_solve(A, b, x, none, st, res) : cg_solve(A, b, x, none, st, res);
  }
  const int64_t n = A.n;
  IlState init;
  std::memset(&init, 0, sizeof(init));
  init.tol = cfg.tolerance;
  init.max_iter = cfg.max_iterations;
  init.iter = 1;
  init.status = EMG_MAX_ITER_REACHED;
  init.alpha = 1.0;
  init.omega = 1.0;
  init.res = 1.0;
  init.prev = 1.0;
  init.loop_limit = std::max(cfg.max_iterations, 0) + 2;
  EMG_CK(cudaMemcpyAsync(s.st, &init, sizeof(IlState), cudaMemcpyHostToDevice, st));
  k_il_start<<<kIlGrid, kIlThreads, 0, st>>>(n, b, s.x, s.r, s.rh, s.p, s.v, s.part, s.st, bicg ? 1 : 0);
  if (!bicg) {  // z = M^-1 r, p = z, rz = r.z
    ilu_apply(A, s, s.r, s.z, st);
    k_il_copy<<<kIlGrid, kIlThreads, 0, st>>>(n, s.z, s.p);
    k_il_dot<<<kIlGrid, kIlThreads, 0, st>>>(n, s.r, s.z, s.part, s.st, kInitCg);
  } else {
    k_il_dot<<<kIlGrid, kIlThreads, 0, st>>>(n, s.r, s.rh, s.part, s.st, kInitBi);
  }
  EMG_CK(cudaGetLastError());
  IlState h;
  EMG_CK(cudaMemcpyAsync(&h, s.st, sizeof(IlState), cudaMemcpyDeviceToHost, st));
  EMG_CK(cudaStreamSynchronize(st));
  if (h.bnorm < 1e-15) {  // :520-526 / :1137-1143
    EMG_CK(cudaMemsetAsync(x, 0, sizeof(double) * n, st));
    EMG_CK(cudaStreamSynchronize(st));
    res->status = EMG_SUCCESS;
    res->iterations = 0;
    res->residual_norm = 0.0;
    res->solve_time_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return EMG_SUCCESS;
  }
  if (cfg.max_iterations > 0) {
    cudaGraphExec_t loop = ilu_loop_graph(A, s, bicg);
    if (loop) {
      EMG_CK(cudaGraphLaunch(loop, st));
    } else {
      for (int32_t k = 0; k <= cfg.max_iterations; ++k) {
        ilu_body(A, s, bicg, st);
        k_il_host_control<<<1, 32, 0, st>>>(s.st);
        EMG_CK(cudaMemcpyAsync(&h, s.st, sizeof(IlState), cudaMemcpyDeviceToHost, st));
        EMG_CK(cudaStreamSynchronize(st));
        if (h.done) break;
      }
    }
    EMG_CK(cudaGetLastError());
  }
  k_il_copy<<<kIlGrid, kIlThreads, 0, st>>>(n, s.x, x);
  EMG_CK(cudaMemcpyAsync(&h, s.st, sizeof(IlState), cudaMemcpyDeviceToHost, st));
  EMG_CK(cudaStreamSynchronize(st));
  EMG_CK(cudaGetLastError());
  res->status = cfg.max_iterations > 0 ? (h.done ? h.status : EMG_ERR_INTERNAL) : EMG_MAX_ITER_REACHED;
  res->iterations = cfg.max_iterations > 0 ? std::min(h.iter, cfg.max_iterations) : 0;
  res->residual_norm = h.res;
  res->solve_time_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  if (res->status == EMG_ERR_INTERNAL) set_error("ILU0 solve: the loop ended before the solver state did");
  return res->status;
}

}  // namespace emg
