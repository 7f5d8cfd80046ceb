// Device GMRES with Householder orthogonalisation (FP64).
//
// Restates dgmresr_hh (fmex/solve3d.c:339-518).  The reference applies the
// reflectors P_r = I - 2 u_r u_r' one after another; each needs a global
// inner product before its update, so a step that applies j of them one by
// one meets j grid barriers.  Here the product of the reflectors is kept in
// compact WY form (Schreiber and Van Loan, SIAM J. Sci. Stat. Comput. 10
// (1989) 53-57), P_0 ... P_j = I - U T U' with U = [u_0 .. u_j] and T upper
// triangular, T(j,j) = 2, T(0:j,j) = -2 T U(:,0:j)' u_j: all inner products
// of a step are taken at once.  Outside the matvec one Arnoldi step is one
// cooperative launch with two grid barriers:
//   hh_init   : restart vector, u_0, v_0 = P_0 e_0                 (:376-392)
//   hh_step   : w = P_j ... P_0 (B v_j), next reflector, Givens    (:421-473),
//               then v_{j+1} = P_0 ... P_{j+1} e_{j+1}             (:396-406)
//   hh_correct: triangular solve and the correction x += Q y       (:487-507)
// Partial sums are reduced in a fixed order, so results are deterministic
// run to run.  Every barrier wait is bounded: on timeout the kernel raises
// the context error flag and runs to completion, and the host returns
// TTG_ERR_TIMEOUT.
#include <cmath>
#include <cstring>

#include "gmres.h"
#include "group.cuh"

namespace ttg {

namespace {

constexpr int HH_THREADS = 512;
constexpr int HH_WARPS = HH_THREADS / 32;
constexpr long long BAR_SPIN_LIMIT = 1LL << 24;

// Restart lengths up to which k_hh_correct stages R in shared memory.
constexpr int64_t HH_CORRECT_STAGE_MAX = 64;

// Restart lengths up to which T is kept a second time (34 MB at most) in the
// order that T' (U' w2) reads it; beyond, those reads are strided.  64 x 64 x 64, a
// restart of 250: 67.8 ms for 68.5; of 900: 774 for 822; of 120 and less the same.
constexpr int64_t HH_OWN_T_MAX = 2048;

// Shared memory of k_hh_step: three vectors over the reflectors and the
// per-warp partial inner products (the Givens section reuses the space).
size_t hh_step_smem(int64_t nrestart) {
  return sizeof(double) * size_t(4 * (nrestart + 1) + 4 * HH_WARPS);
}
size_t hh_correct_smem(int64_t nrestart, int64_t ni) {
  return sizeof(double) * size_t(3 * ni + (nrestart <= HH_CORRECT_STAGE_MAX ? ni * ni : 0));
}

struct HhArgs {
  int64_t sz;
  int64_t nrestart;
  double* U;  // sz x (nrestart+1)
  double* w;
  double* w2;
  double* sol;
  const double* rhs;
  double* tau;   // nrestart+1
  double* J;     // 2 x nrestart
  // R (upper triangle, ld nrestart + 2) and, from the row below its diagonal on, the
  // transpose TT of the WY factor (lower triangle) in one array; T itself, element
  // (q, r) at q tq + r tr: the same entries, or for short restarts an array of its own.
  double* R;
  double* TT;
  double* T;
  int64_t tq, tr;
  double* scal;  // [0] nrmrhs [1] curres [2] nrmr [3] exact-flag [4] w[j+1]
  double* part;  // 2 x (nrestart+2) x gridDim.x partial sums
  unsigned* bar; // [0] count [1] generation
  int* err;
  int* stop;     // [0] converged flag, [1] step at which it converged
  double tol;    // relative stopping tolerance of the current solve
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum, result broadcast to every thread.
__device__ double block_sum_all(double v) {
  __shared__ double sh[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double r = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
    r = warp_sum(r);
    if (threadIdx.x == 0) sh[32] = r;
  }
  __syncthreads();
  return sh[32];
}

__device__ void grid_barrier(TTG_BLOCK, unsigned* bar, int* err,
                             long long limit = BAR_SPIN_LIMIT) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* vgen = bar + 1;
    volatile int* verr = err;
    const unsigned gen = *vgen;
    __threadfence();
    const unsigned arrived = atomicAdd(bar, 1u);
    if (arrived == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      long long spins = 0;
      while (*vgen == gen) {
        if (*verr) break;
        if (++spins > limit) {
          atomicExch(err, 1);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// First row and end of this block's share of the rows.
__device__ __forceinline__ int64_t row_at(int64_t sz, int64_t b, int64_t nb) { return sz * b / nb; }

// part[r * nb + b] = sum over this block's rows [i0, i1) of U_r[i] w[i],
// r < nr.  Four columns per warp share the loads of w; with fewer column
// groups than warps the rows of a group are split over several warps.
__device__ void hh_dots(const double* U, int64_t sz, int64_t nr, const double* w, int64_t i0,
                        int64_t i1, double* sp, double* part, int64_t b, int64_t nb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t G = (nr + 3) / 4, RP = G >= HH_WARPS ? 1 : HH_WARPS / G;
  for (int64_t unit = warp; unit < G * RP; unit += HH_WARPS) {
    const int64_t g = unit / RP, p = unit % RP;
    const double* u0 = U + 4 * g * sz;
    const double* u1 = U + min(4 * g + 1, nr - 1) * sz;
    const double* u2 = U + min(4 * g + 2, nr - 1) * sz;
    const double* u3 = U + min(4 * g + 3, nr - 1) * sz;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    const int64_t lo = i0 + (i1 - i0) * p / RP, hi = i0 + (i1 - i0) * (p + 1) / RP;
#pragma unroll 4
    for (int64_t i = lo + lane; i < hi; i += 32) {
      const double x = w[i];
      s0 = fma(u0[i], x, s0);
      s1 = fma(u1[i], x, s1);
      s2 = fma(u2[i], x, s2);
      s3 = fma(u3[i], x, s3);
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    s3 = warp_sum(s3);
    if (lane < 4 && 4 * g + lane < nr)
      sp[(4 * g + lane) * RP + p] = lane == 0 ? s0 : lane == 1 ? s1 : lane == 2 ? s2 : s3;
  }
  __syncthreads();
  for (int64_t r = threadIdx.x; r < nr; r += blockDim.x) {
    double s = 0.0;
    for (int64_t p = 0; p < RP; ++p) s += sp[r * RP + p];
    part[r * nb + b] = s;
  }
}

// out[r] = sum over the blocks of part[r * nb + b] in a fixed order, r < nr.
__device__ void hh_gather(const double* part, int64_t nb, int64_t nr, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t r = warp; r < nr; r += HH_WARPS) {
    double s = 0.0;
    for (int64_t b = lane; b < nb; b += 32) s += __ldcg(part + r * nb + b);
    s = warp_sum(s);
    if (lane == 0) out[r] = s;
  }
  __syncthreads();
}

// v - sum_r U_r[i] y[r], r < nr
__device__ __forceinline__ double hh_row(const double* U, int64_t sz, int64_t nr, int64_t i,
                                         const double* y, double v) {
  const double* u = U + i;
#pragma unroll 8
  for (int64_t r = 0; r < nr; ++r) v = fma(-u[r * sz], y[r], v);
  return v;
}

// w = rhs - w2 ; U_0 = Householder vector of w ; tau_0 = -beta  (:376-392);
// then v_0 = P_0 e_0 into w.
TTG_BODY(k_hh_init)(TTG_BLOCK, HhArgs a, int it) {
  const int64_t sz = a.sz, nb = gridDim.x, b = blockIdx.x;
  const int64_t i0 = row_at(sz, b, nb), i1 = row_at(sz, b + 1, nb);
  __shared__ double tot;
  double s = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const double v = a.rhs[i] - a.w2[i];
    a.w[i] = v;
    s = fma(v, v, s);
    if (i == 0) a.scal[4] = v;  // read by every block after the barrier
  }
  s = block_sum_all(s);
  if (threadIdx.x == 0) a.part[b] = s;
  grid_barrier(blockIdx, gridDim, a.bar, a.err);
  hh_gather(a.part, nb, 1, &tot);
  const double nrmr = sqrt(tot);
  if (b == 0 && threadIdx.x == 0) {
    if (it == 0) a.scal[0] = nrmr;
    a.scal[2] = nrmr;
    a.scal[3] = (nrmr == 0.0) ? 1.0 : 0.0;
  }
  if (nrmr == 0.0) return;
  const double w0 = __ldcg(a.scal + 4);
  const double beta = (w0 < 0.0) ? -nrmr : nrmr;
  const double nu = sqrt(2.0 * nrmr * nrmr + 2.0 * beta * w0);
  const double u0 = (w0 + beta) / nu;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const double u = i == 0 ? u0 : a.w[i] / nu;
    a.U[i] = u;
    a.w[i] = fma(-2.0 * u0, u, i == 0 ? 1.0 : 0.0);
  }
  if (b == 0) {
    for (int64_t k = threadIdx.x; k <= a.nrestart; k += blockDim.x) a.tau[k] = 0.0;
    __syncthreads();
    if (threadIdx.x == 0) {
      a.tau[0] = -beta;
      a.T[0] = a.TT[0] = 2.0;
    }
  }
}
TTG_COOP_KERNEL(k_hh_init, HH_THREADS, COOP_CTAS);

// One Arnoldi step around the matvec w2 = B v_j:
//   w2 = P_j ... P_0 w2 = w2 - U T' (U' w2)                     (:421-427)
//   next reflector u_{j+1} from w2 below row j                  (:428-443)
//   Givens rotations, R(:,j), residual estimate                 (:445-473)
//   v_{j+1} = P_0 ... P_{j+1} e_{j+1}, into w                   (:396-406)
// Row j + 1 of U gives U' e_{j+1}, so v_{j+1} takes no further inner products
// but those of the new column of T, U' u_{j+1}: they are formed from the
// rows of w2 below j together with their norm, before u_{j+1} is known
// (u_{j+1} = (w2 + alpha e_{j+1}) / nu there).  v_{j+1} has unit norm by
// construction.  Bound by the four reads of U a step (41 columns of 64 x 64 x
// 64 are 86 MB, mostly L2 hits): a local solve of two restarts of 40 at that
// size takes 5.8 ms, 40 us of it this kernel per step, against 20.3 ms with
// one grid barrier per reflector (225 us per step) and the same matvec.
TTG_BODY(k_hh_step)(TTG_BLOCK, HhArgs a, int64_t j) {
  if (*(volatile int*)a.stop) return;  // queued after convergence
  extern __shared__ double hsm[];
  const int64_t sz = a.sz, m1 = a.nrestart + 1, ld = m1 + 1, nr = j + 1;
  const int64_t nb = gridDim.x, b = blockIdx.x;
  const int64_t i0 = row_at(sz, b, nb), i1 = row_at(sz, b + 1, nb);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* sd = hsm;       // inner products
  double* sy = sd + m1;   // coefficients of the columns of U
  double* su = sy + m1;   // row j + 1 of U
  double* sp = su + m1;   // per-warp partials
  double* part2 = a.part + (m1 + 1) * nb;
  double* w = a.w2;

  hh_dots(a.U, sz, nr, w, i0, i1, sp, a.part, b, nb);
  grid_barrier(blockIdx, gridDim, a.bar, a.err);
  hh_gather(a.part, nb, nr, sd);
  for (int64_t r = warp; r < nr; r += HH_WARPS) {  // T' (U' w2)
    double s = 0.0;
    for (int64_t q = lane; q <= r; q += 32) s = fma(a.T[q * a.tq + r * a.tr], sd[q], s);
    s = warp_sum(s);
    if (lane == 0) sy[r] = s;
  }
  __syncthreads();
  const bool next = j < sz - 1;          // a new reflector exists
  const bool build = j + 1 < a.nrestart;  // and another step follows
  double s = 0.0;
  for (int64_t i = i0 + tid; i < i1; i += blockDim.x) {
    const double v = hh_row(a.U, sz, nr, i, sy, w[i]);
    w[i] = v;
    if (i > j) s = fma(v, v, s);
    if (i == j + 1) a.scal[4] = v;
  }
  s = block_sum_all(s);  // and every thread's rows of w are written
  if (next && build)
    hh_dots(a.U, sz, nr, w, max(i0, min(nr, i1)), i1, sp, part2, b, nb);
  if (tid == 0) part2[nr * nb + b] = s;
  grid_barrier(blockIdx, gridDim, a.bar, a.err);

  double alpha = 0.0;
  if (next) {
    if (build) {
      hh_gather(part2, nb, nr + 1, sd);
      alpha = sqrt(sd[nr]);
    } else {
      hh_gather(part2 + nr * nb, nb, 1, sd);
      alpha = sqrt(sd[0]);
    }
    const double wj1 = __ldcg(a.scal + 4);
    if (wj1 < 0.0) alpha = -alpha;
    if (build) {
      const double nu = alpha != 0.0 ? sqrt(2.0 * alpha * alpha + 2.0 * alpha * wj1) : 1.0;
      const double uj1 = (wj1 + alpha) / nu;
      for (int64_t r = tid; r < nr; r += blockDim.x) {
        const double ur = __ldcg(a.U + (j + 1) + r * sz);
        su[r] = ur;
        sd[r] = fma(alpha, ur, sd[r]) / nu;  // U' u_{j+1}
      }
      __syncthreads();
      for (int64_t q = warp; q < nr; q += HH_WARPS) {
        double t = 0.0, y = 0.0;
        for (int64_t r = q + lane; r < nr; r += 32) {
          const double Tqr = a.TT[r + q * ld];
          t = fma(Tqr, sd[r], t);
          y = fma(Tqr, su[r], y);
        }
        t = -2.0 * warp_sum(t);
        y = warp_sum(y);
        if (lane == 0) {
          sy[q] = fma(t, uj1, y);
          if (b == 0) a.T[q * a.tq + nr * a.tr] = a.TT[nr + q * ld] = t;
        }
      }
      if (b == 0 && tid == 0) a.T[nr * a.tq + nr * a.tr] = a.TT[nr + nr * ld] = 2.0;
      __syncthreads();
      double* Un = a.U + nr * sz;
      const double yn = 2.0 * uj1;
      for (int64_t i = i0 + tid; i < i1; i += blockDim.x) {
        const double u = i <= j ? 0.0 : (i == j + 1 ? uj1 : w[i] / nu);
        Un[i] = u;
        a.w[i] = hh_row(a.U, sz, nr, i, sy, fma(-u, yn, i == j + 1 ? 1.0 : 0.0));
      }
    }
  }
  if (b == 0) {
    // Givens rotations of the new Hessenberg column (:445-449) by one thread
    // on shared-memory copies of the column and of the rotators.
    __syncthreads();
    double* wl = hsm;                 // nrestart + 1
    double* Jl = hsm + a.nrestart + 1;  // 2 nrestart
    for (int64_t e = tid; e <= j; e += blockDim.x) wl[e] = __ldcg(w + e);
    for (int64_t e = tid; e < 2 * j; e += blockDim.x) Jl[e] = a.J[e];
    __syncthreads();
    if (tid == 0) {
      if (next) wl[j + 1] = -alpha;
      for (int64_t i = 0; i < j; ++i) {
        const double x = wl[i], x1 = wl[i + 1];
        const double c0 = Jl[2 * i], c1 = Jl[2 * i + 1];
        wl[i] = c0 * x + c1 * x1;
        wl[i + 1] = -c1 * x + c0 * x1;
      }
      if (next) {  // new rotator (:454-465)
        const double wj = wl[j], wj1 = wl[j + 1];
        const double rho = sqrt(wj * wj + wj1 * wj1);
        const double c0 = wj / rho, c1 = wj1 / rho;
        a.J[2 * j] = c0;
        a.J[2 * j + 1] = c1;
        a.tau[j + 1] = -c1 * a.tau[j];
        a.tau[j] = c0 * a.tau[j];
        wl[j] = rho;
      }
      const double curres = fabs(a.tau[j + 1]) / a.scal[0];
      a.scal[1] = curres;
      if (curres < a.tol) {  // (:476) later queued steps see the flag and return
        a.stop[1] = int(j);
        __threadfence();
        a.stop[0] = 1;
      }
    }
    __syncthreads();
    for (int64_t k = tid; k <= j; k += blockDim.x) a.R[k + j * ld] = wl[k];
  }
}
TTG_COOP_KERNEL(k_hh_step, HH_THREADS, COOP_CTAS);

// y = R^{-1} tau, then sol += P_0 ... P_j (sum_i y_i e_i)
//                        = sol + y - U T (U' y)                 (:487-507)
// Every block solves the small system for itself; no barrier.
TTG_BODY(k_hh_correct)(TTG_BLOCK, HhArgs a, int64_t ni) {
  pdl_begin();
  extern __shared__ double y[];  // y (ni), U' y (ni), T U' y (ni), R when staged (ld ni)
  const int64_t sz = a.sz, ld = a.nrestart + 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool staged = a.nrestart <= HH_CORRECT_STAGE_MAX;
  double* sc = y + ni;
  double* st = sc + ni;
  double* Rs = st + ni;
  if (staged)
    for (int64_t e = tid; e < ni * ni; e += blockDim.x)
      Rs[e] = a.R[(e % ni) + (e / ni) * ld];
  for (int64_t e = tid; e < ni; e += blockDim.x) y[e] = a.tau[e];
  __syncthreads();
  if (warp == 0) {  // back-substitution, one column at a time
    const double* R = staged ? Rs : a.R;
    const int64_t ldr = staged ? ni : ld;
    for (int64_t c = ni - 1; c >= 0; --c) {
      const double v = y[c] / R[c + c * ldr];
      __syncwarp();
      if (lane == 0) y[c] = v;
      for (int64_t r = lane; r < c; r += 32) y[r] = fma(-R[r + c * ldr], v, y[r]);
      __syncwarp();
    }
  }
  __syncthreads();
  for (int64_t r = warp; r < ni; r += HH_WARPS) {  // u_r has no entries above row r
    double s = 0.0;
    for (int64_t i = r + lane; i < ni; i += 32) s = fma(a.U[i + r * sz], y[i], s);
    s = warp_sum(s);
    if (lane == 0) sc[r] = s;
  }
  __syncthreads();
  for (int64_t q = warp; q < ni; q += HH_WARPS) {
    double s = 0.0;
    for (int64_t r = q + lane; r < ni; r += 32) s = fma(a.TT[r + q * ld], sc[r], s);
    s = warp_sum(s);
    if (lane == 0) st[q] = s;
  }
  __syncthreads();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + tid; i < sz;
       i += int64_t(gridDim.x) * blockDim.x)
    a.sol[i] += hh_row(a.U, sz, ni, i, st, i < ni ? y[i] : 0.0);
}
TTG_KERNEL(k_hh_correct, HH_THREADS);

// Blocks of the cooperative kernels: contiguous row ranges of at least HH_ROWS
// rows, at most two blocks per SM (Context::coop_ctas).  Two keep twice the loads of U in flight
// (64 x 64 x 64, 80 steps: one block an SM takes 8 us a step longer); small systems take
// few blocks, and 256 or 512 rows as the least share measure the same.
constexpr int64_t HH_ROWS = 256;
int coop_blocks(Context* c, const void* kernel, size_t smem, int64_t sz) {
  const int occ = std::max(1, max_active_blocks(kernel, HH_THREADS, smem));
  const int64_t cap = int64_t(c->num_sms) * std::min(occ, c->coop_ctas);
  return int(std::max<int64_t>(1, std::min((sz + HH_ROWS - 1) / HH_ROWS, cap)));
}

}  // namespace

GmresResult gmres_hh_f64(Context* c, const ApplyFn& apply, const double* rhs, int64_t sz,
                         int64_t nrestart, double tol, int64_t niters, double* sol) {
  GmresResult res;
  TTG_REQUIRE(nrestart >= 1 && nrestart <= 4096, "nrestart %lld out of range",
              (long long)nrestart);
  DBuf<double> U(c, size_t(sz) * (nrestart + 1)), w(c, sz), w2(c, sz);
  const int64_t m1 = nrestart + 1;
  const int64_t ld = m1 + 1, square = ld * m1;
  const bool own_t = nrestart <= HH_OWN_T_MAX;
  DBuf<double> small(c, m1 + 2 * nrestart + (own_t ? 2 : 1) * square + 8);
  const size_t step_smem = hh_step_smem(nrestart);
  ensure_smem_attr(k_hh_step.fn(), c->device, int(hh_step_smem(4096)));
  ensure_smem_attr(k_hh_correct.fn(), c->device, int(hh_correct_smem(4096, 4096)));
  const int blocks = std::min(coop_blocks(c, k_hh_init.fn(), 0, sz),
                              coop_blocks(c, k_hh_step.fn(), step_smem, sz));
  DBuf<double> part(c, 2 * (m1 + 1) * blocks);
  DBuf<unsigned> bar(c, 4);
  DBuf<int> stop(c, 4);
  memset_async(c, bar.p(), 0, 4 * sizeof(unsigned));
  memset_async(c, c->d_err, 0, sizeof(int));

  HhArgs a;
  a.sz = sz;
  a.nrestart = nrestart;
  a.U = U.p();
  a.w = w.p();
  a.w2 = w2.p();
  a.sol = sol;
  a.rhs = rhs;
  a.tau = small.p();
  a.J = a.tau + (nrestart + 1);
  a.R = a.J + 2 * nrestart;
  a.TT = a.R + 1;
  a.T = own_t ? a.R + square : a.TT;
  a.tq = own_t ? 1 : ld;
  a.tr = own_t ? m1 : 1;
  a.scal = a.R + (own_t ? 2 : 1) * square;
  a.part = part.p();
  a.bar = bar.p();
  a.err = c->d_err;
  a.stop = stop.p();
  a.tol = tol;
  fill_f64(c, sz, 0.0, sol);

  // Arnoldi steps are queued in chunks of growing length without a host
  // round trip per step; k_hh_step raises a device flag on convergence and
  // every kernel queued after it (further steps and the matvec GEMMs,
  // through Context::skip) returns at once.  The host reads the flag, the
  // converged step and the residual estimate once per chunk.
  struct Probe {
    int flag[2];
    double curres;
  };
  auto probe = [&](Probe& p) {
    double* stage = c->h_scal;
    const int* sp = stop.p();
    const double* cp = a.scal + 1;
    if (c->rec) {
      rec_read(c, 0, sp, 2 * sizeof(int));
      rec_read(c, sizeof(double), cp, sizeof(double));
      rec_wait(c->rec);
    } else {
      TTG_CUDA(cudaMemcpyAsync(stage, sp, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
      TTG_CUDA(
          cudaMemcpyAsync(stage + 1, cp, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
      sync(c);
    }
    memcpy(p.flag, stage, 2 * sizeof(int));
    p.curres = stage[1];
  };
  double curres = INFINITY;
  for (int64_t it = 0; it < niters; ++it) {
    apply(sol, w2.p());
    res.matvecs++;
    launch(c, k_hh_init, blocks, HH_THREADS, 0, a, int(it));
    memset_async(c, stop.p(), 0, 2 * sizeof(int));
    double hs[4];
    read_scalars(c, a.scal, hs, 4);
    if (hs[3] != 0.0) {  // exact solution: nothing to correct
      curres = 0.0;
      break;
    }
    bool broke = false;
    int64_t j = 0, chunk = 3;
    SkipGuard guard(c, stop.p());
    while (j < nrestart) {
      const int64_t jend = std::min(nrestart, j + chunk);
      for (int64_t jj = j; jj < jend; ++jj) {
        apply(w.p(), w2.p());
        launch(c, k_hh_step, blocks, HH_THREADS, step_smem, a, jj);
      }
      Probe p;
      probe(p);
      curres = p.curres;
      if (p.flag[0]) {
        broke = true;
        j = p.flag[1];
        break;
      }
      j = jend;
      chunk *= 2;
    }
    guard.release();
    const int64_t steps = broke ? j + 1 : nrestart;
    res.iters += steps;
    res.matvecs += steps;
    int64_t ni;
    if (!broke) {
      j = nrestart - 1;
      ni = nrestart;
    } else {
      ni = j + 1;
    }
    launch(c, k_hh_correct, blocks, HH_THREADS, hh_correct_smem(nrestart, ni), a, ni);
    if (curres < tol) break;
  }
  res.relres = curres;
  return res;
}

// Self-test of the bounded grid barrier: block 1 never arrives, so block 0
// waits until its (small) poll limit runs out and raises *flag.
__global__ void k_selftest_grid_barrier(unsigned* bar, int* flag, long long limit) {
  if (blockIdx.x != 0) return;
  grid_barrier(blockIdx, gridDim, bar, flag, limit);
}

void selftest_wait_gmres(Context* c, int* flag, long long limit) {
  DBuf<unsigned> bar(c, 2);
  TTG_CUDA(cudaMemsetAsync(bar.p(), 0, 2 * sizeof(unsigned), c->stream));
  k_selftest_grid_barrier<<<2, 32, 0, c->stream>>>(bar.p(), flag, limit);
  TTG_CHECK_LAUNCH();
  sync(c);
}

}  // namespace ttg
