// Mixed-precision local solve: FP64 iterative refinement around an FP32
// GMRES whose matvecs run on BF16 tensor cores (mixed_ops.cu).
//
// Same contract as the MEX local solver (fmex/solve3d_2.c:254-279): start
// from sol_prev and stop once ||rhs - B sol|| <= tol ||rhs||, with the true
// residual always evaluated by the FP64 matvec.  Each refinement step solves
// B dx = r approximately in low precision (relative tolerance 1e-3 or the
// remaining target, whichever is looser), then sol += dx and r is recomputed
// in FP64.  The inner Krylov solver is GMRES(restart) with classical
// Gram-Schmidt applied twice (CGS2): one cooperative kernel per Arnoldi step
// performs both projections, the normalisation and the Givens update of the
// least-squares residual; partial sums are reduced in a fixed order.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "group.cuh"
#include "jacobi.h"
#include "mixed.h"
#include "mixed_ops.h"

namespace ttg {

namespace {

constexpr int AR_THREADS = 512;
constexpr int AR_WARPS = AR_THREADS / 32;
constexpr long long AR_SPIN_LIMIT = 1LL << 24;
constexpr int MAX_OUTER = 8;
constexpr double INNER_TOL = 1e-3;
// Least rows of a block of the cooperative Arnoldi kernels: 512 measures the
// same, 2048 4% slower on solves of 97 x 64 x 83 and on batches of small ones.
constexpr int64_t AR_ROWS = 1024;

struct ArArgs {
  int64_t sz;
  int64_t ldv;     // sz rounded up to a multiple of 4 (float4 loads)
  int m;           // restart length
  float* V;        // ldv x (m+1), zero in rows sz..ldv
  float* w;        // matvec output (ldv, zero in rows sz..ldv), orthogonalised in place
  double* H;       // (m+1) x m, column-major
  double* cs;      // m
  double* sn;      // m
  double* g;       // m+1
  double* scal;    // [0] |g_{j+1}|  [1] norm of the new Arnoldi vector  [2] beta
                   // [3] norm of the solve's right-hand side  [4] stop threshold
  double* part;    // 2 * (m+2) * gridDim.x
  unsigned* bar;   // [0] count [1] generation
  int* err;
  int* stop;       // [0] converged flag, [1] step at which it converged (-1: at start)
  double reltol;   // stop once |g_{j+1}| <= reltol * scal[3]
  // BF16 operand of the next local matvec, written with each new basis
  // vector: X[b + ldx * row] = bf16(V[b + rx2 * row]) (padding b >= rx2 stays
  // zero), so the matvec needs no conversion launch.
  __nv_bfloat16* X;
  int rx2;
  int ldx;
};

// Four consecutive entries i..i+3 of a new basis vector (those below sz).
__device__ __forceinline__ void put_x4(const ArArgs& a, int64_t i, const float4& v) {
  if (!a.X) return;  // preconditioned solve: the operand is P v, written apart
  int64_t row;
  int b;
  if (a.sz <= 0xffffffffll) {  // 32-bit division where it holds the index
    row = unsigned(i) / unsigned(a.rx2);
    b = int(unsigned(i) - unsigned(row) * unsigned(a.rx2));
  } else {
    row = i / a.rx2;
    b = int(i - row * a.rx2);
  }
  const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i + k < a.sz) a.X[b + int64_t(a.ldx) * row] = __float2bfloat16_rn(e[k]);
    if (++b == a.rx2) {
      b = 0;
      ++row;
    }
  }
}

__device__ __forceinline__ double warp_sumd(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ void ar_barrier(TTG_BLOCK, unsigned* bar, int* err, long long limit = AR_SPIN_LIMIT) {
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
          atomicExch(err, 4);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
}

#define AR_LOOP(idx, n)                                                             \
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < (n);    \
       idx += int64_t(gridDim.x) * blockDim.x)

// This block's share of the rows, in groups of four.
__device__ __forceinline__ int64_t quad_at(const ArArgs& a, int64_t b, int64_t nb) {
  return (a.ldv / 4) * b / nb;
}

__device__ __forceinline__ float dot4(const float4& u, const float4& x) {
  return fmaf(u.w, x.w, fmaf(u.z, x.z, fmaf(u.y, x.y, u.x * x.x)));
}

// part[c*nb + block] = block partial of V(:,c)'w, c < ncol.  Four columns per
// warp share the loads of w; with fewer column groups than warps the rows of
// a group are split over several warps.  Products of four rows are summed in
// FP32, everything beyond in FP64.  sp: m + 1 + 4 AR_WARPS doubles.
__device__ void partial_dots(const ArArgs& a, int ncol, int64_t q0, int64_t q1, int64_t b,
                             int64_t nb, double* part, double* sp) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = (ncol + 3) / 4, RP = G >= AR_WARPS ? 1 : AR_WARPS / G;
  const int64_t ldq = a.ldv / 4;
  const float4* V = reinterpret_cast<const float4*>(a.V);
  const float4* w = reinterpret_cast<const float4*>(a.w);
  for (int unit = warp; unit < G * RP; unit += AR_WARPS) {
    const int g = unit / RP, p = unit % RP;
    const float4* v0 = V + 4 * g * ldq;
    const float4* v1 = V + min(4 * g + 1, ncol - 1) * ldq;
    const float4* v2 = V + min(4 * g + 2, ncol - 1) * ldq;
    const float4* v3 = V + min(4 * g + 3, ncol - 1) * ldq;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    const int64_t lo = q0 + (q1 - q0) * p / RP, hi = q0 + (q1 - q0) * (p + 1) / RP;
#pragma unroll 2
    for (int64_t q = lo + lane; q < hi; q += 32) {
      const float4 x = w[q];
      s0 += double(dot4(v0[q], x));
      s1 += double(dot4(v1[q], x));
      s2 += double(dot4(v2[q], x));
      s3 += double(dot4(v3[q], x));
    }
    s0 = warp_sumd(s0);
    s1 = warp_sumd(s1);
    s2 = warp_sumd(s2);
    s3 = warp_sumd(s3);
    if (lane < 4 && 4 * g + lane < ncol)
      sp[(4 * g + lane) * RP + p] = lane == 0 ? s0 : lane == 1 ? s1 : lane == 2 ? s2 : s3;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
    double s = 0.0;
    for (int p = 0; p < RP; ++p) s += sp[c * RP + p];
    part[c * nb + b] = s;
  }
}

// Sum the block partials of ncol columns (same fixed order in every block).
__device__ void reduce_parts(TTG_BLOCK, const double* part, int ncol, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = warp; c < ncol; c += AR_WARPS) {
    double s = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(part + int64_t(c) * gridDim.x + b);
    s = warp_sumd(s);
    if (lane == 0) out[c] = s;
  }
  __syncthreads();
}

// Block-wide sum in thread 0; red: AR_WARPS doubles.
__device__ __forceinline__ double block_sum0(double v, double* red) {
  v = warp_sumd(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int q = 0; q < AR_WARPS; ++q) t += red[q];
  return t;
}

// w - sum_c V(q, c) h[c] for the four rows of group q
__device__ __forceinline__ float4 project4(const float4* V, int64_t ldq, int ncol, int64_t q,
                                           const float* h, float4 w) {
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int c = 0; c < ncol; ++c) {
    const float4 v = V[c * ldq + q];
    const float hc = h[c];
    s.x = fmaf(v.x, hc, s.x);
    s.y = fmaf(v.y, hc, s.y);
    s.z = fmaf(v.z, hc, s.z);
    s.w = fmaf(v.w, hc, s.w);
  }
  w.x -= s.x;
  w.y -= s.y;
  w.z -= s.z;
  w.w -= s.w;
  return w;
}

// Shared memory of k_arnoldi, in doubles: hp (m+2), ht (m+2), partials
// (m+1 + 4 AR_WARPS), the rotations of the Givens update (2 m), and hf (m+1
// floats).
__host__ __device__ __forceinline__ size_t arnoldi_doubles(int m) {
  return size_t(2 * (m + 2) + (m + 1 + 4 * AR_WARPS) + 2 * m);
}

// One Arnoldi step for column j: w -= V h twice (CGS2), normalise into
// V(:, j+1), Givens update of H(:, j) and g; scal[0] = |g_{j+1}|.
// Two grid barriers, one per projection: with w1 the vector after the first
// and h2 its coefficients, the norm after the second is |w1|^2 - |h2|^2; only
// when the second projection removes more than a quarter of it (w lies in the
// span of the basis to rounding) is the norm summed over the result, at a
// third barrier.  Bound by reading V four times from L2 at large sizes (97 x
// 64 x 83, mean over 40 columns: 24 us per step, against 50 us with three
// barriers, scalar loads and the norm in a pass of its own) and by the two
// barriers at small ones (13 against 22 us in a batch of twelve systems).
TTG_BODY(k_arnoldi)(TTG_BLOCK, ArArgs a, int j) {
  if (*(volatile int*)a.stop) return;  // queued after convergence
  extern __shared__ double shd[];
  const int m = a.m, ncol = j + 1;
  const int64_t b = blockIdx.x, nb = gridDim.x;
  const int64_t q0 = quad_at(a, b, nb), q1 = quad_at(a, b + 1, nb), ldq = a.ldv / 4;
  const int tid = threadIdx.x;
  double* hp = shd;              // this pass's coefficients, then |w1|^2
  double* ht = hp + (m + 2);     // accumulated coefficients
  double* sp = ht + (m + 2);
  double* cl = sp + (m + 1 + 4 * AR_WARPS);
  float* hf = reinterpret_cast<float*>(cl + 2 * m);
  double* part0 = a.part;
  double* part1 = a.part + int64_t(m + 2) * nb;
  const float4* V = reinterpret_cast<const float4*>(a.V);
  float4* w = reinterpret_cast<float4*>(a.w);
  float4* Vn = reinterpret_cast<float4*>(a.V) + int64_t(j + 1) * ldq;

  partial_dots(a, ncol, q0, q1, b, nb, part0, sp);
  ar_barrier(blockIdx, gridDim, a.bar, a.err);
  reduce_parts(blockIdx, gridDim, part0, ncol, hp);
  for (int c = tid; c < ncol; c += blockDim.x) {
    ht[c] = hp[c];
    hf[c] = float(hp[c]);
  }
  __syncthreads();
  double n1 = 0.0;
  for (int64_t q = q0 + tid; q < q1; q += blockDim.x) {
    const float4 v = project4(V, ldq, ncol, q, hf, w[q]);
    w[q] = v;
    n1 += double(dot4(v, v));
  }
  n1 = block_sum0(n1, sp);  // and every thread's rows of w are written
  __syncthreads();
  if (tid == 0) part1[int64_t(ncol) * nb + b] = n1;
  partial_dots(a, ncol, q0, q1, b, nb, part1, sp);
  ar_barrier(blockIdx, gridDim, a.bar, a.err);
  reduce_parts(blockIdx, gridDim, part1, ncol + 1, hp);
  for (int c = tid; c < ncol; c += blockDim.x) {
    ht[c] += hp[c];
    hf[c] = float(hp[c]);
  }
  double n2 = hp[ncol];
  for (int c = 0; c < ncol; ++c) n2 = fma(-hp[c], hp[c], n2);
  __syncthreads();
  const bool direct = n2 > 0.75 * hp[ncol];  // the same value in every block
  if (!direct) {
    double s = 0.0;
    for (int64_t q = q0 + tid; q < q1; q += blockDim.x) {
      const float4 v = project4(V, ldq, ncol, q, hf, w[q]);
      w[q] = v;
      s += double(dot4(v, v));
    }
    s = block_sum0(s, sp);
    if (tid == 0) part0[b] = s;  // every block is past its reads of part0
    ar_barrier(blockIdx, gridDim, a.bar, a.err);
    reduce_parts(blockIdx, gridDim, part0, 1, hp);
    n2 = hp[0];
  }
  const double nrm = sqrt(n2);
  const float inv = nrm > 0.0 ? float(1.0 / nrm) : 0.f;
  // Block 0 leaves its rows to the other warps while warp 0 runs the Givens
  // update: one thread over shared-memory copies of the column (ht) and of
  // the previous rotations, a chain of dependent accesses.
  const bool givens = b == 0 && tid < 32;
  if (!givens) {
    const int64_t t0 = b == 0 ? tid - 32 : tid, dt = b == 0 ? blockDim.x - 32 : blockDim.x;
    for (int64_t q = q0 + t0; q < q1; q += dt) {
      float4 v = direct ? project4(V, ldq, ncol, q, hf, w[q]) : w[q];
      v.x *= inv;
      v.y *= inv;
      v.z *= inv;
      v.w *= inv;
      Vn[q] = v;
      put_x4(a, 4 * q, v);
    }
    return;
  }
  double* sl = cl + m;
  for (int i = tid; i < j; i += 32) {
    cl[i] = a.cs[i];
    sl[i] = a.sn[i];
  }
  __syncwarp();
  if (tid == 0) {
    ht[j + 1] = nrm;
    for (int i = 0; i < j; ++i) {  // previous rotations
      const double x = ht[i], y = ht[i + 1];
      ht[i] = cl[i] * x + sl[i] * y;
      ht[i + 1] = -sl[i] * x + cl[i] * y;
    }
    const double x = ht[j], y = ht[j + 1];
    const double rho = sqrt(x * x + y * y);
    const double c0 = rho > 0.0 ? x / rho : 1.0, s0 = rho > 0.0 ? y / rho : 0.0;
    a.cs[j] = c0;
    a.sn[j] = s0;
    ht[j] = rho;
    ht[j + 1] = 0.0;
    a.g[j + 1] = -s0 * a.g[j];
    a.g[j] = c0 * a.g[j];
    a.scal[0] = fabs(a.g[j + 1]);
    a.scal[1] = nrm;
    if (a.scal[0] <= a.scal[4]) {
      a.stop[1] = j;
      __threadfence();
      a.stop[0] = 1;
    }
  }
  __syncwarp();
  double* Hj = a.H + int64_t(m + 1) * j;
  for (int c = tid; c <= j + 1; c += 32) Hj[c] = ht[c];
}
TTG_COOP_KERNEL(k_arnoldi, AR_THREADS, COOP_CTAS);

// V(:,0) = r / ||r||, g = [||r||, 0, ...]; scal[2] = ||r||.  On the first
// restart (first != 0) r is the right-hand side: scal[3] = ||r||.  The stop
// threshold reltol * scal[3] goes to scal[4]; a residual already below it
// (or zero) raises the stop flag with step -1, so the queued steps return at
// once and the host learns it at its next read of the flags.  The rows of V
// and w beyond sz are cleared here.
TTG_BODY(k_ar_init)(TTG_BLOCK, ArArgs a, const float* r, int first) {
  __shared__ double red[AR_WARPS];
  __shared__ double tot[1];
  const int64_t b = blockIdx.x, nb = gridDim.x;
  const int64_t q0 = quad_at(a, b, nb), q1 = quad_at(a, b + 1, nb);
  auto load = [&](int64_t q) {  // r has sz entries
    const int64_t i = 4 * q;
    float4 v;
    v.x = r[i];
    v.y = i + 1 < a.sz ? r[i + 1] : 0.f;
    v.z = i + 2 < a.sz ? r[i + 2] : 0.f;
    v.w = i + 3 < a.sz ? r[i + 3] : 0.f;
    return v;
  };
  double s = 0.0;
  for (int64_t q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
    const float4 v = load(q);
    s += double(dot4(v, v));
  }
  s = block_sum0(s, red);
  if (threadIdx.x == 0) a.part[b] = s;
  ar_barrier(blockIdx, gridDim, a.bar, a.err);
  reduce_parts(blockIdx, gridDim, a.part, 1, tot);
  const double beta = sqrt(tot[0]);
  const float inv = beta > 0.0 ? float(1.0 / beta) : 0.f;
  for (int64_t q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
    float4 v = load(q);
    v.x *= inv;
    v.y *= inv;
    v.z *= inv;
    v.w *= inv;
    reinterpret_cast<float4*>(a.V)[q] = v;
    put_x4(a, 4 * q, v);
  }
  if (b == 0 && threadIdx.x == 0) {
    for (int64_t i = a.sz; i < a.ldv; ++i) a.w[i] = 0.f;
    for (int k = 0; k <= a.m; ++k) a.g[k] = 0.0;
    a.g[0] = beta;
    a.scal[2] = beta;
    a.scal[0] = beta;
    if (first) a.scal[3] = beta;
    const double thr = a.reltol * a.scal[3];
    a.scal[4] = thr;
    if (beta <= thr || beta == 0.0) {
      a.stop[1] = -1;
      __threadfence();
      a.stop[0] = 1;
    }
  }
}
TTG_COOP_KERNEL(k_ar_init, AR_THREADS, COOP_CTAS);

// x += V(:, 0:k) y with H(0:k,0:k) y = g(0:k) (upper triangular after Givens).
TTG_BODY(k_ar_update)(TTG_BLOCK, ArArgs a, int k, float* x) {
  pdl_begin();
  // y (m+1), then H's leading k x k block (ld k) and g (k), copied in
  // parallel so that the back-substitution on one thread reads shared memory.
  extern __shared__ double y[];
  double* Hs = y + (a.m + 1);
  double* gs = Hs + int64_t(k) * k;
  for (int e = threadIdx.x; e < k * k; e += blockDim.x) {
    const int row = e % k, col = e / k;
    Hs[e] = a.H[row + int64_t(a.m + 1) * col];
  }
  for (int e = threadIdx.x; e < k; e += blockDim.x) gs[e] = a.g[e];
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int row = k - 1; row >= 0; --row) {
      double v = gs[row];
      for (int col = row + 1; col < k; ++col) v -= Hs[row + k * col] * y[col];
      const double d = Hs[row + k * row];
      y[row] = d != 0.0 ? v / d : 0.0;
    }
  }
  __syncthreads();
  float* yf = reinterpret_cast<float*>(Hs);  // H is done with
  for (int e = threadIdx.x; e < k; e += blockDim.x) yf[e] = -float(y[e]);
  __syncthreads();
  const float4* V = reinterpret_cast<const float4*>(a.V);
  AR_LOOP(q, a.ldv / 4) {
    const int64_t i = 4 * q;
    const float4 s = project4(V, a.ldv / 4, k, q, yf, make_float4(0.f, 0.f, 0.f, 0.f));
    x[i] += s.x;
    if (i + 1 < a.sz) x[i + 1] += s.y;
    if (i + 2 < a.sz) x[i + 2] += s.z;
    if (i + 3 < a.sz) x[i + 3] += s.w;
  }
}
TTG_KERNEL(k_ar_update, AR_THREADS);

// Centre block-Jacobi on vectors in the reversed layout v[k + rx2 (j + n i)]:
// out[k, j, i] = sum_m J[i, j, m, k] v[k, m, i] with the FP64 blocks J of
// jac_gen_c_f64 (natural layout J[i + rx1 (j + n (m + n k))]).  To BF16 in
// the matvec's K-major operand layout (xb, ld ldx) or to FP32 (xf).
TTG_BODY(k_prec_rev)(TTG_BLOCK, int64_t rx1, int64_t n, int64_t rx2, const double* __restrict__ J,
                           const float* __restrict__ v, __nv_bfloat16* __restrict__ xb,
                           int64_t ldx, float* __restrict__ xf, const int* skip) {
  pdl_begin();
  if (skip && *skip) return;
  const int64_t total = rx1 * n * rx2;
  AR_LOOP(e, total) {
    const int64_t k = e % rx2, j = (e / rx2) % n, i = e / (rx2 * n);
    const double* Jr = J + i + rx1 * j + rx1 * n * n * k;
    const float* vr = v + k + rx2 * n * i;
    double s = 0.0;
    for (int64_t m = 0; m < n; ++m) s += Jr[rx1 * n * m] * double(vr[rx2 * m]);
    if (xb)
      xb[k + ldx * (j + n * i)] = __float2bfloat16_rn(float(s));
    else
      xf[e] = float(s);
  }
}
TTG_KERNEL(k_prec_rev, 0);

// r = b - y (FP32)
TTG_BODY(k_sub_f32)(TTG_BLOCK, int64_t n, const float* b, const float* y, float* r) {
  pdl_begin();
  AR_LOOP(i, n) r[i] = b[i] - y[i];
}
TTG_KERNEL(k_sub_f32, 0);

struct Gmres32 {
  Context* c;
  int64_t sz;
  int m;
  int blocks;
  DBuf<float> V, w, r;
  DBuf<double> small, part;
  DBuf<unsigned> bar;
  DBuf<int> stop;
  ArArgs a{};

  Gmres32(Context* cc, int64_t n, int restart) : c(cc), sz(n), m(restart) {
    const int64_t ldv = (sz + 3) & ~int64_t(3);
    V.reset(c, size_t(ldv) * (m + 1));
    w.reset(c, ldv);
    r.reset(c, sz);
    small.reset(c, size_t(m + 1) * m + 2 * m + (m + 1) + 8);
    int occ = 0;
    occ = max_active_blocks(k_arnoldi.fn(), AR_THREADS, arnoldi_smem());
    if (occ < 1) occ = 1;
    const int64_t want = (sz + AR_ROWS - 1) / AR_ROWS;
    const int64_t cap = int64_t(c->num_sms) * std::min(occ, c->coop_ctas);
    blocks = int(std::max<int64_t>(1, std::min(want, cap)));
    part.reset(c, size_t(2) * (m + 2) * blocks);
    bar.reset(c, 4);
    memset_async(c, bar.p(), 0, 4 * sizeof(unsigned));
    a.sz = sz;
    a.ldv = ldv;
    a.m = m;
    a.V = V.p();
    a.w = w.p();
    a.H = small.p();
    a.cs = a.H + size_t(m + 1) * m;
    a.sn = a.cs + m;
    a.g = a.sn + m;
    a.scal = a.g + (m + 1);
    a.part = part.p();
    a.bar = bar.p();
    a.err = c->d_err + 2;
    stop.reset(c, 4);
    a.stop = stop.p();
    a.reltol = 0.0;
    a.X = nullptr;
  }

  size_t arnoldi_smem() const {
    return sizeof(double) * arnoldi_doubles(m) + sizeof(float) * (m + 1);
  }

  // Right-preconditioned operand: X = bf16(P v) for the centre block-Jacobi
  // blocks J (FP64, natural layout), v in the reversed layout.
  void prec_x(MixedOp& op, const double* J, const float* v) {
    launch(c, k_prec_rev, blocks, AR_THREADS, 0, op.d.rx1, op.d.n, op.d.rx2, J, v, op.X.p(),
           op.ldx, static_cast<float*>(nullptr), c->skip);
    TTG_CHECK_LAUNCH();
  }

  // Solve B x = b approximately (B P y = b, x = y, when J is given: the
  // caller applies P to x); x (FP32, zeroed here); returns Krylov steps.
  int64_t solve(MixedOp& op, const float* b, float* x, double reltol, int64_t max_restarts,
                const double* J = nullptr) {
    int64_t steps = 0;
    a.X = J ? nullptr : op.X.p();
    a.rx2 = int(op.d.rx2);
    a.ldx = int(op.ldx);
    a.reltol = reltol;
    memset_async(c, x, 0, sizeof(float) * sz);
    for (int64_t it = 0; it < max_restarts; ++it) {
      const float* rr = b;
      if (it > 0) {
        if (J) {
          prec_x(op, J, x);
          op.apply_converted(c, w.p());
        } else {
          op.apply(c, x, w.p());
        }
        launch(c, k_sub_f32, blocks, AR_THREADS, 0, sz, b, w.p(), r.p());
        rr = r.p();
      }
      memset_async(c, stop.p(), 0, 2 * sizeof(int));
      const int first = it == 0 ? 1 : 0;
      launch(c, k_ar_init, blocks, AR_THREADS, 0, a, rr, first);
      // Steps queued in chunks; k_arnoldi (or k_ar_init, for a residual
      // already below the threshold) raises the stop flag and later queued
      // kernels return at once (see gmres.cu).  The first chunk is the step
      // count of the context's previous inner solve, later ones half of it,
      // so that most solves need one or two reads of the flags.  Matvecs
      // queued past the converged step are taken out of the counters and
      // timings afterwards.
      int j = 0, queued = 0;
      const int hint = std::max(3, c->krylov_hint);
      int chunk = std::min(m, hint);
      bool conv = false, at_start = false;
      std::vector<uint64_t> seqs;
      SkipGuard guard(c, stop.p());
      while (j < m) {
        const int jend = std::min(m, j + chunk);
        for (int jj = j; jj < jend; ++jj) {
          const int jv = jj;
          seqs.push_back(c->ev_seq);
          if (J) prec_x(op, J, V.p() + int64_t(jj) * a.ldv);  // X = bf16(P V(:, jv))
          op.apply_converted(c, w.p());  // X holds V(:, jv) (k_ar_init / k_arnoldi)
          launch(c, k_arnoldi, blocks, AR_THREADS, arnoldi_smem(), a, jv);
        }
        queued = jend;
        int flag[2];
        read_device(c, flag, stop.p(), sizeof(flag));
        if (flag[0]) {
          if (flag[1] < 0) {
            at_start = true;
          } else {
            conv = true;
            j = flag[1];
          }
          break;
        }
        j = jend;
        chunk = std::max(3, hint / 2);
      }
      guard.release();
      {
        const int done = at_start ? 0 : (conv ? j + 1 : m);
        const int skipped = queued - done;
        if (skipped > 0) {
          const double fl = op.d.flops();
          c->matvecs -= skipped;
          c->matvec_flops -= int64_t(fl) * skipped;
          c->mv_count[1] -= skipped;
          c->mv_flops[1] -= fl * skipped;
          c->mv_bytes_lp -= op.bytes_per_matvec() * skipped;
          // three recorded GEMMs per queued matvec (grouped: three-launch form)
          if (c->rec) rec_retract_flop(c->rec, fl * skipped, 3 * int64_t(skipped));
          if (c->time_matvec) c->ev_void(seqs[done], c->ev_seq);
        }
      }
      if (at_start) break;  // nothing left to reduce: x stays as it is
      const int k = conv ? j + 1 : m;
      steps += k;
      c->krylov_hint = k;
      launch(c, k_ar_update, blocks, AR_THREADS,
             sizeof(double) * (size_t(m + 1) + size_t(k) * k + size_t(k)), a, k, x);
      TTG_CHECK_LAUNCH();
      if (conv) break;
    }
    return steps;
  }
};

}  // namespace

LocalSolveResult local_solve_mixed(Context* c, const MvDims& d, const double* Phi1,
                                   const double* A, const double* Phi2, const double* rhs,
                                   const double* dres, double nres, double nrhs, double tol,
                                   const double* sol_prev, int64_t nrestart, int64_t niters,
                                   double* sol, double* bsol_out, int prec) {
  LocalSolveResult out;
  const int64_t sz = d.in_size();
  TTG_REQUIRE(prec == 0 || prec == 1,
              "the mixed-precision local solve has the 'cjacobi' preconditioner only");
  // Centre block-Jacobi blocks (FP64) for the right preconditioning of the
  // low-precision Krylov solves and of the FP64 fallback.
  DBuf<double> J, pw;
  if (prec == 1) {
    J.reset(c, jac_size(1, d.rx1, d.n, d.rx2));
    pw.reset(c, sz);
    jac_gen_c_f64(c, d.rx1, d.n, d.rx2, d.ra1, d.ra2, Phi1, A, Phi2, J.p());
  }
  if (nrestart > sz) nrestart = sz;
  TTG_REQUIRE(nrestart <= 1024, "mixed solve: restart length %lld too large", (long long)nrestart);
  MixedOp op;
  op.prepare(c, d, Phi1, A, Phi2);
  Gmres32 gm(c, sz, int(nrestart));
  DBuf<double> t1(c, d.t1_size()), t2(c, d.t2_size()), r64(c, sz), prev(c, sz), s(c, 2);
  DBuf<float> rrev(c, sz), dx(c, sz), dxp;
  if (prec == 1) dxp.reset(c, sz);
  copy_f64(c, sz, sol_prev, sol);
  auto residual = [&]() -> double {
    if (bsol_out) {
      local_matvec_f64(c, d, Phi1, A, Phi2, sol, bsol_out, t1.p(), t2.p());
      copy_f64(c, sz, bsol_out, r64.p());
    } else {
      local_matvec_f64(c, d, Phi1, A, Phi2, sol, r64.p(), t1.p(), t2.p());
    }
    out.matvecs_fp64++;
    axpby_f64(c, sz, 1.0, rhs, -1.0, r64.p());
    dot_f64(c, sz, r64.p(), nullptr, s.p(), true);
    double h;
    read_scalars(c, s.p(), &h, 1);
    return h;
  };
  const double target = tol * nrhs;
  copy_f64(c, sz, dres, r64.p());
  double nr = nres;
  bool r64_valid = true;  // r64 = rhs - B sol for the current sol
  for (int outer = 0; outer < MAX_OUTER; ++outer) {
    if (!(nr > target)) break;
    nat_to_rev(c, d.rx1, d.n, d.rx2, r64.p(), rrev.p(), 1.0 / nr);
    const double reltol = std::max(target / nr, INNER_TOL);
    out.iters += gm.solve(op, rrev.p(), dx.p(), reltol, niters, prec ? J.p() : nullptr);
    copy_f64(c, sz, sol, prev.p());
    if (prec) {  // the correction is P y
      launch(c, k_prec_rev, gm.blocks, AR_THREADS, 0, d.rx1, d.n, d.rx2, J.p(), dx.p(),
             static_cast<__nv_bfloat16*>(nullptr), int64_t(0), dxp.p(),
             static_cast<const int*>(nullptr));
      TTG_CHECK_LAUNCH();
      rev_to_nat_add(c, d.rx1, d.n, d.rx2, dxp.p(), sol, nr);
    } else {
      rev_to_nat_add(c, d.rx1, d.n, d.rx2, dx.p(), sol, nr);
    }
    const double nr_new = residual();
    out.have_bsol = bsol_out != nullptr;
    if (!(nr_new < nr)) {  // no progress: keep the better iterate and stop
      copy_f64(c, sz, prev.p(), sol);
      out.have_bsol = false;
      r64_valid = false;
      break;
    }
    const bool stagnating = nr_new > 0.5 * nr;
    nr = nr_new;
    if (stagnating) break;
  }
  if (nr > target) {
    // The low-precision corrections stopped paying (the local operator is
    // too ill-conditioned for BF16 products): finish with the FP64
    // Householder GMRES of the FP64 path on the remaining residual, so the
    // local solve meets the same tolerance as there.
    if (!r64_valid) nr = residual();
    if (nr > target) {
      DBuf<double> dsol(c, sz);
      auto mv = [&](const double* x, double* y) {
        if (prec == 1) {  // B P x
          jac_apply_c_f64(c, d.rx1, d.n, d.rx2, J.p(), x, pw.p());
          local_matvec_f64(c, d, Phi1, A, Phi2, pw.p(), y, t1.p(), t2.p());
        } else {
          local_matvec_f64(c, d, Phi1, A, Phi2, x, y, t1.p(), t2.p());
        }
      };
      GmresResult g = gmres_hh_f64(c, mv, r64.p(), sz, nrestart, target / nr, niters, dsol.p());
      if (prec == 1) {
        jac_apply_c_f64(c, d.rx1, d.n, d.rx2, J.p(), dsol.p(), pw.p());
        copy_f64(c, sz, pw.p(), dsol.p());
      }
      axpby_f64(c, sz, 1.0, dsol.p(), 1.0, sol);
      out.iters += g.iters;
      out.matvecs_fp64 += g.matvecs;
      out.have_bsol = false;
      c->mixed_fallbacks += 1;
    }
  }
  // Bounded-wait timeouts are reported through the context error slots 1-2,
  // checked by the caller once its sequence is done.
  out.matvecs = out.iters;
  return out;
}

namespace {
__global__ void k_selftest_ar_barrier(unsigned* bar, int* flag, long long limit) {
  if (blockIdx.x != 0) return;
  ar_barrier(blockIdx, gridDim, bar, flag, limit);
}
}  // namespace

// Self-test of the bounded barrier of the Arnoldi kernels: block 1 never
// arrives; block 0 gives up after `limit` polls and raises *flag.
void selftest_wait_arnoldi(Context* c, int* flag, long long limit) {
  DBuf<unsigned> bar(c, 2);
  TTG_CUDA(cudaMemsetAsync(bar.p(), 0, 2 * sizeof(unsigned), c->stream));
  k_selftest_ar_barrier<<<2, 32, 0, c->stream>>>(bar.p(), flag, limit);
  TTG_CHECK_LAUNCH();
  sync(c);
}

}  // namespace ttg
