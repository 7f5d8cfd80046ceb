// Single-CTA FP64 dense factorizations for the small matrices of the AMEn
// and rounding sweeps (replacing library calls whose host-side sequencing
// cost milliseconds on 64x64 inputs):
//
//   k_jacobi_svd :     one-sided block Jacobi SVD of a square n x n matrix,
//                      n <= 96, in one CTA: A and V in shared memory, blocks
//                      of eight columns rotated by 16 x 16 Gram matrices.
//   k_jacobi_cluster : the same for n <= 256 on a cluster, a pair of blocks a
//                      CTA; k_jacobi_coop column pairs over the grid beyond.
//   k_house_qr_blk :   Householder QR (LAPACK sign convention: beta =
//                      -sign(alpha) ||x||, as geqrf/orgqr and MATLAB's qr(A,0))
//                      of an m x n matrix in shared memory, in panels of
//                      eight columns; forms the thin Q and R.  k_house_qr, a
//                      column at a time, takes the shapes of one or two
//                      reflectors, of three with up to 256 rows, and those
//                      that fit only without the panel's workspace.
// Singular values descend.  One launch each, no host round trip.
#include <cmath>
#include <cstdlib>

#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "dmma.cuh"
#include "group.cuh"
#include "small_dense.h"

namespace ttg {

namespace {

constexpr int SD_THREADS = 1024;
constexpr int SD_WARPS = SD_THREADS / 32;
constexpr size_t SMEM_LIMIT = 200 * 1024;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Column index of slot k in round r of a round-robin tournament on ne (even)
// players: slot 0 is fixed, the others rotate.  k - 1 + r < 2 (ne - 1), so a
// conditional subtraction replaces the modulo.
__device__ __forceinline__ int rr_player(int k, int r, int ne) {
  int x = k - 1 + r;
  if (x >= ne - 1) x -= ne - 1;
  return k == 0 ? 0 : 1 + x;
}

// ---------------------------------------------------------------------------
// Pieces of the block Jacobi SVDs
// ---------------------------------------------------------------------------

constexpr int JK_MAX_CS = 16;          // CTAs of a cluster
constexpr int JK_W = 8;                // columns of a block
constexpr int JK_COLS = 2 * JK_W;      // columns of a CTA
constexpr int JK_MAX_N = JK_MAX_CS * JK_COLS;
constexpr int JK_THREADS = 512;
constexpr int JK_WARPS = JK_THREADS / 32;
constexpr int JK_GP = JK_COLS + 1;     // pitch of the Gram matrix
constexpr int JK_JP = JK_COLS + 4;     // pitch of J (mma operand: 4 mod 16)

// Rows of a column's A (or V) part, and column pitches in global and shared
// memory (the latter 4 mod 16, so that mma fragments meet no bank twice).
__host__ __device__ __forceinline__ int jk_rows(int n) { return (n + 7) & ~7; }
__host__ __device__ __forceinline__ int jk_pitch(int n) {
  return ((2 * jk_rows(n) + 15) & ~15) + 4;
}
int jk_blocks(int64_t n) { return int((n + JK_COLS - 1) / JK_COLS) * 2; }
int64_t jk_work(int64_t n) {  // columns, then the column norms
  return int64_t(jk_blocks(n)) * JK_W * (2 * jk_rows(int(n)) + 1);
}
size_t jk_smem(int64_t n) {
  return sizeof(double) * (size_t(JK_COLS) * jk_pitch(int(n)) + JK_WARPS * 192 + JK_COLS * JK_GP +
                           JK_COLS * JK_JP);
}

// Blocks of CTA c in round r of a tournament on nb (even) blocks: block nb - 1
// is fixed and meets r, the others pair as p + q = 2 r (mod nb - 1).
__device__ __forceinline__ void jk_pair(int c, int r, int nb, int& p, int& q) {
  const int m = nb - 1;
  if (c == 0) {
    p = r;
    q = m;
    return;
  }
  p = r + c;
  if (p >= m) p -= m;
  q = r - c;
  if (q < 0) q += m;
}

// Cosine and sine of the rotation that makes a pair orthogonal, the smaller of
// the two angles: with dd = be - al, g = 2 ga (scaled by the exponent of al + be)
// and h = hypot(dd, g), c = sqrt((1 + |dd| / h) / 2) and s = |g| / (2 h c) with the
// sign of dd g: two reciprocal roots, where the tangent takes a root, a quotient
// and a reciprocal root.  Both are then multiplied by 1 / sqrt(c^2 + s^2): a bias
// of 1e-16 in c^2 + s^2 adds up over a sweep's thousands of rotations.
// The angle takes double precision throughout: from single precision, the 1e-7
// of a pair's inner product that it leaves comes to rest below the stopping
// threshold in the last sweep, and the left factors of graded matrices lose
// 10-45% of their orthogonality.
__device__ __forceinline__ void jk_rotation(double al, double be, double ga, double& c,
                                            double& s) {
  const double dd = be - al, gg = 2.0 * ga;
  // 2^-e for the exponent e of al + be (2^-1022 at the top of the range)
  const int field = max(0x7fe00000 - (__double2hiint(al + be) & 0x7ff00000), 0x00100000);
  const double scale = __hiloint2double(field, 0);
  const double x = fabs(dd) * scale, y = fabs(gg) * scale;
  // (a pair of zero columns keeps clear of rsqrt's special cases, which take a
  // call: 18% of an SVD whose last block is padded)
  const double rh = rsqrt(fmax(fma(x, x, y * y), 1e-200));
  const double v = fma(0.5 * x, rh, 0.5);  // c^2
  const double rv = rsqrt(v);
  const double c0 = v * rv, s0 = 0.5 * y * rh * rv;
  const double d = fma(s0, s0, fma(c0, c0, -1.0));  // some 1e-16
  c = fma(-0.5 * c0, d, c0);
  s = fma(-0.5 * s0, d, s0);
  if ((dd >= 0.0) != (gg > 0.0) && dd != 0.0) s = -s;
}

// The rotations of a round on the Gram matrix sG of a block pair, by one warp,
// collected in sJ (the identity at the start): eight disjoint pairs per step,
// those across the two blocks in eight steps, or all 120 in fifteen.  Pairs
// within the tolerance (cosine squared at most tol2) stay.  Returns whether
// any pair was rotated.
__device__ __forceinline__ int jk_rotate(double* sG, double* sJ, bool all, double tol2) {
  const int lane = threadIdx.x & 31;
  const int steps = all ? JK_COLS - 1 : JK_W;
  int any = 0;
  for (int ir = 0; ir < steps; ++ir) {
    auto pair = [&](int k, int& p, int& q) {
      if (all) {
        p = rr_player(k, ir, JK_COLS);
        q = rr_player(JK_COLS - 1 - k, ir, JK_COLS);
      } else {
        p = k;
        q = JK_W + ((k + ir) & (JK_W - 1));
      }
    };
    int p, q;
    pair(lane & 7, p, q);
    const double al = sG[p * JK_GP + p], be = sG[q * JK_GP + q], ga = sG[p * JK_GP + q];
    // the lane's 2 x 2 blocks of G: pair a by pairs b and b + 4; its rows of J
    const int a = lane >> 2;
    int pa, qa, pb[2], qb[2];
    pair(a, pa, qa);
    pair(lane & 3, pb[0], qb[0]);
    pair((lane & 3) + 4, pb[1], qb[1]);
    double x[2][4], jp[4], jq[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      x[h][0] = sG[pa * JK_GP + pb[h]];
      x[h][1] = sG[pa * JK_GP + qb[h]];
      x[h][2] = sG[qa * JK_GP + pb[h]];
      x[h][3] = sG[qa * JK_GP + qb[h]];
    }
    double* row = sJ + (lane & 3) * JK_JP;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      jp[h] = row[4 * h * JK_JP + pa];
      jq[h] = row[4 * h * JK_JP + qa];
    }
    double c, s;
    jk_rotation(al, be, ga, c, s);
    const double ab = al * be;
    const bool rot = ab != 0.0 && ga * ga > tol2 * ab;
    if (!rot) {
      c = 1.0;
      s = 0.0;
    }
    any |= __any_sync(0xffffffffu, rot);
    const double ca = __shfl_sync(0xffffffffu, c, a), sa = __shfl_sync(0xffffffffu, s, a);
    // columns p, q <- c p - s q, s p + c q, on both sides of G
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double cb = __shfl_sync(0xffffffffu, c, (lane & 3) + 4 * h);
      const double sb = __shfl_sync(0xffffffffu, s, (lane & 3) + 4 * h);
      const double y00 = fma(cb, x[h][0], -sb * x[h][1]), y01 = fma(sb, x[h][0], cb * x[h][1]);
      const double y10 = fma(cb, x[h][2], -sb * x[h][3]), y11 = fma(sb, x[h][2], cb * x[h][3]);
      sG[pa * JK_GP + pb[h]] = fma(ca, y00, -sa * y10);
      sG[pa * JK_GP + qb[h]] = fma(ca, y01, -sa * y11);
      sG[qa * JK_GP + pb[h]] = fma(sa, y00, ca * y10);
      sG[qa * JK_GP + qb[h]] = fma(sa, y01, ca * y11);
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      row[4 * h * JK_JP + pa] = fma(ca, jp[h], -sa * jq[h]);
      row[4 * h * JK_JP + qa] = fma(sa, jp[h], ca * jq[h]);
    }
    __syncwarp();
  }
  return any;
}

// ---------------------------------------------------------------------------
// Block Jacobi SVD in one CTA, for n <= JS_MAX_N: the columns, each A over V,
// in shared memory in blocks of 8.  A round of a round-robin tournament on the
// blocks takes all block pairs at once: the Gram matrix of each pair's 16
// columns of A (mma.m8n8k4, its K split over the warps of the pair), the
// rotations on it by one warp per pair (jk_rotate: the 64 pairs across the
// blocks, in a sweep's first round all 120), and [A; V] J (mma).  A rotation on
// the Gram matrix is that of one-sided Jacobi on the columns (al = |a_p|^2, be
// = |a_q|^2, ga = <a_p, a_q>), whose entries round relative to the columns'
// norms; each round forms the matrices anew from the columns.  A sweep that
// rotates no pair ends the iteration (|ga| <= 4 eps sqrt(al be) for all).
// Bound by the chain of rotation steps, about 700 cycles each, n of them per
// sweep where one pair per warp took n barriers and as many passes over the
// columns.  Triangular factors (mean of six): 0.066 ms for 0.107 at n = 16, 0.244
// for 0.318 at 33, 0.264 for 0.547 at 47.
// Status: *err = 5 if the sweep limit is reached.
// ---------------------------------------------------------------------------

constexpr int JS_MAX_N = 96;

size_t js_smem(int64_t n) {
  const int pairs = jk_blocks(n) / 2;
  return sizeof(double) * (size_t(jk_blocks(n)) * JK_W * jk_pitch(int(n)) + JK_WARPS * 192 +
                           size_t(pairs) * JK_COLS * (JK_GP + JK_JP));
}

TTG_BODY(k_jacobi_svd)(TTG_BLOCK, int n, const double* __restrict__ Ain, int lda,
                       double* __restrict__ U, double* __restrict__ S, double* __restrict__ VT,
                       int trans, int* err, int max_sweeps) {
  pdl_begin();
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_any[JS_MAX_N / JK_COLS], s_found;
  const int np = jk_rows(n), ldx = 2 * np, P = jk_pitch(n);
  const int nb = 2 * ((n + JK_COLS - 1) / JK_COLS), pairs = nb / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  double* sX = sm;                          // nb * 8 columns of A over V
  double* sP = sX + nb * JK_W * P;          // partial Gram matrices of the warps
  double* sG = sP + JK_WARPS * 192;         // per pair
  double* sJ = sG + pairs * JK_COLS * JK_GP;
  for (int col = warp; col < nb * JK_W; col += JK_WARPS)
    for (int i = lane; i < ldx; i += 32) {
      double v = 0.0;
      if (col < n) {
        if (i < n)
          v = trans ? Ain[col + int64_t(i) * lda] : Ain[i + int64_t(col) * lda];
        else if (i >= np)
          v = i - np == col ? 1.0 : 0.0;
      }
      sX[col * P + i] = v;
    }
  const double tol = 4.0 * 2.220446049250313e-16, tol2 = tol * tol;
  const int wpp = JK_WARPS / pairs;  // warps per pair in the Gram products
  int sweep = 0;
  for (sweep = 0; sweep < max_sweeps; ++sweep) {
    int found = 0;
    for (int r = 0; r < nb - 1; ++r) {
      __syncthreads();  // columns of the previous round are written
      if (warp < wpp * pairs) {
        int bp, bq;
        jk_pair(warp / wpp, r, nb, bp, bq);
        const double* x0 = sX + (bp * JK_W + g) * P + t;
        const double* x1 = sX + (bq * JK_W + g) * P + t;
        double acc[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        for (int k4 = warp % wpp; k4 < np / 4; k4 += wpp) {
          const double u = x0[4 * k4], v = x1[4 * k4];
          dmma(acc[0][0], acc[0][1], u, u);
          dmma(acc[1][0], acc[1][1], u, v);
          dmma(acc[2][0], acc[2][1], v, v);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          sP[warp * 192 + q * 64 + g * 8 + 2 * t] = acc[q][0];
          sP[warp * 192 + q * 64 + g * 8 + 2 * t + 1] = acc[q][1];
        }
      }
      __syncthreads();
      for (int e = tid; e < pairs * 192; e += JK_THREADS) {
        const int pr = e / 192, el = e % 192;
        double v = 0.0;
        for (int w = 0; w < wpp; ++w) v += sP[(pr * wpp + w) * 192 + el];
        const int q = el / 64, i = (el >> 3) & 7, j = el & 7;
        const int row = q == 2 ? 8 + i : i, col = q == 0 ? j : 8 + j;
        double* G = sG + pr * JK_COLS * JK_GP;
        if (q == 1 || i <= j) G[row * JK_GP + col] = G[col * JK_GP + row] = v;
      }
      for (int e = tid; e < pairs * JK_COLS * JK_COLS; e += JK_THREADS) {
        const int pr = e / (JK_COLS * JK_COLS), i = (e / JK_COLS) % JK_COLS, j = e % JK_COLS;
        sJ[pr * JK_COLS * JK_JP + i * JK_JP + j] = i == j ? 1.0 : 0.0;
      }
      __syncthreads();
      if (warp < pairs) {
        const int any = jk_rotate(sG + warp * JK_COLS * JK_GP, sJ + warp * JK_COLS * JK_JP, r == 0,
                                  tol2);
        found |= any;
        if (lane == 0) s_any[warp] = any;
      }
      __syncthreads();
      const int mts = ldx / 8;
      for (int u = warp; u < pairs * mts; u += JK_WARPS) {
        const int pr = u / mts, mt = u % mts;
        if (!s_any[pr]) continue;
        int bp, bq;
        jk_pair(pr, r, nb, bp, bq);
        const double* J = sJ + pr * JK_COLS * JK_JP;
        double* xp = sX + bp * JK_W * P + 8 * mt + g;
        double* xq = sX + bq * JK_W * P + 8 * mt + g;
        double o[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double x = k < 2 ? xp[(4 * k + t) * P] : xq[(4 * (k - 2) + t) * P];
          dmma(o[0][0], o[0][1], x, J[(4 * k + t) * JK_JP + g]);
          dmma(o[1][0], o[1][1], x, J[(4 * k + t) * JK_JP + 8 + g]);
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          xp[(2 * t + h) * P] = o[0][h];
          xq[(2 * t + h) * P] = o[1][h];
        }
      }
    }
    if (tid == 0) s_found = 0;
    __syncthreads();
    if (found && lane == 0) s_found = 1;
    __syncthreads();
    if (!s_found) break;
  }
  if (tid == 0 && sweep >= max_sweeps) atomicExch(err, 5);
  // Singular values = column norms, ranked descending (stable on index), and
  // the factors in that order.  With trans the rotated matrix is the transpose
  // of the input (X = In^T = Ux S Vx^T), so the input's factors swap: U = Vx,
  // VT = Ux^T.
  double* sn = sP;
  int* pos = reinterpret_cast<int*>(sn + n);
  for (int col = warp; col < n; col += JK_WARPS) {
    double v = 0.0;
    for (int i = lane; i < n; i += 32) v = fma(sX[col * P + i], sX[col * P + i], v);
    v = wsum(v);
    if (lane == 0) sn[col] = sqrt(v);
  }
  __syncthreads();
  for (int col = tid; col < n; col += JK_THREADS) {
    const double sj = sn[col];
    int before = 0;
    for (int k = 0; k < n; ++k) before += (sn[k] > sj) || (sn[k] == sj && k < col);
    S[before] = sj;
    pos[col] = before;
  }
  __syncthreads();
  for (int col = warp; col < n; col += JK_WARPS) {
    const double sj = sn[col];
    const int at = pos[col];
    for (int i = lane; i < n; i += 32) {
      const double ua = sj > 0.0 ? sX[col * P + i] / sj : (i == at ? 1.0 : 0.0);
      const double v = sX[col * P + np + i];
      U[i + int64_t(at) * n] = trans ? v : ua;
      VT[at + int64_t(i) * n] = trans ? ua : v;
    }
  }
}
TTG_KERNEL(k_jacobi_svd, JK_THREADS);


// Singular values = column norms of the rotated A, ranked descending
// (stable on index); U = A diag(1/s), VT = V^T in that order.  With trans the
// rotated matrix is the transpose of the input (X = In^T = Ux S Vx^T), so the
// input's factors swap: U = Vx, VT = Ux^T.  One CTA of SD_THREADS; sig: 2n
// doubles of scratch.
__device__ void jacobi_finish(int n, const double* A, const double* V, double* __restrict__ U,
                              double* __restrict__ S, double* __restrict__ VT, double* sig,
                              int trans) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j = warp; j < n; j += SD_WARPS) {
    const double* aj = A + int64_t(j) * n;
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += aj[i] * aj[i];
    s = wsum(s);
    if (lane == 0) sig[j] = sqrt(s);
  }
  __syncthreads();
  for (int j = tid; j < n; j += SD_THREADS) {
    const double sj = sig[j];
    int pos = 0;
    for (int k = 0; k < n; ++k) {
      const double sk = sig[k];
      pos += (sk > sj) || (sk == sj && k < j);
    }
    S[pos] = sj;
    sig[n + j] = double(pos);
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += SD_THREADS) {
    const int i = e % n, j = e / n;
    const int pos = int(sig[n + j]);
    const double sj = sig[j];
    const double ua = sj > 0.0 ? A[e] / sj : (i == pos ? 1.0 : 0.0);
    if (!trans) {
      U[i + int64_t(pos) * n] = ua;
      VT[pos + int64_t(i) * n] = V[e];
    } else {
      U[i + int64_t(pos) * n] = V[e];
      VT[pos + int64_t(i) * n] = ua;
    }
  }
}

// ---------------------------------------------------------------------------
// Grid-wide one-sided Jacobi SVD for matrices too large for one CTA's shared
// memory: one CTA per column pair of a round-robin round, a bounded grid
// barrier between rounds (cooperative launch).  The rotation of a pair is that of
// k_jacobi_svd, taken from the columns' own inner products by the tangent, with
// the same stopping rule.
// ---------------------------------------------------------------------------

constexpr int JC_THREADS = 256;
constexpr long long JC_SPIN_LIMIT = 1LL << 24;

__device__ void jc_barrier(TTG_BLOCK, unsigned* bar, int* err, long long limit = JC_SPIN_LIMIT) {
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
          atomicExch(err, 6);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// A (n x n work copy, ld n) and V (n x n) in global memory; offmax: three
// u64 slots holding the per-sweep maximum off-diagonal measure (bit pattern
// of a non-negative double).  *sweeps_out = sweeps run.
TTG_BODY(k_jacobi_coop)(TTG_BLOCK, int n, const double* __restrict__ Ain,
                                                           int lda, double* A, double* V,
                                                           unsigned* bar,
                                                           unsigned long long* offmax, int* err,
                                                           int* sweep_err, int trans,
                                                           int max_sweeps) {
  __shared__ double red[3][JC_THREADS / 32];
  __shared__ double s_rot[2];
  __shared__ int s_skip;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nn = int64_t(n) * n;
  for (int64_t e = blockIdx.x * int64_t(JC_THREADS) + tid; e < nn;
       e += int64_t(gridDim.x) * JC_THREADS) {
    const int64_t i = e % n, j = e / n;
    A[e] = trans ? Ain[j + i * lda] : Ain[i + j * lda];
    V[e] = (i == j) ? 1.0 : 0.0;
  }
  if (blockIdx.x == 0 && tid < 3) offmax[tid] = 0ull;
  jc_barrier(blockIdx, gridDim, bar, err);
  const int ne = (n + 1) & ~1;
  const double tol = 4.0 * 2.220446049250313e-16;
  int sweep = 0;
  for (sweep = 0; sweep < max_sweeps; ++sweep) {
    const int slot = sweep % 3;
    if (blockIdx.x == 0 && tid == 0) offmax[(sweep + 1) % 3] = 0ull;
    double off = 0.0;
    for (int r = 0; r < ne - 1; ++r) {
      for (int pr = blockIdx.x; pr < ne / 2; pr += gridDim.x) {
        int p = rr_player(pr, r, ne), q = rr_player(ne - 1 - pr, r, ne);
        if (p > q) {
          const int t = p;
          p = q;
          q = t;
        }
        if (q >= n) continue;  // dummy player (uniform in the CTA)
        double* ap = A + int64_t(p) * n;
        double* aq = A + int64_t(q) * n;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int i = tid; i < n; i += JC_THREADS) {
          const double x = ap[i], y = aq[i];
          al += x * x;
          be += y * y;
          ga += x * y;
        }
        al = wsum(al);
        be = wsum(be);
        ga = wsum(ga);
        if (lane == 0) {
          red[0][warp] = al;
          red[1][warp] = be;
          red[2][warp] = ga;
        }
        __syncthreads();
        if (tid == 0) {
          double a2 = 0.0, b2 = 0.0, g2 = 0.0;
          for (int w = 0; w < JC_THREADS / 32; ++w) {
            a2 += red[0][w];
            b2 += red[1][w];
            g2 += red[2][w];
          }
          const double nrm = sqrt(a2 * b2);
          if (nrm == 0.0 || fabs(g2) <= tol * nrm) {
            s_skip = 1;
          } else {
            s_skip = 0;
            off = fmax(off, fabs(g2) / nrm);
            const double zeta = (b2 - a2) / (2.0 * g2);
            const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
            const double cc = 1.0 / sqrt(1.0 + t * t);
            s_rot[0] = cc;
            s_rot[1] = cc * t;
          }
        }
        __syncthreads();
        if (!s_skip) {
          const double cc = s_rot[0], sn = s_rot[1];
          double* vp = V + int64_t(p) * n;
          double* vq = V + int64_t(q) * n;
          for (int i = tid; i < n; i += JC_THREADS) {
            const double x = ap[i], y = aq[i];
            ap[i] = cc * x - sn * y;
            aq[i] = sn * x + cc * y;
            const double vx = vp[i], vy = vq[i];
            vp[i] = cc * vx - sn * vy;
            vq[i] = sn * vx + cc * vy;
          }
        }
        __syncthreads();
      }
      jc_barrier(blockIdx, gridDim, bar, err);
    }
    if (tid == 0) atomicMax(offmax + slot, (unsigned long long)__double_as_longlong(off));
    jc_barrier(blockIdx, gridDim, bar, err);
    const double m = __longlong_as_double((long long)(*(volatile unsigned long long*)(offmax + slot)));
    if (m <= tol) break;
    if (*(volatile int*)err) break;
  }
  if (blockIdx.x == 0 && tid == 0 && sweep >= max_sweeps) atomicExch(sweep_err, 5);
}
TTG_COOP_KERNEL(k_jacobi_coop, JC_THREADS, -1);

// ---------------------------------------------------------------------------
// Block Jacobi SVD in one thread-block cluster, for n <= JK_MAX_N columns (the
// R factors of the rounding sweeps and of AMEn's truncations).  The columns,
// each A over V, fall into blocks of 8; a round of a round-robin tournament
// on the blocks gives every CTA one block pair.  A round takes
//   the Gram matrix of the pair's 16 columns of A (mma.m8n8k4, K split over
//   the warps),
//   the 8 x 8 cross pairs of the two blocks rotated on that matrix, one warp,
//   eight disjoint pairs at a time (in a sweep's first round all 120 pairs),
//   with the rotations collected in a 16 x 16 orthogonal J,
//   and [A; V] J for the 16 columns (mma), skipped when nothing rotated.
// The columns live in L2 (1 MB at n = 256) and are read at the start of a
// round and written at its end, with one hardware cluster barrier between:
// distributed shared memory moves 14 bytes per cycle and SM here, L2 four
// times that.  V arrives while the Gram matrix is rotated.
// A rotation on the Gram matrix is that of one-sided Jacobi on the columns
// (al = |a_p|^2, be = |a_q|^2, ga = <a_p, a_q>), whose entries round relative to
// the columns' norms; each round forms the matrix anew from the columns.  A
// sweep that rotates no pair ends the iteration: k_jacobi_svd's stopping rule.
// Bound by the chain of rounds, 7.5 us each at n = 256: the eight rotation steps
// on one warp 3 us, [A; V] J 1.8, the Gram matrix 1.1, loads and the barrier
// 1.3.  Whole SVD of triangular factors (mean of six), against one column pair per
// warp and a cluster barrier per column round: 2.26 ms for 7.98 at n = 256, 0.99 for
// 1.93 at 130, 0.46 for 0.68 at 65, with the same errors against 64 bits.
// All CTAs of a cluster are co-resident by construction, and every CTA takes
// the same number of rounds (the stopping decision is read by all from the
// same published values): the barriers cannot wait for a CTA that is not
// running.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(JK_THREADS, 1)
    k_jacobi_cluster(int n, const double* __restrict__ Ain, int lda, int trans, double* X,
                     double* __restrict__ U, double* __restrict__ S, double* __restrict__ VT,
                     int* err, int max_sweeps) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_rot[2][JK_MAX_CS];  // rank 0: whether a CTA found a pair, by sweep parity
  __shared__ int s_any;                // this round rotated
  const int rank = int(cl.block_rank()), cs = int(cl.num_blocks());
  const int np = jk_rows(n), ldx = 2 * np, P = jk_pitch(n);
  const int nb = 2 * ((n + JK_COLS - 1) / JK_COLS);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const bool work = rank < nb / 2;
  double* sX = sm;                       // JK_COLS columns of A over V
  double* sP = sX + JK_COLS * P;         // partial Gram matrices of the warps
  double* sG = sP + JK_WARPS * 192;
  double* sJ = sG + JK_COLS * JK_GP;
  double* norms = X + int64_t(nb) * JK_W * ldx;
  if (work) {
    const int c0 = rank * JK_COLS;
    for (int e = tid; e < JK_COLS * ldx; e += JK_THREADS) {
      const int col = c0 + e / ldx, i = e % ldx;
      double v = 0.0;
      if (col < n) {
        if (i < n)
          v = trans ? Ain[col + int64_t(i) * lda] : Ain[i + int64_t(col) * lda];
        else if (i >= np)
          v = i - np == col ? 1.0 : 0.0;
      }
      X[int64_t(c0) * ldx + e] = v;
    }
  }
  cl.sync();
  const double tol = 4.0 * 2.220446049250313e-16, tol2 = tol * tol;
  int sweep = 0;
  for (sweep = 0; sweep < max_sweeps; ++sweep) {
    int found = 0;  // warp 0: a pair was rotated in this sweep
    for (int r = 0; r < nb - 1; ++r) {
      if (work) {
        int bp, bq;
        jk_pair(rank, r, nb, bp, bq);
        auto column = [&](int k) {
          return X + int64_t((k < JK_W ? bp * JK_W : bq * JK_W - JK_W) + k) * ldx;
        };
        // a column per warp: its A, and later its V (16-byte copies; np is even)
        const double* src = column(warp);
        for (int i = 2 * lane; i < np; i += 64) cp_async16(sX + warp * P + i, src + i, 16);
        cp_async_commit();
        if (tid < JK_COLS * JK_COLS)
          sJ[(tid / JK_COLS) * JK_JP + tid % JK_COLS] = tid / JK_COLS == tid % JK_COLS;
        cp_async_wait<0>();
        __syncthreads();
        for (int i = np + 2 * lane; i < ldx; i += 64) cp_async16(sX + warp * P + i, src + i, 16);
        cp_async_commit();
        // Gram matrix: 8 x 8 tiles (0,0), (0,1), (1,1)
        double acc[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        for (int k4 = warp; k4 < np / 4; k4 += JK_WARPS) {
          const double x0 = sX[g * P + 4 * k4 + t], x1 = sX[(8 + g) * P + 4 * k4 + t];
          dmma(acc[0][0], acc[0][1], x0, x0);
          dmma(acc[1][0], acc[1][1], x0, x1);
          dmma(acc[2][0], acc[2][1], x1, x1);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          sP[warp * 192 + q * 64 + g * 8 + 2 * t] = acc[q][0];
          sP[warp * 192 + q * 64 + g * 8 + 2 * t + 1] = acc[q][1];
        }
        __syncthreads();
        if (tid < 192) {
          double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int w = 0; w < JK_WARPS; ++w) v[w & 3] += sP[w * 192 + tid];
          const int q = tid / 64, i = (tid >> 3) & 7, j = tid & 7;
          const int row = q == 2 ? 8 + i : i, col = q == 0 ? j : 8 + j;
          if (q == 1 || i <= j)  // one of (i, j), (j, i) where both were formed
            sG[row * JK_GP + col] = sG[col * JK_GP + row] = (v[0] + v[1]) + (v[2] + v[3]);
        }
        __syncthreads();
        if (warp == 0) {
          const int any = jk_rotate(sG, sJ, r == 0, tol2);
          found |= any;
          if (lane == 0) s_any = any;
        }
        cp_async_wait<0>();
        __syncthreads();
        if (s_any) {
          // [A; V] J, from shared memory straight to the columns in L2
          double bj[4][2];
          double* out[2][2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int k = 0; k < 4; ++k) bj[k][j] = sJ[(4 * k + t) * JK_JP + 8 * j + g];
#pragma unroll
            for (int h = 0; h < 2; ++h) out[j][h] = column(8 * j + 2 * t + h) + g;
          }
#pragma unroll 4
          for (int mt = warp; mt < ldx / 8; mt += JK_WARPS) {
            double o[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const double x = sX[(4 * k + t) * P + 8 * mt + g];
              dmma(o[0][0], o[0][1], x, bj[k][0]);
              dmma(o[1][0], o[1][1], x, bj[k][1]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int h = 0; h < 2; ++h) out[j][h][8 * mt] = o[j][h];
          }
        }
      }
      if (r == nb - 2 && tid == 0) {
        int* so = cl.map_shared_rank(&s_rot[sweep & 1][0], 0);
        so[rank] = found;
      }
      cl.sync();
    }
    const int* so = cl.map_shared_rank(&s_rot[sweep & 1][0], 0);
    int any = 0;
    for (int k = 0; k < cs; ++k) any |= so[k];
    if (!any) break;
  }
  if (rank == 0 && tid == 0 && sweep >= max_sweeps) atomicExch(err, 5);
  // Singular values = column norms, ranked descending (stable on index), and
  // the factors in that order, as in jacobi_finish.
  const int c0 = rank * JK_COLS;
  if (work) {
    for (int k = warp; k < JK_COLS; k += JK_WARPS) {
      const double* x = X + int64_t(c0 + k) * ldx;
      double v = 0.0;
      for (int i = lane; i < n; i += 32) {
        const double xi = __ldcg(x + i);
        v = fma(xi, xi, v);
      }
      v = wsum(v);
      if (lane == 0) norms[c0 + k] = sqrt(v);
    }
  }
  cl.sync();
  if (work) {
    double* sn = sm;
    int* pos = reinterpret_cast<int*>(sP);
    for (int k = tid; k < n; k += JK_THREADS) sn[k] = __ldcg(norms + k);
    __syncthreads();
    for (int k = warp; k < JK_COLS; k += JK_WARPS) {
      const int col = c0 + k;
      int before = 0;
      if (col < n)
        for (int i = lane; i < n; i += 32)
          before += (sn[i] > sn[col]) || (sn[i] == sn[col] && i < col);
      for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
      if (lane == 0) {
        pos[k] = before;
        if (col < n) S[before] = sn[col];
      }
    }
    __syncthreads();
    for (int e = tid; e < JK_COLS * n; e += JK_THREADS) {
      const int k = e / n, i = e % n, col = c0 + k;
      if (col >= n) continue;
      const double sj = sn[col];
      const double* x = X + int64_t(col) * ldx;
      const double ua = sj > 0.0 ? __ldcg(x + i) / sj : (i == pos[k] ? 1.0 : 0.0);
      const double v = __ldcg(x + np + i);
      U[i + int64_t(pos[k]) * n] = trans ? v : ua;
      VT[pos[k] + int64_t(i) * n] = trans ? ua : v;
    }
  }
  cl.sync();  // rank 0's published flags are read until here
}

// ---------------------------------------------------------------------------
// Block-cyclic form of the grid-wide Jacobi SVD: the n columns fall into
// blocks of JB_W; each round of a round-robin tournament on the blocks
// gives every CTA one block pair, whose 2 JB_W columns of A and of V it
// loads into shared memory and rotates through one full inner sweep of
// one-sided Jacobi (every pair of its columns) before writing them back.
// One grid barrier per block round instead of one per column round (31
// instead of 255 barriers per sweep at n = 256); the rotations and the
// stopping rule are those of k_jacobi_coop.
// ---------------------------------------------------------------------------

constexpr int JB_W = 8;
constexpr int JB_THREADS = 256;
constexpr int JB_WARPS = JB_THREADS / 32;

TTG_BODY(k_jacobi_block)(TTG_BLOCK, int n, const double* __restrict__ Ain,
                                                            int lda, double* A, double* V,
                                                            unsigned* bar,
                                                            unsigned long long* offmax, int* err,
                                                            int* sweep_err, int trans,
                                                            int max_sweeps) {
  extern __shared__ double sjb[];  // [2 JB_W][n] columns of A, then of V
  __shared__ int s_col[2 * JB_W];
  __shared__ double s_off[JB_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nn = int64_t(n) * n;
  for (int64_t e = blockIdx.x * int64_t(JB_THREADS) + tid; e < nn;
       e += int64_t(gridDim.x) * JB_THREADS) {
    const int64_t i = e % n, j = e / n;
    A[e] = trans ? Ain[j + i * lda] : Ain[i + j * lda];
    V[e] = (i == j) ? 1.0 : 0.0;
  }
  if (blockIdx.x == 0 && tid < 3) offmax[tid] = 0ull;
  jc_barrier(blockIdx, gridDim, bar, err);
  double* sA = sjb;
  double* sV = sjb + int64_t(2 * JB_W) * n;
  const int nb = (n + JB_W - 1) / JB_W;
  const int nbe = (nb + 1) & ~1;  // even number of block players (dummy block if odd)
  const double tol = 4.0 * 2.220446049250313e-16;
  int sweep = 0;
  for (sweep = 0; sweep < max_sweeps; ++sweep) {
    const int slot = sweep % 3;
    if (blockIdx.x == 0 && tid == 0) offmax[(sweep + 1) % 3] = 0ull;
    double off = 0.0;  // per warp
    for (int r = 0; r < nbe - 1; ++r) {
      for (int pr = blockIdx.x; pr < nbe / 2; pr += gridDim.x) {
        const int P = rr_player(pr, r, nbe), Q = rr_player(nbe - 1 - pr, r, nbe);
        // the block pair's columns (a dummy block contributes none)
        int nc = 0;
        if (tid == 0) {
          for (int b : {P, Q})
            for (int c = b * JB_W; c < (b + 1) * JB_W && c < n && b < nb; ++c) s_col[nc++] = c;
          for (int k = nc; k < 2 * JB_W; ++k) s_col[k] = -1;
        }
        __syncthreads();
        nc = 0;
        for (int k = 0; k < 2 * JB_W; ++k) nc += s_col[k] >= 0;
        for (int64_t e = tid; e < int64_t(nc) * n; e += JB_THREADS) {
          const int k = int(e / n);
          const int64_t i = e % n;
          sA[e] = A[i + int64_t(s_col[k]) * n];
          sV[e] = V[i + int64_t(s_col[k]) * n];
        }
        __syncthreads();
        // one inner sweep over all column pairs of the block pair
        const int ne = (nc + 1) & ~1;
        for (int ir = 0; ir < ne - 1; ++ir) {
          for (int ip = warp; ip < ne / 2; ip += JB_WARPS) {
            int p = rr_player(ip, ir, ne), q = rr_player(ne - 1 - ip, ir, ne);
            if (p > q) {
              const int t = p;
              p = q;
              q = t;
            }
            if (q >= nc) continue;  // dummy
            double* ap = sA + int64_t(p) * n;
            double* aq = sA + int64_t(q) * n;
            double al = 0.0, be = 0.0, ga = 0.0;
            for (int i = lane; i < n; i += 32) {
              const double x = ap[i], y = aq[i];
              al += x * x;
              be += y * y;
              ga += x * y;
            }
            al = wsum(al);
            be = wsum(be);
            ga = wsum(ga);
            const double nrm = sqrt(al * be);
            if (nrm == 0.0 || fabs(ga) <= tol * nrm) continue;  // uniform in the warp
            off = fmax(off, fabs(ga) / nrm);
            const double zeta = (be - al) / (2.0 * ga);
            const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
            const double cc = 1.0 / sqrt(1.0 + t * t), sn = cc * t;
            double* vp = sV + int64_t(p) * n;
            double* vq = sV + int64_t(q) * n;
            for (int i = lane; i < n; i += 32) {
              const double x = ap[i], y = aq[i];
              ap[i] = cc * x - sn * y;
              aq[i] = sn * x + cc * y;
              const double vx = vp[i], vy = vq[i];
              vp[i] = cc * vx - sn * vy;
              vq[i] = sn * vx + cc * vy;
            }
          }
          __syncthreads();
        }
        for (int64_t e = tid; e < int64_t(nc) * n; e += JB_THREADS) {
          const int k = int(e / n);
          const int64_t i = e % n;
          A[i + int64_t(s_col[k]) * n] = sA[e];
          V[i + int64_t(s_col[k]) * n] = sV[e];
        }
        __syncthreads();
      }
      jc_barrier(blockIdx, gridDim, bar, err);
    }
    if (lane == 0) s_off[warp] = off;
    __syncthreads();
    if (tid == 0) {
      double m = 0.0;
      for (int w = 0; w < JB_WARPS; ++w) m = fmax(m, s_off[w]);
      atomicMax(offmax + slot, (unsigned long long)__double_as_longlong(m));
    }
    jc_barrier(blockIdx, gridDim, bar, err);
    const double m = __longlong_as_double((long long)(*(volatile unsigned long long*)(offmax + slot)));
    if (m <= tol) break;
    if (*(volatile int*)err) break;
  }
  if (blockIdx.x == 0 && tid == 0 && sweep >= max_sweeps) atomicExch(sweep_err, 5);
}
TTG_COOP_KERNEL(k_jacobi_block, JB_THREADS, -1);

TTG_BODY(k_jacobi_finish)(TTG_BLOCK, int n, const double* A,
                                                             const double* V, double* U,
                                                             double* S, double* VT, double* sig,
                                                             int trans) {
  pdl_begin();
  jacobi_finish(n, A, V, U, S, VT, sig, trans);
}
TTG_KERNEL(k_jacobi_finish, SD_THREADS);

// Householder QR of the m x n matrix A (column-major, lda) held in shared
// memory: Q (m x k, ld m), R (k x n, ld k), k = min(m, n).
TTG_BODY(k_house_qr)(TTG_BLOCK, int m, int n, const double* __restrict__ Ain,
                                                        int lda, double* __restrict__ Q,
                                                        double* __restrict__ R,
                                                        const int* skip) {
  pdl_begin();
  if (skip && *skip) return;  // conditional factorization (Context::skip)
  const int ldr = m < n ? m : n;
  extern __shared__ double sm[];
  double* A = sm;                 // m x n
  double* tau = sm + int64_t(m) * n;  // k
  __shared__ double red[SD_WARPS];
  __shared__ double bcast[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = m < n ? m : n;
  for (int e = tid; e < m * n; e += SD_THREADS) A[e] = Ain[(e % m) + int64_t(e / m) * lda];
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    double* aj = A + int64_t(j) * m;
    // ||x(2:end)||^2
    double s = 0.0;
    for (int i = j + 1 + tid; i < m; i += SD_THREADS) s += aj[i] * aj[i];
    s = wsum(s);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < SD_WARPS; ++w) t += red[w];
      const double alpha = aj[j];
      double beta, tj, scal;
      if (t == 0.0) {
        beta = alpha;
        tj = 0.0;
        scal = 0.0;
      } else {
        beta = -copysign(sqrt(alpha * alpha + t), alpha);
        tj = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      tau[j] = tj;
      aj[j] = beta;
      bcast[0] = scal;
    }
    __syncthreads();
    const double scal = bcast[0];
    for (int i = j + 1 + tid; i < m; i += SD_THREADS) aj[i] *= scal;  // v(2:end), v(1) = 1
    __syncthreads();
    const double tj = tau[j];
    if (tj != 0.0) {
      for (int c = j + 1 + warp; c < n; c += SD_WARPS) {
        double* ac = A + int64_t(c) * m;
        double w = 0.0;
        for (int i = j + lane; i < m; i += 32) w += (i == j ? 1.0 : aj[i]) * ac[i];
        w = wsum(w) * tj;
        for (int i = j + lane; i < m; i += 32) ac[i] -= w * (i == j ? 1.0 : aj[i]);
      }
    }
    __syncthreads();
  }
  // R
  for (int e = tid; e < k * n; e += SD_THREADS) {
    const int i = e % k, c = e / k;
    R[i + int64_t(c) * ldr] = (i <= c) ? A[i + int64_t(c) * m] : 0.0;
  }
  __syncthreads();
  // Q = H_0 H_1 ... H_{k-1} I(:, 0:k), applied right to left in place of the
  // reflectors (LAPACK dorg2r's scheme): when H_j is applied, columns c > j
  // of A already hold Q's columns (zero in rows <= j, as I's are), so H_j
  // updates them, and then column j becomes H_j e_j = e_j - tau_j v_j, with
  // its rows above j cleared.  The arithmetic is that of applying H_j to I's
  // column j (w = tau_j exactly), so Q matches a product formed on I.
  for (int j = k - 1; j >= 0; --j) {
    const double tj = tau[j];
    double* v = A + int64_t(j) * m;
    if (tj != 0.0) {
      for (int c = j + 1 + warp; c < k; c += SD_WARPS) {
        double* qc = A + int64_t(c) * m;
        double w = 0.0;
        for (int i = j + lane; i < m; i += 32) w += (i == j ? 1.0 : v[i]) * qc[i];
        w = wsum(w) * tj;
        for (int i = j + lane; i < m; i += 32) qc[i] -= w * (i == j ? 1.0 : v[i]);
      }
    }
    __syncthreads();
    for (int i = tid; i < m; i += SD_THREADS)
      v[i] = i < j ? 0.0 : (i == j ? 1.0 - tj : 0.0 - tj * v[i]);
    __syncthreads();
  }
  for (int e = tid; e < m * k; e += SD_THREADS) Q[e] = A[e];
}
TTG_KERNEL(k_house_qr, SD_THREADS);


// ---------------------------------------------------------------------------
// Blocked Householder QR in one CTA (LAPACK's reflectors and signs), for
// matrices that fit in shared memory with their rows and columns padded to 8.
// A panel of 8 columns takes one barrier and one block-wide reduction per
// column: the inner products of the column with itself and with the panel's
// later columns are summed in one pass, together with the update by the
// previous reflector, and give the norm and all coefficients at once (the
// reflector is x scaled below the diagonal, so v'a = a_j + scal x'a).  The
// panel's reflectors then act on the columns behind it as I - V T V' (mma),
// and in reverse order on I's columns to form Q.
// Bound by the chain of columns, 1.6 us each with Q: 54 x 54 104 us for 178 with
// one reflector at a time and four barriers each, 198 x 54 125 / 255, 200 x 100
// 240 / 623, 1600 x 15 72 / 168; residual and orthogonality as before.
// ---------------------------------------------------------------------------

constexpr int QB_THREADS = 512;
constexpr int QB_WARPS = QB_THREADS / 32;
constexpr int QB_WP = 12;  // pitch of the 8-row coefficient columns (mma operand)
constexpr size_t QB_SMEM = 224 * 1024;  // beside 3 KB of static arrays

// Column pitch: at least m rounded to 8, and 4 mod 16.
__host__ __device__ __forceinline__ int64_t qb_pitch(int64_t m) {
  const int64_t mp = (m + 7) & ~int64_t(7);
  return mp + ((20 - mp % 16) & 15);
}
// Columns (and 8 more for the reflectors of a wide matrix, whose last panel may
// end inside a tile), T, and the coefficients; the partial tiles share the
// second coefficient array.
size_t qb_smem(int64_t m, int64_t n) {
  const int64_t np = (n + 7) & ~int64_t(7), kb = (std::min(m, n) + 7) / 8;
  return sizeof(double) * size_t((np + (n > m ? 8 : 0)) * qb_pitch(m) + 64 * kb + QB_WP * (np + 8) +
                                 std::max<int64_t>(QB_WP * (np + 8), 64 * QB_WARPS));
}

// Sums of eight values over a warp, value 4 b4 + 2 b3 + b2 in the lanes with
// those bits of their index (b4 highest).
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int half = 4; half >= 1; half >>= 1) {
    const bool hi = lane & (4 * half);
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = hi ? v[i] : v[i + half], keep = hi ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * half);
    }
  }
  double r = v[0];
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

TTG_BODY(k_house_qr_blk)(TTG_BLOCK, int m, int n, const double* __restrict__ Ain, int lda,
                         double* __restrict__ Q, double* __restrict__ R, const int* skip) {
  pdl_begin();
  if (skip && *skip) return;  // conditional factorization (Context::skip)
  extern __shared__ __align__(16) double sm[];
  __shared__ double s_part[2][QB_WARPS][8];
  __shared__ double s_r[8][8];  // the panel's rows of R
  __shared__ double s_tau[8];
  const int k = m < n ? m : n, mp = (m + 7) & ~7, np = (n + 7) & ~7, kb = (k + 7) / 8;
  const int P = int(qb_pitch(m));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  double* sA = sm;                        // np columns
  // A panel's reflectors, explicit (unit lower trapezoidal): in their columns'
  // place, or apart in a wide matrix.
  const bool apart = n > m;
  double* sT = sA + (np + (apart ? 8 : 0)) * P;  // T of every panel, 8 x 8 column-major
  double* sW = sT + 64 * kb;              // V'A: columns of 8 (pitch QB_WP)
  double* sW2 = sW + QB_WP * (np + 8);    // T'V'A or T V'A
  double* sK = sW2;                       // partial tiles of the warps
  double* sV = sA + np * P;
  for (int c = warp; c < np; c += QB_WARPS)
    for (int i = lane; i < mp; i += 32)
      sA[c * P + i] = c < n && i < m ? Ain[i + int64_t(c) * lda] : 0.0;

  auto explicit_v = [&](int j0, int pw) {
    if (!apart) {  // only the block on the diagonal holds anything else (R)
      sV = sA + j0 * P;
      if (tid < 64 && (tid & 7) <= tid >> 3)
        sV[(tid >> 3) * P + j0 + (tid & 7)] = (tid & 7) == tid >> 3 && tid >> 3 < pw;
      return;
    }
    for (int c = warp >> 1; c < 8; c += QB_WARPS / 2)
      for (int i = j0 + lane + 32 * (warp & 1); i < mp; i += 64) {
        const int d = i - j0 - c;
        sV[c * P + i] = c < pw && d >= 0 ? (d == 0 ? 1.0 : sA[(j0 + c) * P + i]) : 0.0;
      }
  };
  // sW = V' [V | A(:, c0 ..)] over the rows from j0 on: 1 + nt tiles of 8
  // columns, K split over the warps where there are fewer tiles than warps.
  auto project = [&](int j0, int c0, int nt) {
    const int tiles = 1 + nt, wpt = tiles < QB_WARPS ? QB_WARPS / tiles : 1;
    for (int u = warp; u < tiles * wpt; u += QB_WARPS) {
      const int tile = u / wpt;
      const double* b = tile == 0 ? sV : sA + (c0 + 8 * (tile - 1)) * P;
      // four chains: shorter sums round less, and run side by side
      double x[4][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
      for (int k4 = j0 / 4 + u % wpt; k4 < mp / 4; k4 += 4 * wpt)
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (k4 + h * wpt < mp / 4) {
            const int i = g * P + 4 * (k4 + h * wpt) + t;
            dmma(x[h][0], x[h][1], sV[i], b[i]);
          }
      const double x0 = (x[0][0] + x[1][0]) + (x[2][0] + x[3][0]);
      const double x1 = (x[0][1] + x[1][1]) + (x[2][1] + x[3][1]);
      if (wpt == 1) {
        sW[(8 * tile + 2 * t) * QB_WP + g] = x0;
        sW[(8 * tile + 2 * t + 1) * QB_WP + g] = x1;
      } else {  // u == warp: one slot per warp
        sK[u * 64 + 16 * t + g] = x0;
        sK[u * 64 + 16 * t + 8 + g] = x1;
      }
    }
    __syncthreads();
    if (wpt > 1) {
      for (int e = tid; e < tiles * 64; e += QB_THREADS) {
        const int tile = e / 64, el = e % 64;
        double v = 0.0;
        for (int w = 0; w < wpt; ++w) v += sK[(tile * wpt + w) * 64 + el];
        sW[(8 * tile + el / 8) * QB_WP + el % 8] = v;
      }
      __syncthreads();
    }
  };
  // Tiles of A -= V w2 for the columns from c0 on (nt tiles), rows from j0 on;
  // with `fresh` the columns start as those of I instead of A's (the panel's
  // own, where a tile of V is read by the warp that replaces it).
  auto apply = [&](int j0, int c0, int nt, const double* w2, bool fresh) {
    const int r0 = j0 / 8, rows = mp / 8 - r0;
    for (int u = warp; u < nt * rows; u += QB_WARPS) {
      const int ct = u / rows, rt = r0 + u % rows;
      double* M = sA + (c0 + 8 * ct) * P + 8 * rt;
      double x0 = M[2 * t * P + g], x1 = M[(2 * t + 1) * P + g], a[2];
      if (fresh) {
        x0 = rt == r0 && g == 2 * t ? 1.0 : 0.0;
        x1 = rt == r0 && g == 2 * t + 1 ? 1.0 : 0.0;
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) a[s] = -sV[(4 * s + t) * P + 8 * rt + g];
      __syncwarp();
#pragma unroll
      for (int s = 0; s < 2; ++s) dmma(x0, x1, a[s], w2[(8 * ct + g) * QB_WP + 4 * s + t]);
      M[2 * t * P + g] = x0;
      M[(2 * t + 1) * P + g] = x1;
    }
  };

  for (int p = 0; p < kb; ++p) {
    const int j0 = 8 * p, pw = min(8, k - j0);
    __syncthreads();  // loaded, or updated by the previous panel
    double* A0 = sA + j0 * P;
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = 0.0;
    for (int i = tid; i < m; i += QB_THREADS) {
      if (i <= j0) continue;
      const double x = A0[i];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = fma(x, A0[c * P + i], v[c]);
    }
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      if (jj >= pw) break;
      const int j = j0 + jj;
      // inner products of column jj, below its diagonal, with columns jj .. 7
      {
        const double s = warp_sum8(v, lane);
        const int idx = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
        if ((lane & 3) == 0) s_part[jj & 1][warp][idx] = s;
      }
      __syncthreads();  // and the rows updated by reflector jj - 1 are written
      double d = 0.0;
#pragma unroll
      for (int w = 0; w < QB_WARPS; w += 4) d += s_part[jj & 1][w + (lane >> 3)][lane & 7];
      d += __shfl_xor_sync(0xffffffffu, d, 8);
      d += __shfl_xor_sync(0xffffffffu, d, 16);
      const double tt = __shfl_sync(0xffffffffu, d, jj);
      const double alpha = A0[jj * P + j];
      double beta = alpha, tau = 0.0, scal = 0.0;
      if (tt != 0.0) {
        beta = -copysign(sqrt(alpha * alpha + tt), alpha);
        scal = 1.0 / (alpha - beta);
        tau = (beta - alpha) / beta;
      }
      double w[8];
#pragma unroll
      for (int c = jj + 1; c < 8; ++c) {
        const double a = A0[c * P + j];
        w[c] = tau * fma(scal, __shfl_sync(0xffffffffu, d, c), a);
        if (tid == 0) s_r[jj][c] = a - w[c];
      }
      if (tid == 0) {
        s_r[jj][jj] = beta;
        s_tau[jj] = tau;
      }
      // the reflector, the update of the later columns, and the inner products
      // of the next column
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = 0.0;
      for (int i = tid; i < m; i += QB_THREADS) {
        if (i <= j) continue;
        const double x = A0[jj * P + i] * scal;
        A0[jj * P + i] = x;
        double a[8];
#pragma unroll
        for (int c = jj + 1; c < 8; ++c) {
          a[c] = fma(-w[c], x, A0[c * P + i]);
          A0[c * P + i] = a[c];
        }
        if (jj < 7 && i > j + 1) {
#pragma unroll
          for (int c = jj + 1; c < 8; ++c) v[c] = fma(a[jj + 1 < 8 ? jj + 1 : 7], a[c], v[c]);
        }
      }
    }
    __syncthreads();
    if (tid < 64) {  // the panel's block of R
      const int i = tid & 7, c = tid >> 3;
      if (i < pw && j0 + c < n)
        R[j0 + i + int64_t(j0 + c) * k] = c >= i ? s_r[i][c] : 0.0;
    }
    explicit_v(j0, pw);
    __syncthreads();
    const int c0 = j0 + 8, nt = (np - c0) / 8;
    project(j0, c0, nt);
    if (warp == 0) {  // T(0:j, j) = -tau_j T(0:j, 0:j) V'v_j, row `lane`
      double T[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double tau = j < pw ? s_tau[j] : 0.0;
        double x = 0.0;
#pragma unroll
        for (int l = 0; l < j; ++l) x = fma(T[l], sW[j * QB_WP + l], x);
        T[j] = lane == j ? tau : (lane < j ? -tau * x : 0.0);
        if (lane < 8) sT[64 * p + 8 * j + lane] = T[j];
      }
    }
    __syncthreads();
    for (int e = tid; e < 64 * nt; e += QB_THREADS) {  // T' (V'A)
      const int c = e / 8, i = e % 8;
      double x = 0.0;
#pragma unroll
      for (int l = 0; l < 8; ++l)
        if (l <= i) x = fma(sT[64 * p + 8 * i + l], sW[(8 + c) * QB_WP + l], x);
      sW2[c * QB_WP + i] = x;
    }
    __syncthreads();
    apply(j0, c0, nt, sW2, false);
  }
  __syncthreads();
  // The rest of R: above each panel's block, and zeros below.
  for (int c = warp; c < n; c += QB_WARPS) {
    const int b0 = min(c & ~7, 8 * kb);
    for (int i = lane; i < k; i += 32)
      if (i < b0 || i >= b0 + 8) R[i + int64_t(c) * k] = i < b0 ? sA[c * P + i] : 0.0;
  }
  // Q = (I - V_0 T_0 V_0') ... I, the last panel first: a panel acts on the
  // columns behind it, which hold Q's already, and replaces its own.
  const int qc = 8 * kb;
  for (int p = kb - 1; p >= 0; --p) {
    const int j0 = 8 * p, pw = min(8, k - j0);
    __syncthreads();
    explicit_v(j0, pw);
    __syncthreads();
    const int c0 = j0 + 8, nt = (qc - c0) / 8;
    project(j0, c0, nt);
    for (int e = tid; e < 64 * (nt + 1); e += QB_THREADS) {
      const int c = e / 8, i = e % 8;
      double x = 0.0;
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        const double b = c < 8 ? sV[l * P + j0 + c] : sW[c * QB_WP + l];
        if (l >= i) x = fma(sT[64 * p + 8 * l + i], b, x);
      }
      sW2[c * QB_WP + i] = x;
    }
    for (int c = warp; c < 8; c += QB_WARPS)  // Q's rows above the panel's
      for (int i = lane; i < j0; i += 32) sA[(j0 + c) * P + i] = 0.0;
    __syncthreads();
    apply(j0, c0, nt, sW2 + 8 * QB_WP, false);
    __syncthreads();
    apply(j0, j0, 1, sW2, true);
  }
  __syncthreads();
  for (int c = warp; c < k; c += QB_WARPS)
    for (int i = lane; i < m; i += 32) Q[i + int64_t(c) * m] = sA[c * P + i];
}
TTG_KERNEL(k_house_qr_blk, QB_THREADS);

// ---------------------------------------------------------------------------
// Householder QR of a skinny m x n matrix (n <= SK_MAX_N) too tall for shared
// memory: the work copy W lives in global memory (L2), every thread owns the
// rows i = tid (mod SD_THREADS), and each reflector needs two block-wide
// reductions -- the column norm, then the n - j - 1 inner products of all
// trailing columns at once -- instead of one warp per column.  Same
// reflectors and signs as k_house_qr (LAPACK's dlarfg convention).
// ---------------------------------------------------------------------------

constexpr int SK_MAX_N = 8;

// Block-wide sums of cnt <= SK_MAX_N values per thread; every thread gets
// the totals in out[0..cnt).  scratch: SD_WARPS * SK_MAX_N doubles (shared).
__device__ void block_sums(const double* v, int cnt, double* scratch, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = 0; q < cnt; ++q) {
    const double s = wsum(v[q]);
    if (lane == 0) scratch[warp * SK_MAX_N + q] = s;
  }
  __syncthreads();
  if (threadIdx.x < cnt) {
    double t = 0.0;
    for (int w = 0; w < SD_WARPS; ++w) t += scratch[w * SK_MAX_N + threadIdx.x];
    scratch[SD_WARPS * SK_MAX_N + threadIdx.x] = t;
  }
  __syncthreads();
  for (int q = 0; q < cnt; ++q) out[q] = scratch[SD_WARPS * SK_MAX_N + q];
  __syncthreads();
}

TTG_BODY(k_house_qr_skinny)(TTG_BLOCK, int64_t m, int n,
                                                               const double* __restrict__ Ain,
                                                               int64_t lda, double* __restrict__ W,
                                                               double* __restrict__ Q,
                                                               double* __restrict__ R) {
  pdl_begin();
  __shared__ double scratch[(SD_WARPS + 1) * SK_MAX_N];
  __shared__ double tau[SK_MAX_N];
  const int tid = threadIdx.x;
  const int k = int(m < n ? m : n);
  for (int64_t e = tid; e < m * n; e += SD_THREADS) W[e] = Ain[(e % m) + (e / m) * lda];
  __syncthreads();
  double part[SK_MAX_N], tot[SK_MAX_N];
  for (int j = 0; j < k; ++j) {
    double* wj = W + int64_t(j) * m;
    double s = 0.0;
    for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) s += wj[i] * wj[i];
    part[0] = s;
    block_sums(part, 1, scratch, tot);
    const double alpha = wj[j];
    __syncthreads();  // every thread has read alpha before wj[j] changes
    double beta, tj, scal;
    if (tot[0] == 0.0) {
      beta = alpha;
      tj = 0.0;
      scal = 0.0;
    } else {
      beta = -copysign(sqrt(alpha * alpha + tot[0]), alpha);
      tj = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) wj[i] *= scal;  // v, v(j) = 1
    if (tid == 0) {
      tau[j] = tj;
      wj[j] = beta;
    }
    __syncthreads();
    const int nc = n - j - 1;
    if (tj != 0.0 && nc > 0) {
      for (int q = 0; q < nc; ++q) part[q] = 0.0;
      for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) {
        const double vi = wj[i];
        for (int q = 0; q < nc; ++q) part[q] += vi * W[i + int64_t(j + 1 + q) * m];
      }
      block_sums(part, nc, scratch, tot);
      for (int q = 0; q < nc; ++q) tot[q] = tj * (tot[q] + W[j + int64_t(j + 1 + q) * m]);
      __syncthreads();  // row j read by all before it changes
      for (int q = 0; q < nc; ++q) {
        double* wc = W + int64_t(j + 1 + q) * m;
        for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) wc[i] -= tot[q] * wj[i];
        if (tid == 0) wc[j] -= tot[q];
      }
      __syncthreads();
    }
  }
  for (int e = tid; e < k * n; e += SD_THREADS) {
    const int i = e % k, c = e / k;
    R[i + int64_t(c) * k] = (i <= c) ? W[i + int64_t(c) * m] : 0.0;
  }
  // Q = H_0 ... H_{k-1} I(:, 0:k), right to left.
  for (int64_t e = tid; e < m * k; e += SD_THREADS) Q[e] = ((e % m) == (e / m)) ? 1.0 : 0.0;
  __syncthreads();
  for (int j = k - 1; j >= 0; --j) {
    const double tj = tau[j];
    if (tj == 0.0) continue;  // uniform
    const double* v = W + int64_t(j) * m;
    const int nc = k - j;
    for (int q = 0; q < nc; ++q) part[q] = 0.0;
    for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) {
      const double vi = v[i];
      for (int q = 0; q < nc; ++q) part[q] += vi * Q[i + int64_t(j + q) * m];
    }
    block_sums(part, nc, scratch, tot);
    for (int q = 0; q < nc; ++q) tot[q] = tj * (tot[q] + Q[j + int64_t(j + q) * m]);
    __syncthreads();  // row j read by all before it changes
    for (int q = 0; q < nc; ++q) {
      double* qc = Q + int64_t(j + q) * m;
      for (int64_t i = j + 1 + tid; i < m; i += SD_THREADS) qc[i] -= tot[q] * v[i];
      if (tid == 0) qc[j] -= tot[q];
    }
    __syncthreads();
  }
}
TTG_KERNEL(k_house_qr_skinny, SD_THREADS);

// ---------------------------------------------------------------------------
// Cholesky factor and its inverse for shifted Cholesky QR
// ---------------------------------------------------------------------------

// G (n x n SPD Gram matrix, ldg) -> R = chol(G + shift I) upper (R' R = G +
// shift I) and Rinv = R^{-1}, both n x n with leading dimension n.  shift =
// shift_factor * trace(G).  err_slot |= 1 if a pivot is not positive.
//
// Right-looking Cholesky G = L L' in blocks of 8 columns, with the forward
// elimination L X = I applied to X = I in the same steps.  A step's diagonal
// block is factored and inverted by one warp in registers, every lane the
// whole block (no exchange inside its chain of 8 reciprocal roots); the block
// column of L and the block row of X take one 8 x 8 x 8 product per warp, and
// the trailing tiles of L and X below them two mma each.  Warp 0 updates the
// next diagonal block first and factors it while the others update the rest.
// Bound by that chain, about 4000 cycles per step: 25 us at n = 96, against some
// 80 us with one column per step (rounding at d = 20, n = 16, ranks 256 runs 300
// of them: 104 -> 77 ms).
// Tiles are column-major with a pitch of 4 mod 16 doubles (mma fragments meet
// no bank twice); rows and columns beyond n are those of the identity.
constexpr int CI_THREADS = 512;
constexpr int CI_WARPS = CI_THREADS / 32;
constexpr int CI_MAX_N = 96;

__host__ __device__ __forceinline__ int ci_pitch(int n) { return (((n + 7) & ~7) + 15 & ~15) + 4; }

// 1 / sqrt(d): two Newton steps from single precision where its range holds d.
__device__ __forceinline__ double ci_rsqrt(double d) {
  if (!(d > 1e-30 && d < 1e30)) return rsqrt(d);
  double r = double(rsqrtf(float(d)));
  r = fma(0.5 * r, fma(-d * r, r, 1.0), r);
  return fma(0.5 * r, fma(-d * r, r, 1.0), r);
}

TTG_BODY(k_chol_inv)(TTG_BLOCK, int n, const double* __restrict__ G,
                                                        int ldg, double shift_factor,
                                                        double* __restrict__ R,
                                                        double* __restrict__ Rinv, int* err) {
  pdl_begin();
  extern __shared__ double sm[];
  const int np = (n + 7) & ~7, nb = np / 8, P = ci_pitch(n);
  double* L = sm;            // np x np, lower triangle = Cholesky factor
  double* X = sm + P * np;   // np x np, L^{-1}
  __shared__ double s_li[64];  // inverse of the step's diagonal block, row k at 8 k
  __shared__ double s_shift;
  __shared__ int s_bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  if (warp == 0) {
    double tr = 0.0;
    for (int i = lane; i < n; i += 32) tr += G[i + int64_t(i) * ldg];
    tr = wsum(tr);
    if (lane == 0) {
      s_shift = shift_factor * tr;
      s_bad = 0;
    }
  }
  __syncthreads();
  const double shift = s_shift;
  for (int c = warp; c < np; c += CI_WARPS)
    for (int r = lane; r < np; r += 32) {
      double v = r == c ? 1.0 : 0.0;
      X[c * P + r] = v;
      if (r < n && c < n) v = G[r + int64_t(c) * ldg] + (r == c ? shift : 0.0);
      L[c * P + r] = v;
    }
  __syncthreads();

  // Factor the diagonal block at j0 (in place) and leave its inverse in s_li.
  auto diagonal = [&](int j0) {
    double a[8][8], inv[8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int r = c; r < 8; ++r) a[r][c] = L[(j0 + c) * P + j0 + r];
    bool bad = false;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double d = a[c][c];
      const bool pos = d > 0.0;
      bad |= !pos;
      inv[c] = pos ? ci_rsqrt(d) : 1.0;
      a[c][c] = pos ? d * inv[c] : 1.0;
#pragma unroll
      for (int r = c + 1; r < 8; ++r) a[r][c] *= inv[c];
#pragma unroll
      for (int k = c + 1; k < 8; ++k)
#pragma unroll
        for (int r = k; r < 8; ++r) a[r][k] = fma(-a[r][c], a[k][c], a[r][k]);
    }
    // column `lane` of the inverse
    double x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      double v = r == lane ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < r; ++k) v = fma(-a[r][k], x[k], v);
      x[r] = v * inv[r];
    }
    __syncwarp();
    if (lane < 8) {
#pragma unroll
      for (int r = 0; r < 8; ++r) s_li[lane * 8 + r] = x[r];
    }
    if (lane == 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = c; r < 8; ++r) L[(j0 + c) * P + j0 + r] = a[r][c];
      if (bad) s_bad = 1;
    }
  };
  // Tile at M (column-major, pitch P) -= A B, the two k slices of A and B given.
  auto update = [&](double* M, const double (&a)[2], const double (&b)[2]) {
    double c0 = M[(2 * t) * P + g], c1 = M[(2 * t + 1) * P + g];
    dmma(c0, c1, -a[0], b[0]);
    dmma(c0, c1, -a[1], b[1]);
    M[(2 * t) * P + g] = c0;
    M[(2 * t + 1) * P + g] = c1;
  };

  if (warp == 0) diagonal(0);
  for (int jb = 0; jb < nb; ++jb) {
    const int j0 = 8 * jb;
    __syncthreads();  // diagonal block factored, trailing tiles up to date
    for (int u = warp; u < nb; u += CI_WARPS) {
      double c0 = 0.0, c1 = 0.0, a[2], b[2];
      double* M;
      if (u > jb) {  // L_u = W_u inv(L_jj)'
        M = L + j0 * P + 8 * u;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          a[s] = M[(4 * s + t) * P + g];
          b[s] = s_li[(4 * s + t) * 8 + g];
        }
      } else {  // X_j = inv(L_jj) X_j, column block u
        M = X + 8 * u * P + j0;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          a[s] = s_li[(4 * s + t) * 8 + g];
          b[s] = M[g * P + 4 * s + t];
        }
      }
      __syncwarp();
      dmma(c0, c1, a[0], b[0]);
      dmma(c0, c1, a[1], b[1]);
      M[(2 * t) * P + g] = c0;
      M[(2 * t + 1) * P + g] = c1;
    }
    if (jb + 1 == nb) break;
    __syncthreads();  // block column of L and block row of X are final
    // Tiles (i, k) below: L for k > jb (i >= k), X for k <= jb.
    auto tile = [&](int i, int k) {
      double a[2], b[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        a[s] = L[(j0 + 4 * s + t) * P + 8 * i + g];
        b[s] = k > jb ? L[(j0 + 4 * s + t) * P + 8 * k + g] : X[(8 * k + g) * P + j0 + 4 * s + t];
      }
      update((k > jb ? L : X) + 8 * k * P + 8 * i, a, b);
    };
    if (warp == 0) {
      tile(jb + 1, jb + 1);
      __syncwarp();
      diagonal(j0 + 8);
    } else {
      // the other tiles row by row, every CI_WARPS - 1st of them
      int i = jb + 1, k = warp - 1, len = jb + 1;  // row jb + 1 without its last tile
      while (true) {
        while (i < nb && k >= len) {
          k -= len;
          ++i;
          len = i + 1;
        }
        if (i >= nb) break;
        tile(i, k);
        k += CI_WARPS - 1;
      }
    }
  }
  __syncthreads();
  for (int c = warp; c < n; c += CI_WARPS)
    for (int i = lane; i < n; i += 32) {
      R[i + int64_t(n) * c] = i <= c ? L[i * P + c] : 0.0;
      Rinv[i + int64_t(n) * c] = i <= c ? X[i * P + c] : 0.0;
    }
  if (tid == 0 && s_bad) atomicOr(err, 1);
}
TTG_KERNEL(k_chol_inv, CI_THREADS);


// ---------------------------------------------------------------------------
// One-sided Jacobi SVD of a tall m x n matrix with few columns (n <=
// TS_MAX_N, m >= n), held in shared memory and rotated directly (no QR
// first): one warp per column pair of a round-robin round, the rotation and
// stopping rule of k_jacobi_svd.  U = A V diag(1/s) (m x n, ld m); columns of
// exactly zero norm are completed to an orthonormal set (Gram-Schmidt of unit
// vectors against the other columns), so U always has orthonormal columns.
// S descending, VT (n x n, ld n).  One launch replaces QR + square SVD +
// U = Q Ur for the small SVDs of the sweeps (Z updates, early truncations).
// ---------------------------------------------------------------------------

constexpr int TS_THREADS = 256;
constexpr int TS_WARPS = TS_THREADS / 32;
constexpr int TS_MAX_N = 8;

TTG_BODY(k_svd_tall_small)(TTG_BLOCK, int m, int n,
                                                              const double* __restrict__ Ain,
                                                              int lda, double* __restrict__ U,
                                                              double* __restrict__ S,
                                                              double* __restrict__ VT,
                                                              int* err, int max_sweeps) {
  pdl_begin();
  extern __shared__ double A[];  // m x n
  __shared__ double V[TS_MAX_N * TS_MAX_N];
  __shared__ double sig[TS_MAX_N];
  __shared__ int pos[TS_MAX_N];
  __shared__ double s_off[TS_WARPS];
  __shared__ int s_done;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < m * n; e += TS_THREADS) {
    const int i = e % m, j = e / m;
    A[e] = Ain[i + int64_t(j) * lda];
  }
  for (int e = tid; e < n * n; e += TS_THREADS) V[e] = (e % n == e / n) ? 1.0 : 0.0;
  __syncthreads();
  const int ne = (n + 1) & ~1;
  const double tol = 4.0 * 2.220446049250313e-16, tol2 = tol * tol;
  int sweep = 0;
  for (sweep = 0; sweep < max_sweeps; ++sweep) {
    double off = 0.0;
    for (int r = 0; r < ne - 1; ++r) {
      for (int pr = warp; pr < ne / 2; pr += TS_WARPS) {
        int p = rr_player(pr, r, ne), q = rr_player(ne - 1 - pr, r, ne);
        if (p > q) {
          const int t = p;
          p = q;
          q = t;
        }
        if (q >= n) continue;  // dummy player
        double* ap = A + int64_t(p) * m;
        double* aq = A + int64_t(q) * m;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int i = lane; i < m; i += 32) {
          const double x = ap[i], y = aq[i];
          al += x * x;
          be += y * y;
          ga += x * y;
        }
        al = wsum(al);
        be = wsum(be);
        ga = wsum(ga);
        const double ab = al * be, g2 = ga * ga;
        if (ab == 0.0 || g2 <= tol2 * ab) continue;
        off = fmax(off, g2 / ab);
        const double dd = be - al, gg = 2.0 * ga;
        const double sg = ((dd >= 0.0) == (gg > 0.0) || dd == 0.0) ? 1.0 : -1.0;
        const double t = sg * fabs(gg) / (fabs(dd) + sqrt(dd * dd + gg * gg));
        const double c = rsqrt(1.0 + t * t), s = c * t;
        for (int i = lane; i < m; i += 32) {
          const double x = ap[i], y = aq[i];
          ap[i] = c * x - s * y;
          aq[i] = s * x + c * y;
        }
        if (lane < n) {
          const double vx = V[lane + p * n], vy = V[lane + q * n];
          V[lane + p * n] = c * vx - s * vy;
          V[lane + q * n] = s * vx + c * vy;
        }
      }
      __syncthreads();
    }
    if (lane == 0) s_off[warp] = off;
    __syncthreads();
    if (tid == 0) {
      double mx = 0.0;
      for (int w = 0; w < TS_WARPS; ++w) mx = fmax(mx, s_off[w]);
      s_done = (mx <= tol2) ? 1 : 0;
    }
    __syncthreads();
    if (s_done) break;
  }
  if (tid == 0 && sweep >= max_sweeps) atomicExch(err, 5);
  // singular values = column norms, ranked descending (stable on index)
  if (warp < n) {
    const double* aj = A + int64_t(warp) * m;
    double s = 0.0;
    for (int i = lane; i < m; i += 32) s += aj[i] * aj[i];
    s = wsum(s);
    if (lane == 0) sig[warp] = sqrt(s);
  }
  __syncthreads();
  if (tid < n) {
    const double sj = sig[tid];
    int p = 0;
    for (int k = 0; k < n; ++k) p += (sig[k] > sj) || (sig[k] == sj && k < tid);
    pos[tid] = p;
  }
  for (int e = tid; e < m * n; e += TS_THREADS) {
    const double sj = sig[e / m];
    if (sj > 0.0) A[e] /= sj;
  }
  __syncthreads();
  // complete zero columns: e_k minus its projections on the columns kept so
  // far (twice), accepted when at least 0.3 of it is left (the mean left
  // over all k is at least 1 - (n - 1) / m >= 1 / n)
  if (warp == 0) {
    for (int j = 0; j < n; ++j) {
      if (sig[j] > 0.0) continue;
      double* aj = A + int64_t(j) * m;
      for (int k = 0; k < m; ++k) {
        for (int i = lane; i < m; i += 32) aj[i] = (i == k) ? 1.0 : 0.0;
        __syncwarp();
        for (int pass = 0; pass < 2; ++pass) {
          for (int q = 0; q < n; ++q) {
            if (q == j || (sig[q] == 0.0 && q > j)) continue;
            const double* aq = A + int64_t(q) * m;
            double d = 0.0;
            for (int i = lane; i < m; i += 32) d += aq[i] * aj[i];
            d = wsum(d);
            for (int i = lane; i < m; i += 32) aj[i] -= d * aq[i];
            __syncwarp();
          }
        }
        double nr = 0.0;
        for (int i = lane; i < m; i += 32) nr += aj[i] * aj[i];
        nr = sqrt(wsum(nr));
        if (nr > 0.3) {
          for (int i = lane; i < m; i += 32) aj[i] /= nr;
          __syncwarp();
          break;
        }
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < m * n; e += TS_THREADS) {
    const int i = e % m, j = e / m;
    U[i + int64_t(pos[j]) * m] = A[e];
  }
  for (int e = tid; e < n * n; e += TS_THREADS) {
    const int i = e % n, j = e / n;
    VT[pos[j] + i * n] = V[e];
  }
  if (tid < n) S[pos[tid]] = sig[tid];
}
TTG_KERNEL(k_svd_tall_small, TS_THREADS);

// ---------------------------------------------------------------------------
// LU with partial pivoting and the two triangular solves (LAPACK getf2 +
// getrs, unblocked) of an n x n matrix held in shared memory, for the dense
// local systems of AMEn (n < max_full_size): X <- B^{-1} X for nrhs
// right-hand sides.  The pivot is the first entry of largest magnitude in
// its column (idamax); the multipliers are formed with the pivot's
// reciprocal; the row swaps and the unit-lower elimination are applied to X
// as the factorization proceeds, then X is solved with the upper factor
// column by column.  *err |= 1 on an exactly zero pivot (getrf's info > 0).
// ---------------------------------------------------------------------------

TTG_BODY(k_lu_small)(TTG_BLOCK, int n, const double* __restrict__ B, int nrhs,
                     double* __restrict__ X, int* err) {
  pdl_begin();
  extern __shared__ double slu[];
  double* a = slu;             // n x n, column-major
  double* x = slu + n * n;     // n x nrhs
  __shared__ int s_piv, s_bad;
  const int tid = threadIdx.x;
  for (int e = tid; e < n * n; e += blockDim.x) a[e] = B[e];
  for (int e = tid; e < n * nrhs; e += blockDim.x) x[e] = X[e];
  if (tid == 0) s_bad = 0;
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    if (tid < 32) {  // idamax over rows k..n-1 of column k
      double best = -1.0;
      int bi = k;
      for (int i = k + tid; i < n; i += 32) {
        const double v = fabs(a[i + n * k]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
        }
      }
      if (tid == 0) {
        s_piv = bi;
        if (!(best > 0.0)) s_bad = 1;
      }
    }
    __syncthreads();
    const int p = s_piv;
    if (p != k) {
      for (int j = tid; j < n; j += blockDim.x) {
        const double t = a[k + n * j];
        a[k + n * j] = a[p + n * j];
        a[p + n * j] = t;
      }
      for (int r = tid; r < nrhs; r += blockDim.x) {
        const double t = x[k + n * r];
        x[k + n * r] = x[p + n * r];
        x[p + n * r] = t;
      }
    }
    __syncthreads();
    const double piv = a[k + n * k];
    if (piv != 0.0) {
      const double rinv = 1.0 / piv;
      for (int i = k + 1 + tid; i < n; i += blockDim.x) a[i + n * k] *= rinv;
    }
    __syncthreads();
    const int rows = n - k - 1;
    if (rows > 0) {
      const int tot = rows * (n - k - 1 + nrhs);
      for (int e = tid; e < tot; e += blockDim.x) {
        const int i = k + 1 + e % rows, c = e / rows;
        const double l = a[i + n * k];
        if (c < n - k - 1) {
          const int j = k + 1 + c;
          a[i + n * j] -= l * a[k + n * j];
        } else {
          const int r = c - (n - k - 1);
          x[i + n * r] -= l * x[k + n * r];
        }
      }
    }
    __syncthreads();
  }
  for (int k = n - 1; k >= 0; --k) {
    for (int r = tid; r < nrhs; r += blockDim.x) x[k + n * r] /= a[k + n * k];
    __syncthreads();
    for (int e = tid; e < k * nrhs; e += blockDim.x) {
      const int i = e % k, r = e / k;
      x[i + n * r] -= x[k + n * r] * a[i + n * k];
    }
    __syncthreads();
  }
  for (int e = tid; e < n * nrhs; e += blockDim.x) X[e] = x[e];
  if (tid == 0 && s_bad) atomicOr(err, 1);
}
TTG_KERNEL(k_lu_small, SD_THREADS);

}  // namespace

bool lu_small_fits(int64_t n, int64_t nrhs) {
  return n >= 1 && nrhs >= 1 && sizeof(double) * size_t(n) * size_t(n + nrhs) <= SMEM_LIMIT;
}

void lu_small_f64(Context* c, int64_t n, const double* B, double* X, int64_t nrhs) {
  TTG_REQUIRE(lu_small_fits(n, nrhs), "lu_small: n = %lld, nrhs = %lld out of range",
              (long long)n, (long long)nrhs);
  const size_t smem = sizeof(double) * size_t(n) * size_t(n + nrhs);
  ensure_smem_attr(k_lu_small.fn(), c->device, int(SMEM_LIMIT + 1024));
  launch(c, k_lu_small, 1, SD_THREADS, smem, int(n), B, int(nrhs), X, c->d_err + 4);
  TTG_CHECK_LAUNCH();
}

bool chol_inv_fits(int64_t n) { return n <= CI_MAX_N; }

void chol_inv_f64(Context* c, int64_t n, const double* G, int64_t ldg, double shift_factor,
                  double* R, double* Rinv, int* flag) {
  TTG_REQUIRE(chol_inv_fits(n), "chol_inv: n = %lld too large", (long long)n);
  auto bytes = [](int64_t k) {
    return 2 * sizeof(double) * size_t(ci_pitch(int(k))) * size_t((k + 7) & ~int64_t(7));
  };
  ensure_smem_attr(k_chol_inv.fn(), c->device, int(bytes(CI_MAX_N)));
  launch(c, k_chol_inv, 1, CI_THREADS, bytes(n), int(n), G, int(ldg), shift_factor, R, Rinv,
         flag ? flag : c->d_err + 4);
  TTG_CHECK_LAUNCH();
}

bool skinny_qr_fits(int64_t m, int64_t n) { return n >= 1 && n <= SK_MAX_N && m >= n; }

void skinny_qr_f64(Context* c, int64_t m, int64_t n, const double* A, int64_t lda, double* Q,
                   double* R) {
  TTG_REQUIRE(skinny_qr_fits(m, n), "skinny QR: %lld x %lld out of range", (long long)m,
              (long long)n);
  DBuf<double> W(c, m * n);
  launch(c, k_house_qr_skinny, 1, SD_THREADS, 0, m, int(n), A, lda, W.p(), Q, R);
  TTG_CHECK_LAUNCH();
}

bool small_qr_fits(int64_t m, int64_t n) {
  return m * n + std::min(m, n) <= int64_t(SMEM_LIMIT / sizeof(double)) && m <= 0x7fffffff;
}

void small_qr_f64(Context* c, int64_t m, int64_t n, const double* A, int64_t lda, double* Q,
                  double* R) {
  // The blocked kernel where its padded columns fit (the element-wise one is
  // left with shapes like 4 x 5000) and there are more than a few reflectors:
  // its panel takes eight columns' steps whatever their number.  Device time,
  // blocked / one reflector at a time: 2 x 2 6.8 / 4.9 us, 400 x 2 9.1 / 6.8, 2 x
  // 400 21.3 / 11.5, 3 x 3 7.9 / 6.9, 200 x 3 9.3 / 8.8, 3 x 400 22.3 / 20.3; but
  // 400 x 3 10.3 / 10.8, 1600 x 3 18.1 / 22.4, 4 x 4 8.9 / 8.9, 100 x 4 10.1 / 10.7,
  // 4 x 400 23.4 / 28.8.
  const int64_t k = std::min(m, n);
  const bool few = k <= 2 || (k == 3 && m <= 256);
  if (!few && qb_smem(m, n) <= QB_SMEM) {
    ensure_smem_attr(k_house_qr_blk.fn(), c->device, int(QB_SMEM));
    launch(c, k_house_qr_blk, 1, QB_THREADS, qb_smem(m, n), int(m), int(n), A, int(lda), Q, R,
           c->skip);
    TTG_CHECK_LAUNCH();
    return;
  }
  const size_t smem = sizeof(double) * size_t(m * n + std::min(m, n));
  ensure_smem_attr(k_house_qr.fn(), c->device, int(SMEM_LIMIT + 1024));
  launch(c, k_house_qr, 1, SD_THREADS, smem, int(m), int(n), A, int(lda), Q, R, c->skip);
  TTG_CHECK_LAUNCH();
}


bool svd_tall_small_fits(int64_t m, int64_t n) {
  return n >= 1 && n <= TS_MAX_N && m >= n && m * n * int64_t(sizeof(double)) <= int64_t(128 * 1024);
}

void svd_tall_small_f64(Context* c, int64_t m, int64_t n, const double* A, int64_t lda, double* U,
                        double* S, double* VT) {
  TTG_REQUIRE(svd_tall_small_fits(m, n), "svd_tall_small: %lld x %lld out of range",
              (long long)m, (long long)n);
  const size_t smem = sizeof(double) * size_t(m * n);
  ensure_smem_attr(k_svd_tall_small.fn(), c->device,
                   int(128 * 1024 + 1024));
  launch(c, k_svd_tall_small, 1, TS_THREADS, smem, int(m), int(n), A, int(lda), U, S, VT,
         c->d_err + 3, c->jacobi_max_sweeps);
  TTG_CHECK_LAUNCH();
}

// TTG_JACOBI_BLOCK=1 selects the block-cyclic grid-wide Jacobi SVD; the
// default is the one-pair-per-CTA rounds (measured no slower in rounding and
// a little more accurate at n >= 256).
static bool getenv_flag_on(const char* name) {
  const char* e = getenv(name);
  return e && e[0] == '1';
}

// The block-pair columns of A and V (4 JB_W n doubles) fit in shared memory.
static bool jacobi_block_fits(int64_t n) {
  return n >= 4 * JB_W && sizeof(double) * 4 * JB_W * size_t(n) <= SMEM_LIMIT &&
         getenv_flag_on("TTG_JACOBI_BLOCK");
}

// CTAs of the cluster form: one per pair of blocks, a power of two.
int jacobi_cluster_size(int64_t n) {
  int cs = 1;
  while (2 * cs < jk_blocks(n)) cs *= 2;
  return cs;
}

// The cluster form runs where one CTA's shared memory cannot hold both A
// and V (n > JS_MAX_N) up to JK_MAX_N, unless TTG_JACOBI_CLUSTER=0, when the device
// can place a cluster with that shared memory (checked once per device and
// size class: attributes set, cudaOccupancyMaxActiveClusters).  Outside a
// grouped batch it also takes the sizes from TTG_JACOBI_CLUSTER_MIN_N (default
// 48) up, which the one-CTA kernel could hold: a lone solve waits on each SVD
// (triangular factor, cluster against one CTA: 0.18 / 0.16 ms at n = 32, 0.31 /
// 0.31 at 47, 0.40 / 0.53 at 64, 0.58 / 1.18 at 96), while a grouped batch
// fills the GPU with concurrent systems and wants the one-CTA kernel's single
// SM.  Below 48 both run the one-CTA kernel, so that a grouped batch of such
// ranks repeats a lone solve.
int64_t jacobi_cluster_min_n() {
  static const int64_t v = [] {
    const char* e = getenv("TTG_JACOBI_CLUSTER_MIN_N");
    const long long x = e ? atoll(e) : 0;
    return int64_t(x >= 2 ? x : 48);
  }();
  return v;
}

cudaLaunchConfig_t jacobi_cluster_config(int64_t n, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(jacobi_cluster_size(n));
  cfg.blockDim = dim3(JK_THREADS);
  cfg.dynamicSmemBytes = jk_smem(n);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = jacobi_cluster_size(n);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

bool jacobi_cluster_ok(Context* c, int64_t n) {
  static const bool on = [] {
    const char* e = getenv("TTG_JACOBI_CLUSTER");
    return !(e && e[0] == '0');
  }();
  if (!on || n > JK_MAX_N || n < 2) return false;
  static std::mutex mu;
  static std::map<std::pair<int, size_t>, bool> seen;
  std::lock_guard<std::mutex> lk(mu);
  auto key = std::make_pair(c->device, jk_smem(n) * 32 + jacobi_cluster_size(n));
  auto it = seen.find(key);
  if (it != seen.end()) return it->second;
  // The attribute is set once to the largest size any n takes (setting it
  // per size would lower it below a size already admitted).
  bool ok = cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                 1) == cudaSuccess &&
            cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(jk_smem(JK_MAX_N))) == cudaSuccess;
  if (ok) {
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = jacobi_cluster_config(n, attr);
    int clusters = 0;
    ok = cudaOccupancyMaxActiveClusters(&clusters, k_jacobi_cluster, &cfg) == cudaSuccess &&
         clusters >= 1;
  }
  cudaGetLastError();  // a refused attribute or query leaves no sticky state
  seen[key] = ok;
  return ok;
}

void jacobi_svd_f64(Context* c, int64_t n, const double* A, int64_t lda, double* U, double* S,
                    double* VT, bool via_transpose) {
  int trans = via_transpose ? 1 : 0;
  TTG_REQUIRE(n >= 1 && n <= 4096, "jacobi_svd: n = %lld out of range", (long long)n);
  const bool one_cta = n <= JS_MAX_N;
  const bool block = n > 160 && jacobi_block_fits(n);
  if (!block && (!one_cta || (!c->rec && n >= jacobi_cluster_min_n())) &&
      jacobi_cluster_ok(c, n)) {
    // One cluster, the columns in L2.
    DBuf<double> X(c, jk_work(n));
    const int ns = int(n), ilda = int(lda), sweeps = c->jacobi_max_sweeps;
    double* Xw = X.p();
    int* err = c->d_err + 3;
    auto issue = [=](cudaStream_t s) {
      cudaLaunchAttribute attr[1];
      cudaLaunchConfig_t cfg = jacobi_cluster_config(ns, attr);
      cfg.stream = s;
      TTG_CUDA(cudaLaunchKernelEx(&cfg, k_jacobi_cluster, ns, A, ilda, trans, Xw, U, S, VT, err,
                                  sweeps));
    };
    if (c->rec) {
      rec_op(c->rec, [issue](cudaStream_t s, cusolverDnHandle_t) { issue(s); });
    } else {
      issue(c->stream);
    }
    c->launches += 1;
    TTG_CHECK_LAUNCH();
    return;
  }
  if (one_cta) {
    ensure_smem_attr(k_jacobi_svd.fn(), c->device, int(js_smem(JS_MAX_N)));
    launch(c, k_jacobi_svd, 1, JK_THREADS, js_smem(n), int(n), A, int(lda), U, S, VT, trans,
           c->d_err + 3, c->jacobi_max_sweeps);
    TTG_CHECK_LAUNCH();
    return;
  }
  DBuf<double> V(c, n * n), work(c, n * n + 2 * n);
  if (block) {
    // Block-cyclic grid-wide rounds: one CTA per block pair.
    const size_t bsm = sizeof(double) * 4 * JB_W * size_t(n);
    ensure_smem_attr(k_jacobi_block.fn(), c->device, int(bsm));
    int occ = 0;
    TTG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jacobi_block.plain(),
                                                           JB_THREADS, bsm));
    const int64_t bpairs = ((n + JB_W - 1) / JB_W + 1) / 2;
    const int blocks = int(std::max<int64_t>(
        1, std::min<int64_t>(bpairs, int64_t(c->num_sms) * std::max(occ, 1))));
    DBuf<unsigned> bar(c, 2);
    DBuf<unsigned long long> offmax(c, 3);
    memset_async(c, bar.p(), 0, 2 * sizeof(unsigned));
    launch(c, k_jacobi_block, blocks, JB_THREADS, bsm, int(n), A, int(lda), work.p(), V.p(),
           bar.p(), offmax.p(), c->d_err + 0, c->d_err + 3, trans, c->jacobi_max_sweeps);
    launch(c, k_jacobi_finish, 1, SD_THREADS, 0, int(n), work.p(), V.p(), U, S, VT,
           work.p() + int64_t(n) * n, trans);
    TTG_CHECK_LAUNCH();
    return;
  }
  // Grid-wide rounds: one CTA per column pair (up to what fits at once).
  int occ = 0;
  TTG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jacobi_coop.plain(), JC_THREADS,
                                                         0));
  const int64_t pairs = (n + 1) / 2;
  const int blocks =
      int(std::max<int64_t>(1, std::min<int64_t>(pairs, int64_t(c->num_sms) * occ)));
  DBuf<unsigned> bar(c, 2);
  DBuf<unsigned long long> offmax(c, 3);
  memset_async(c, bar.p(), 0, 2 * sizeof(unsigned));
  launch(c, k_jacobi_coop, blocks, JC_THREADS, 0, int(n), A, int(lda), work.p(), V.p(), bar.p(),
         offmax.p(), c->d_err + 0, c->d_err + 3, trans, c->jacobi_max_sweeps);
  launch(c, k_jacobi_finish, 1, SD_THREADS, 0, int(n), work.p(), V.p(), U, S, VT,
         work.p() + int64_t(n) * n, trans);
  TTG_CHECK_LAUNCH();
}

namespace {
__global__ void k_selftest_jc_barrier(unsigned* bar, int* flag, long long limit) {
  if (blockIdx.x != 0) return;
  jc_barrier(blockIdx, gridDim, bar, flag, limit);
}
}  // namespace

// Self-test of the bounded barrier of the cooperative Jacobi SVD: block 1
// never arrives; block 0 gives up after `limit` polls and raises *flag.
void selftest_wait_jacobi(Context* c, int* flag, long long limit) {
  DBuf<unsigned> bar(c, 2);
  TTG_CUDA(cudaMemsetAsync(bar.p(), 0, 2 * sizeof(unsigned), c->stream));
  k_selftest_jc_barrier<<<2, 32, 0, c->stream>>>(bar.p(), flag, limit);
  TTG_CHECK_LAUNCH();
  sync(c);
}

}  // namespace ttg
