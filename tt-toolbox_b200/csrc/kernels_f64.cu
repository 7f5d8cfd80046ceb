// FP64 kernels: DMMA-tiled batched GEMM, deterministic reductions,
// transposes and elementwise helpers.
//
// The GEMM is the contraction engine of the FP64 (parity) path: every local
// matvec (bfun3) and every interface update (compute_next_Phi) is written as
// three batched column-major GEMMs whose operand layouts need no explicit
// permutations (see local_ops.cu).  CTA tiles of 64x64, 32x64 or 32x32 by 16,
// four warps, each warp issuing mma.sync.m8n8k4 f64 (the FP64 tensor path;
// tcgen05 has no FP64 kind, and the larger mma shapes run at the same rate).
// Global->shared staging with cp.async through a ring of three tiles, 16-byte
// granules where the operand's alignment allows, else 8-byte ones.
#include "group.cuh"
#include "kernels.h"
#include "dmma.cuh"

namespace ttg {

namespace {

constexpr int GEMM_STAGES = 3, GEMM_THREADS = 128;
// Split-K partial values one CTA may sum in the GEMM kernel itself.
constexpr int64_t SPLITK_INKERNEL_MAX = 8192;

struct GemmP {
  int64_t M, N, K;
  const double* A;
  int64_t lda, sA;
  const double* B;
  int64_t ldb, sB;
  double* C;
  int64_t ldc, sC;
  double alpha, beta;
  const int* skip;  // optional: return at once when *skip != 0
  int vecA, vecB;   // operand admits 16-byte loads (see vec16)
  // Split-K: nsplit > 1 slices of kc columns of K per batch item, blockIdx.z =
  // item * nsplit + slice.  Each slice writes its partial tile to `part`
  // ([item][slice] blocks of M x N, ld M).  With `cnt` (one arrival counter
  // per tile and item) the slice that arrives last at its tile adds the
  // partials in slice order (deterministic), applies alpha/beta, writes C and
  // resets the counter; without it k_splitk_reduce does the same afterwards.
  int64_t nsplit, kc;
  double* part;
  unsigned* cnt;
};

template <int BM, int BN, bool TA, bool TB>
constexpr size_t gemm_smem() {
  return sizeof(double) * GEMM_STAGES *
         (TileS<BM, TA, GEMM_THREADS>::SIZE + TileS<BN, !TB, GEMM_THREADS>::SIZE);
}

// Bound by the FP64 tensor rate where the tiles fill the device, by the chain
// of launch, first loads and last stores where there are few.  Local matvec
// (three products), measured against pitches of 72 (8-way bank conflicts on k-
// contiguous stores), two stages, 8-byte copies and 64 x 64 tiles only:
// 20 x 32 x 20 19.3 us / 28.0; 61 x 64 x 67 48 / 59; 128 x 64 x 128 138 / 184
// (20.5 TFLOP/s); 187 x 64 x 203 368 / 440; 512 x 64 x 512 3.92 / 4.66 ms (31
// TFLOP/s).  Four stages, eight warps per tile and the larger mma shapes
// measure the same or slower.
template <int BM, int BN, bool TA, bool TB>
__device__ __forceinline__ void gemm_body(TTG_BLOCK, const GemmP& p) {
  pdl_begin();
  extern __shared__ __align__(16) double gsm[];
  constexpr int NT = GEMM_THREADS;
  using SA = TileS<BM, TA, NT>;
  using SB = TileS<BN, !TB, NT>;
  constexpr int MI = BM / 16, NI = BN / 16;  // 8 x 8 fragments of a warp
  if (p.skip && *p.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool split = p.nsplit > 1;
  const int64_t item = split ? blockIdx.z / p.nsplit : blockIdx.z;
  const int64_t slice = split ? blockIdx.z % p.nsplit : 0;
  const int64_t kb0 = slice * p.kc;
  const double* __restrict__ A = p.A + item * p.sA + (TA ? kb0 : kb0 * p.lda);
  const double* __restrict__ B = p.B + item * p.sB + (TB ? kb0 * p.ldb : kb0);
  const int64_t K = split ? min(p.K - kb0, p.kc) : p.K;
  const int64_t m0 = int64_t(blockIdx.x) * BM, n0 = int64_t(blockIdx.y) * BN;
  const int64_t M = p.M, N = p.N;

  double acc[MI][NI][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp & 1) * (BM / 2), wn = (warp >> 1) * (BN / 2);
  const int ktiles = int((K + TILE_K - 1) / TILE_K);
  auto load_tile = [&](int kt) {
    if (kt < ktiles) {
      double* s = gsm + (kt % GEMM_STAGES) * (SA::SIZE + SB::SIZE);
      SA::load(s, A, p.lda, m0, M, int64_t(kt) * TILE_K, K, p.vecA);
      SB::load(s + SA::SIZE, B, p.ldb, n0, N, int64_t(kt) * TILE_K, K, p.vecB);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < GEMM_STAGES - 1; ++s) load_tile(s);
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_async_wait<GEMM_STAGES - 2>();
    __syncthreads();  // tile kt has landed, tile kt - 1 is read out
    load_tile(kt + GEMM_STAGES - 1);
    const double* As = gsm + (kt % GEMM_STAGES) * (SA::SIZE + SB::SIZE);
    const double* Bs = As + SA::SIZE;
    // Fragments of the next k slice are read while the mma of this one run.
    double a[2][MI], b[2][NI];
    auto frag = [&](int kk) {
#pragma unroll
      for (int i = 0; i < MI; ++i) a[kk & 1][i] = SA::at(As, wm + i * 8 + g, kk * 4 + t);
#pragma unroll
      for (int j = 0; j < NI; ++j) b[kk & 1][j] = SB::at(Bs, wn + j * 8 + g, kk * 4 + t);
    };
    frag(0);
#pragma unroll
    for (int kk = 0; kk < TILE_K / 4; ++kk) {
      if (kk + 1 < TILE_K / 4) frag(kk + 1);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
          dmma(acc[i][j][0], acc[i][j][1], a[kk & 1][i], b[kk & 1][j]);
    }
  }

  double* __restrict__ C = p.C + item * p.sC;
  if (!split) {
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int64_t row = m0 + wm + i * 8 + g;
      if (row >= M) continue;
#pragma unroll
      for (int j = 0; j < NI; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int64_t col = n0 + wn + j * 8 + 2 * t + e;
          if (col < N) {
            double* dst = C + row + col * p.ldc;
            double v = p.alpha * acc[i][j][e];
            if (p.beta != 0.0) v += p.beta * *dst;
            *dst = v;
          }
        }
      }
    }
    return;
  }

  // Split-K: publish this slice's partial tile, then the last slice to
  // arrive reduces the tile.
  const int64_t MN = M * N;
  double* Pme = p.part + blockIdx.z * MN;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int64_t row = m0 + wm + i * 8 + g;
    if (row >= M) continue;
#pragma unroll
    for (int j = 0; j < NI; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t col = n0 + wn + j * 8 + 2 * t + e;
        if (col < N) Pme[row + col * M] = acc[i][j][e];
      }
    }
  }
  if (!p.cnt) return;
  __threadfence();
  __syncthreads();
  __shared__ int s_last;
  if (tid == 0) {
    unsigned* ctr = p.cnt + item * (int64_t(gridDim.x) * gridDim.y) + blockIdx.x +
                    int64_t(gridDim.x) * blockIdx.y;
    const unsigned prev = atomicAdd(ctr, 1u);
    s_last = prev == unsigned(p.nsplit - 1);
    if (s_last) *ctr = 0u;  // every slice has arrived: ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // The last slice: every thread sums its elements over the slices in slice
  // order, its loads of one slice in flight together.
  const double* P0 = p.part + item * p.nsplit * MN;
  constexpr int EPT = BM * BN / NT < 8 ? BM * BN / NT : 8;
  for (int e0 = tid; e0 < BM * BN; e0 += NT * EPT) {
    double acc2[EPT];
    bool ok[EPT];
    int64_t off[EPT];
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
      const int e = e0 + q * NT;
      const int64_t row = m0 + e % BM, col = n0 + e / BM;
      ok[q] = row < M && col < N;
      off[q] = ok[q] ? row + col * M : 0;
      acc2[q] = 0.0;
    }
    for (int64_t z = 0; z < p.nsplit; ++z)
#pragma unroll
      for (int q = 0; q < EPT; ++q) acc2[q] += __ldcg(P0 + z * MN + off[q]);
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
      if (!ok[q]) continue;
      const int e = e0 + q * NT;
      double* dst = C + (m0 + e % BM) + (n0 + e / BM) * p.ldc;
      double v = p.alpha * acc2[q];
      if (p.beta != 0.0) v += p.beta * *dst;
      *dst = v;
    }
  }
}
template <int BM, int BN, bool TA, bool TB>
TTG_BODY(k_gemm_f64)(TTG_BLOCK, GemmP p) {
  gemm_body<BM, BN, TA, TB>(blockIdx, gridDim, p);
}
template <int BM, int BN, bool TA, bool TB>
TTG_KERNEL_T(k_gemm_f64, GEMM_THREADS, BM, BN, TA, TB);

// Two independent products in one launch: the first n1 blocks are the first
// product's grid g1, the others the second's.  For chains of short products
// that run side by side (the left and right sweeps of a gradient), which are
// bound by each launch's chain of first loads, k loop and stores: sharing the
// launches takes the gradient of <x, A x> at d = 12, n = 32, rank 64 from 696 to
// 580 us (six cores of 8, rank 16: 167 to 128; twenty of 4, rank 24: 514 to 366).
// 189-190 registers a thread with 32 x 32 tiles, 212-214 with 32 x 64, 255 with
// 64 x 64: at 128, with more CTAs on an SM, the first of these takes 646 us (the
// others 129 and 361).
template <int BM, int BN, bool TA1, bool TB1, bool TA2, bool TB2>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    k_gemm_pair(GemmP p, GemmP q, dim3 g1, dim3 g2) {
  pdl_begin();
  const unsigned n1 = g1.x * g1.y * g1.z;
  const bool first = blockIdx.x < n1;
  const unsigned b = first ? blockIdx.x : blockIdx.x - n1;
  const dim3 g = first ? g1 : g2;
  const uint3 at = {b % g.x, b / g.x % g.y, b / (g.x * g.y)};
  if (first)
    gemm_body<BM, BN, TA1, TB1>(at, g, p);
  else
    gemm_body<BM, BN, TA2, TB2>(at, g, q);
}

// ---------------------------------------------------------------------------
// Reductions
// ---------------------------------------------------------------------------

constexpr int RED_THREADS = 256;
constexpr int RED_MAX_BLOCKS = 1024;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
    r = warp_sum(r);
  }
  return r;  // valid in thread 0
}

// mode 0: sum x*y ; mode 1: sum x^2 ; mode 2: sum (x-y)^2.
// Per-block partial sums; the last block to finish adds the partials in
// block order (deterministic) and writes the result: one launch.  `counter` is a
// device int that is zero between reductions (reset by the last block).
TTG_BODY(k_reduce_fused)(TTG_BLOCK, int64_t n, const double* __restrict__ x,
                               const double* __restrict__ y, int mode, double* __restrict__ part,
                               unsigned* counter, double* out, int do_sqrt) {
  pdl_begin();
  __shared__ double sh[32];
  __shared__ bool last;
  double s = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const double a = x[i];
    if (mode == 0)
      s += a * y[i];
    else if (mode == 1)
      s += a * a;
    else {
      const double dlt = a - y[i];
      s += dlt * dlt;
    }
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < int(gridDim.x); i += blockDim.x)
    t += reinterpret_cast<volatile const double*>(part)[i];
  t = block_sum(t, sh);
  if (threadIdx.x == 0) {
    *out = do_sqrt ? sqrt(t) : t;
    *counter = 0u;
  }
}
TTG_KERNEL(k_reduce_fused, 0);

void reduce_launch(Context* c, int64_t n, const double* x, const double* y, int mode,
                   double* out, bool do_sqrt) {
  int nb = int(std::min<int64_t>((n + RED_THREADS * 4 - 1) / (RED_THREADS * 4), RED_MAX_BLOCKS));
  if (nb < 1) nb = 1;
  DBuf<double> part(c, nb);
  launch(c, k_reduce_fused, nb, RED_THREADS, 0, n, x, y, mode, part.p(),
         reinterpret_cast<unsigned*>(c->d_err + 63), out, do_sqrt ? 1 : 0);
  TTG_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// Elementwise
// ---------------------------------------------------------------------------

TTG_BODY(k_count_nonfinite)(TTG_BLOCK, int64_t n, const double* __restrict__ x,
                                  unsigned long long* __restrict__ out) {
  pdl_begin();
  unsigned long long cnt = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    cnt += isfinite(x[i]) ? 0ull : 1ull;
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(out, cnt);
}
TTG_KERNEL(k_count_nonfinite, 0);

TTG_BODY(k_axpby)(TTG_BLOCK, int64_t n, double a, const double* __restrict__ x, double b,
                        double* __restrict__ y) {
  pdl_begin();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    y[i] = (b == 0.0 ? 0.0 : b * y[i]) + a * x[i];
}
TTG_KERNEL(k_axpby, 0);

TTG_BODY(k_scale_dev)(TTG_BLOCK, int64_t n, const double* __restrict__ x, double* __restrict__ y,
                            const double* num, const double* den) {
  pdl_begin();
  const double s = (num ? *num : 1.0) / (den ? *den : 1.0);
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    y[i] = x[i] * s;
}
TTG_KERNEL(k_scale_dev, 0);

TTG_BODY(k_copy)(TTG_BLOCK, int64_t n, const double* __restrict__ x, double* __restrict__ y) {
  pdl_begin();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    y[i] = x[i];
}
TTG_KERNEL(k_copy, 0);

TTG_BODY(k_fill)(TTG_BLOCK, int64_t n, double v, double* y) {
  pdl_begin();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    y[i] = v;
}
TTG_KERNEL(k_fill, 0);

TTG_BODY(k_transpose)(TTG_BLOCK, int64_t rows, int64_t cols, const double* __restrict__ in,
                            int64_t ldi, int64_t si, double* __restrict__ out, int64_t ldo,
                            int64_t so) {
  pdl_begin();
  __shared__ double tile[32][33];
  const int64_t b = blockIdx.z;
  in += b * si;
  out += b * so;
  const int64_t r0 = int64_t(blockIdx.x) * 32, c0 = int64_t(blockIdx.y) * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int64_t r = r0 + threadIdx.x, cc = c0 + j;
    if (r < rows && cc < cols) tile[j][threadIdx.x] = in[r + cc * ldi];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int64_t cc = c0 + threadIdx.x, r = r0 + j;
    if (r < rows && cc < cols) out[cc + r * ldo] = tile[threadIdx.x][j];
  }
}
TTG_KERNEL(k_transpose, 0);

TTG_BODY(k_copy2d)(TTG_BLOCK, int64_t rows, int64_t cols, const double* __restrict__ in, int64_t ldi,
                         double* __restrict__ out, int64_t ldo, const double* scale_col) {
  pdl_begin();
  const int64_t total = rows * cols;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = i % rows, cidx = i / rows;
    double v = in[r + cidx * ldi];
    if (scale_col) v *= scale_col[cidx];
    out[r + cidx * ldo] = v;
  }
}
TTG_KERNEL(k_copy2d, 0);

// splitmix64-based counter hash -> two uniforms -> Box-Muller normal.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

TTG_BODY(k_randn)(TTG_BLOCK, int64_t n, uint64_t seed, uint64_t offset, double* y) {
  pdl_begin();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const uint64_t h1 = mix64(seed ^ mix64(2 * (offset + i)));
    const uint64_t h2 = mix64(seed ^ mix64(2 * (offset + i) + 1));
    const double u1 = (double((h1 >> 11) + 1)) * (1.0 / 9007199254740993.0);
    const double u2 = double(h2 >> 11) * (1.0 / 9007199254740992.0);
    y[i] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
  }
}
TTG_KERNEL(k_randn, 0);

TTG_BODY(k_normalize_by)(TTG_BLOCK, int64_t n, double* __restrict__ x, double* nrm) {
  pdl_begin();
  const double v = *nrm;
  const double s = v > 0.0 ? 1.0 / v : 1.0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    x[i] *= s;
  // Every block has read *nrm above; a zero norm is reported as 1.
  if (blockIdx.x == 0 && threadIdx.x == 0 && !(v > 0.0)) *nrm = 1.0;
}
TTG_KERNEL(k_normalize_by, 0);

TTG_BODY(k_axpby_dev)(TTG_BLOCK, int64_t n, double a, const double* __restrict__ x,
                            const double* __restrict__ b, double* __restrict__ y) {
  pdl_begin();
  const double bv = *b;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    y[i] = bv * y[i] + a * x[i];
}
TTG_KERNEL(k_axpby_dev, 0);

TTG_BODY(k_scalar_op)(TTG_BLOCK, int op, double* out, const double* p0, const double* p1,
                            const double* p2, double k) {
  pdl_begin();
  switch (op) {
    case 0: *out = *p0 / *p1; break;
    case 1: *out = fmax(*out, *p0); break;
    case 2: *out = *out / (*p0 / (*p1 * *p2)); break;
    case 3: *out = *out * (*p0 / (*p1 * *p2)); break;
    case 4: *out = *out * *p0; break;
    case 5: *out = fmax(*p0, k); break;
    case 6: *out = (*p1 > 0.0) ? *p0 / *p1 : 0.0; break;
    case 7: *out = (*p0 == 0.0) ? 1.0 : *p0; break;
    default: break;
  }
}
TTG_KERNEL(k_scalar_op, 0);

TTG_BODY(k_first_exceeding)(TTG_BLOCK, int64_t nb, const double* cand, const double* den,
                                  const double* thr, double* out) {
  pdl_begin();
  double r = -1.0;
  for (int64_t b = 0; b < nb; ++b) {
    if (cand[b] / *den > *thr) {
      r = double(b);
      break;
    }
  }
  *out = r;
}
TTG_KERNEL(k_first_exceeding, 0);

// C_b = alpha * sum_z part[b][z] + beta * C_b over the split-K slices, in
// slice order (deterministic).  part: batch x s blocks of M x N (ld M).
TTG_BODY(k_splitk_reduce)(TTG_BLOCK, int64_t M, int64_t N, int64_t s, int64_t batch,
                                const double* __restrict__ part, double alpha, double beta,
                                double* __restrict__ C, int64_t ldc, int64_t sC,
                                const int* skip) {
  pdl_begin();
  if (skip && *skip) return;
  const int64_t MN = M * N;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < MN * batch;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t b = e / MN, r = e % MN;
    const double* src = part + b * s * MN + r;
    double acc = 0.0;
    for (int64_t z = 0; z < s; ++z) acc += src[z * MN];
    const int64_t m = r % M, n = r / M;
    double* dst = C + b * sC + m + n * ldc;
    double v = alpha * acc;
    if (beta != 0.0) v += beta * *dst;
    *dst = v;
  }
}
TTG_KERNEL(k_splitk_reduce, 0);

// *keep = 1 when every column j kept G1[j,j] > tau^2 G0[j,j] (one thread).
TTG_BODY(k_collapse_flag)(TTG_BLOCK, int64_t k, const double* G0, int64_t ld0, const double* G1,
                                int64_t ld1, double tau, int* keep) {
  pdl_begin();
  int ok = 1;
  for (int64_t j = 0; j < k; ++j)
    if (!(G1[j + j * ld1] > tau * tau * G0[j + j * ld0])) ok = 0;
  *keep = ok;
}
TTG_KERNEL(k_collapse_flag, 0);

// *flag |= 1 when max |G - I| > tol (G: n x n Gram matrix of a basis).  Columns
// over blocks, rows over threads.
TTG_BODY(k_orth_check)(TTG_BLOCK, int64_t n, const double* G, double tol, int* flag) {
  pdl_begin();
  int bad = 0;
  for (int64_t j = blockIdx.x; j < n; j += gridDim.x)
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      const double v = G[i + j * n] - (i == j ? 1.0 : 0.0);
      if (!(fabs(v) <= tol)) bad = 1;
    }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}
TTG_KERNEL(k_orth_check, 0);

TTG_BODY(k_accumulate_info)(TTG_BLOCK, const int* info, int* err_slot) {
  pdl_begin();
  if (*info != 0) atomicOr(err_slot, 1);
}
TTG_KERNEL(k_accumulate_info, 0);

int grid_for(Context* c, int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = int64_t(c->num_sms) * 8;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return int(b);
}

template <int BM, int BN, bool TA, bool TB>
void gemm_launch(Context* c, dim3 grid, const GemmP& p) {
  constexpr size_t smem = gemm_smem<BM, BN, TA, TB>();
  if (smem > 48 * 1024) ensure_smem_attr(k_gemm_f64<BM, BN, TA, TB>.fn(), c->device, int(smem));
  launch(c, k_gemm_f64<BM, BN, TA, TB>, grid, GEMM_THREADS, smem, p);
}

template <int BM, int BN>
void gemm_launch(Context* c, bool tA, bool tB, dim3 grid, const GemmP& p) {
  if (!tA && !tB)
    gemm_launch<BM, BN, false, false>(c, grid, p);
  else if (!tA && tB)
    gemm_launch<BM, BN, false, true>(c, grid, p);
  else if (tA && !tB)
    gemm_launch<BM, BN, true, false>(c, grid, p);
  else
    gemm_launch<BM, BN, true, true>(c, grid, p);
}

struct GemmTile {
  int bm, bn;
  double cost;  // relative time per tile element
};
constexpr GemmTile GEMM_TILES[] = {{64, 64, 1.0}, {32, 64, 1.1}, {32, 32, 1.25}};

struct GemmPlan {
  GemmTile tile;
  int64_t gx, gy, split, kc;
};

// CTA tile and number of K slices: the pair with the least estimated time, in
// cycles.  An SM multiplies a 64 x 64 x 16 step in 1024 cycles (m8n8k4 at 37
// TFLOP/s on the device) whichever of its CTAs issues it, so the product takes
// the work of the fullest SM, tile edges that hang over the matrix included;
// a smaller tile costs more per element (it loads more operand per product),
// and an SM with fewer than four CTAs leaves the pipe idle between their steps.
// Slices add their partials, written once and read once, and either the
// last CTA's sum or a second kernel.  Interface update with this rule, against
// split-K to two 64 x 64 CTAs per SM: 61 x 64 x 67 54 / 83 us, 128 x 64 x 128
// 136 / 216, 512 x 64 x 512 4.4 / 8.0 ms.
// `sms`: the SMs the product may count on; `only`: plan for this tile; partials
// of one tile stay within `most`.
GemmPlan plan_gemm(int64_t sms, int64_t M, int64_t N, int64_t K, int64_t batch, bool may_split,
                   const GemmTile* only = nullptr, int64_t most = INT64_MAX) {
  const int64_t ktiles = (K + TILE_K - 1) / TILE_K;
  GemmPlan best{};
  double best_t = 0.0;
  for (const GemmTile& t : GEMM_TILES) {
    const int64_t gx = (M + t.bm - 1) / t.bm, gy = (N + t.bn - 1) / t.bn, ctas = gx * gy * batch;
    if (only && only->bm * only->bn != t.bm * t.bn) continue;
    if (!only && &t != GEMM_TILES && (gy > 65535 || gx > 0x7fffffff)) continue;  // the grid's limits
    int64_t smax = 1;
    if (may_split && ctas < 4 * sms && ktiles >= 8 && ctas <= GEMM_TILE_COUNTERS)
      smax = std::min({ktiles / 4, 8 * sms / ctas + 1, 65535 / batch});
    int64_t prev = 0;
    for (int64_t s = 1; s <= smax; s = s < 8 ? s + 1 : s + s / 4) {
      const int64_t kt = (ktiles + s - 1) / s, ns = (ktiles + kt - 1) / kt;
      if (ns == prev) continue;
      prev = ns;
      const int64_t per_sm = (ctas * ns + sms - 1) / sms;
      const double idle = per_sm == 1 ? 2.2 : per_sm == 2 ? 1.45 : per_sm == 3 ? 1.15 : 1.0;
      double est = double(per_sm * kt) * (t.bm * t.bn / 4) * t.cost * idle;
      if (ns > 1) {
        if (ns * std::min<int64_t>(M, t.bm) * std::min<int64_t>(N, t.bn) > most) break;
        const int64_t te = std::min<int64_t>(M, t.bm) * std::min<int64_t>(N, t.bn);
        est += 16.0 * double(ns * M * N * batch) / 2600.0 +
               (ns * te <= SPLITK_INKERNEL_MAX ? 2500.0 : 4500.0);
      }
      if (best_t == 0.0 || est < best_t) {
        best = GemmPlan{t, gx, gy, ns, kt * TILE_K};
        best_t = est;
      }
    }
  }
  return best;
}

}  // namespace

void gemm_f64(Context* c, bool tA, bool tB, int64_t M, int64_t N, int64_t K, double alpha,
              const double* A, int64_t lda, int64_t sA, const double* B, int64_t ldb, int64_t sB,
              double beta, double* C, int64_t ldc, int64_t sC, int64_t batch) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  if (K <= 0) {
    // C = beta*C
    for (int64_t b = 0; b < batch; ++b) {
      if (beta == 0.0) {
        for (int64_t j = 0; j < N; ++j) fill_f64(c, M, 0.0, C + b * sC + j * ldc);
      } else if (beta != 1.0) {
        for (int64_t j = 0; j < N; ++j) axpby_f64(c, M, 0.0, C + b * sC + j * ldc, beta, C + b * sC + j * ldc);
      }
    }
    return;
  }
  TTG_REQUIRE(batch <= 65535, "gemm batch %lld too large", (long long)batch);
  TTG_REQUIRE((N + 63) / 64 <= 65535 && (M + 63) / 64 <= 0x7fffffff, "gemm too large");
  // Split-K cuts a long K into slices of at least 4 k-tiles where the output
  // tiles leave SMs idle (inner products of tall matrices: interface updates,
  // Gram matrices, projections).  The slices of a tile are summed in slice
  // order: by the last slice to finish when the partials are few (no second
  // launch), else by a reduction kernel spread over the device (one CTA
  // reading many partials is latency-bound).
  // (A context without an allocator -- the caller-scratch entry point -- runs
  // every product unsplit.)
  const GemmPlan pl = plan_gemm(c->num_sms, M, N, K, batch, c->alloc && c->d_tile_cnt);
  GemmP p{M,  N,     K,       A,  lda, sA, B, ldb, sB, C, ldc, sC, alpha, beta, c->skip,
          vec16(A, lda, sA, batch), vec16(B, ldb, sB, batch), 1, 0, nullptr, nullptr};
  dim3 grid{unsigned(pl.gx), unsigned(pl.gy), unsigned(batch * pl.split)};
  DBuf<double> part;
  if (pl.split > 1) {
    part.reset(c, batch * pl.split * M * N);
    p.nsplit = pl.split;
    p.kc = pl.kc;
    p.part = part.p();
    const int64_t te = std::min<int64_t>(M, pl.tile.bm) * std::min<int64_t>(N, pl.tile.bn);
    if (pl.split * te <= SPLITK_INKERNEL_MAX) p.cnt = c->d_tile_cnt;
  }
  if (pl.tile.bm == 64)
    gemm_launch<64, 64>(c, tA, tB, grid, p);
  else if (pl.tile.bn == 64)
    gemm_launch<32, 64>(c, tA, tB, grid, p);
  else
    gemm_launch<32, 32>(c, tA, tB, grid, p);
  TTG_CHECK_LAUNCH();
  if (p.nsplit > 1 && !p.cnt) {
    launch(c, k_splitk_reduce, grid_for(c, M * N * batch), 256, 0, M, N, p.nsplit, batch,
           part.p(), alpha, beta, C, ldc, sC, c->skip);
    TTG_CHECK_LAUNCH();
  }
}

namespace {

template <int BM, int BN, bool TA1, bool TB1, bool TA2, bool TB2>
void pair_launch(Context* c, const GemmP& p, const GemmP& q, dim3 g1, dim3 g2) {
  constexpr size_t s1 = gemm_smem<BM, BN, TA1, TB1>(), s2 = gemm_smem<BM, BN, TA2, TB2>();
  constexpr size_t smem = s1 > s2 ? s1 : s2;
  const void* fn = reinterpret_cast<const void*>(k_gemm_pair<BM, BN, TA1, TB1, TA2, TB2>);
  if (smem > 48 * 1024) ensure_smem_attr(fn, c->device, int(smem));
  const unsigned blocks = g1.x * g1.y * g1.z + g2.x * g2.y * g2.z;
  launch(c, k_gemm_pair<BM, BN, TA1, TB1, TA2, TB2>, blocks, GEMM_THREADS, smem, p, q, g1, g2);
  TTG_CHECK_LAUNCH();
}

// Partials of one tile that the last slice of a pair sums: 12 slices of 32 x 32.
// The first gradient above takes 656, 593, 580, 622 us with 4, 8, 12, 16 (one CTA
// reads them); d = 8, n = 24, rank 50 285, 274, 273, 273; six cores of 8, rank 16,
// d = 8, n = 16, rank 32 and ranks from 128 on do not move by more than 2% (rank
// 128 with 4: 8%).
constexpr int64_t PAIR_SPLITK_MAX = 12288;
// Work of the two products up to which they share a launch: 7 us at the FP64
// tensor rate, about a launch's own chain.  Longer ones fill the device by
// themselves, with more CTAs on an SM than the pair kernel's registers leave:
// gradient of <x, A x>, shared / apart, d = 12, n = 32, rank 64 (150 MFLOP a
// pair) 580 / 696 us, d = 10, n = 32, rank 80 (130) 594 / 632; d = 6, n = 32, rank
// 100, operator rank 3 (380) 643 / 610; d = 5, n = 64, rank 128 (1600) 1194 /
// 1172; d = 4, n = 48, rank 200 (3100) 1513 / 1235.
constexpr double PAIR_FLOP_MAX = 256e6;

template <bool TA1, bool TB1, bool TA2, bool TB2>
bool pair_f64(Context* c, const GemmOp& a, const GemmOp& b) {
  if (c->rec || !c->alloc || !c->d_tile_cnt) return false;
  for (const GemmOp* o : {&a, &b})  // gemm_f64 refuses these
    if (o->batch > 65535 || (o->N + 63) / 64 > 65535 || (o->M + 63) / 64 > 0x7fffffff) return false;
  auto flop = [](const GemmOp& o) { return 2.0 * double(o.M) * double(o.N) * double(o.K) * double(o.batch); };
  if (flop(a) + flop(b) > PAIR_FLOP_MAX) return false;
  // Each product plans for half the device, with the first one's tile, and
  // sums its slices in the kernel.
  const int64_t sms = std::max(1, c->num_sms / 2);
  const GemmPlan pa = plan_gemm(sms, a.M, a.N, a.K, a.batch, true, nullptr, PAIR_SPLITK_MAX);
  const GemmPlan pb = plan_gemm(sms, b.M, b.N, b.K, b.batch, true, &pa.tile, PAIR_SPLITK_MAX);
  const int64_t ta = pa.gx * pa.gy * a.batch, tb = pb.gx * pb.gy * b.batch;
  // (products of more tiles than counters fill the device one by one)
  if (ta * pa.split + tb * pb.split > 0x7fffffff || ta + tb > GEMM_TILE_COUNTERS) return false;
  DBuf<double> part1, part2;
  auto params = [&](const GemmOp& o, const GemmPlan& pl, DBuf<double>& part, unsigned* cnt) {
    GemmP p{o.M,   o.N,     o.K,   o.A,  o.lda, o.sA,   o.B,     o.ldb,    o.sB,
            o.C,   o.ldc,   o.sC,  1.0,  o.beta, c->skip, vec16(o.A, o.lda, o.sA, o.batch),
            vec16(o.B, o.ldb, o.sB, o.batch), 1, 0, nullptr, nullptr};
    if (pl.split > 1) {
      part.reset(c, o.batch * pl.split * o.M * o.N);
      p.nsplit = pl.split;
      p.kc = pl.kc;
      p.part = part.p();
      p.cnt = cnt;
    }
    return p;
  };
  const GemmP p = params(a, pa, part1, c->d_tile_cnt), q = params(b, pb, part2, c->d_tile_cnt + ta);
  const dim3 g1{unsigned(pa.gx), unsigned(pa.gy), unsigned(a.batch * pa.split)};
  const dim3 g2{unsigned(pb.gx), unsigned(pb.gy), unsigned(b.batch * pb.split)};
  if (pa.tile.bm == 64)
    pair_launch<64, 64, TA1, TB1, TA2, TB2>(c, p, q, g1, g2);
  else if (pa.tile.bn == 64)
    pair_launch<32, 64, TA1, TB1, TA2, TB2>(c, p, q, g1, g2);
  else
    pair_launch<32, 32, TA1, TB1, TA2, TB2>(c, p, q, g1, g2);
  return true;
}

}  // namespace

void gemm_pair_f64(Context* c, const GemmOp& a, const GemmOp& b) {
  bool done = false;
  if (a.M > 0 && a.N > 0 && a.K > 0 && a.batch > 0 && b.M > 0 && b.N > 0 && b.K > 0 &&
      b.batch > 0) {
    if (a.tA && !a.tB && !b.tA && !b.tB) done = pair_f64<true, false, false, false>(c, a, b);
    if (!a.tA && !a.tB && !b.tA && b.tB) done = pair_f64<false, false, false, true>(c, a, b);
    if (a.tA && !a.tB && !b.tA && b.tB) done = pair_f64<true, false, false, true>(c, a, b);
  }
  if (done) return;
  for (const GemmOp* o : {&a, &b})
    gemm_f64(c, o->tA, o->tB, o->M, o->N, o->K, 1.0, o->A, o->lda, o->sA, o->B, o->ldb, o->sB,
             o->beta, o->C, o->ldc, o->sC, o->batch);
}

void dot_f64(Context* c, int64_t n, const double* x, const double* y, double* out, bool do_sqrt) {
  reduce_launch(c, n, x, y, y ? 0 : 1, out, do_sqrt);
}

void diffnrm_f64(Context* c, int64_t n, const double* x, const double* y, double* out,
                 bool do_sqrt) {
  reduce_launch(c, n, x, y, 2, out, do_sqrt);
}

double nrm2_host(Context* c, int64_t n, const double* x) {
  DBuf<double> s(c, 1);
  dot_f64(c, n, x, nullptr, s.p(), true);
  double h = 0.0;
  read_scalars(c, s.p(), &h, 1);
  return h;
}

int64_t count_nonfinite_f64(Context* c, int64_t n, const double* x) {
  if (n <= 0) return 0;
  DBuf<unsigned long long> cnt(c, 1);
  memset_async(c, cnt.p(), 0, sizeof(unsigned long long));
  launch(c, k_count_nonfinite, grid_for(c, n), 256, 0, n, x, cnt.p());
  TTG_CHECK_LAUNCH();
  unsigned long long h = 0;
  read_device(c, &h, cnt.p(), sizeof(h));
  return int64_t(h);
}

void require_finite(const ttg_tt_s* t, const char* name) {
  if (!t) return;
  require_finite(t->ctx, {{t, name}});
}

void require_finite(Context* c, std::initializer_list<std::pair<const ttg_tt_s*, const char*>> ts) {
  const int64_t k = int64_t(ts.size());
  DBuf<unsigned long long> cnt(c, k);
  memset_async(c, cnt.p(), 0, sizeof(unsigned long long) * k);
  int64_t j = 0;
  for (const auto& t : ts) {
    if (t.first && t.first->numel > 0)
      launch(c, k_count_nonfinite, grid_for(c, t.first->numel), 256, 0, t.first->numel,
             t.first->core, cnt.p() + j);
    ++j;
  }
  TTG_CHECK_LAUNCH();
  unsigned long long h[16] = {};
  TTG_REQUIRE(k <= 16, "require_finite: too many tensors");
  read_device(c, h, cnt.p(), sizeof(unsigned long long) * k);  // one read for all
  j = 0;
  for (const auto& t : ts) {
    TTG_REQUIRE(h[j] == 0, "%s holds %lld non-finite entries (NaN or Inf)", t.second,
                (long long)h[j]);
    ++j;
  }
}

void axpby_f64(Context* c, int64_t n, double a, const double* x, double b, double* y) {
  if (n <= 0) return;
  launch(c, k_axpby, grid_for(c, n), 256, 0, n, a, x, b, y);
  TTG_CHECK_LAUNCH();
}

void scale_dev_f64(Context* c, int64_t n, const double* x, double* y, const double* num,
                   const double* den) {
  if (n <= 0) return;
  launch(c, k_scale_dev, grid_for(c, n), 256, 0, n, x, y, num, den);
  TTG_CHECK_LAUNCH();
}

void fill_f64(Context* c, int64_t n, double v, double* y) {
  if (n <= 0) return;
  launch(c, k_fill, grid_for(c, n), 256, 0, n, v, y);
  TTG_CHECK_LAUNCH();
}

void copy_f64(Context* c, int64_t n, const double* x, double* y) {
  if (n <= 0 || x == y) return;
  // a kernel rather than a memcpy node, so that it chains with its
  // neighbours as a programmatic dependent launch
  launch(c, k_copy, grid_for(c, n), 256, 0, n, x, y);
  TTG_CHECK_LAUNCH();
}

void transpose_f64(Context* c, int64_t rows, int64_t cols, const double* in, int64_t ldi,
                   double* out, int64_t ldo, int64_t batch, int64_t si, int64_t so) {
  if (rows <= 0 || cols <= 0 || batch <= 0) return;
  TTG_REQUIRE((cols + 31) / 32 <= 65535 && batch <= 65535, "transpose too large");
  dim3 grid{unsigned((rows + 31) / 32), unsigned((cols + 31) / 32), unsigned(batch)};
  launch(c, k_transpose, grid, dim3(32, 8), 0, rows, cols, in, ldi, si, out, ldo, so);
  TTG_CHECK_LAUNCH();
}

void copy2d_f64(Context* c, int64_t rows, int64_t cols, const double* in, int64_t ldi,
                double* out, int64_t ldo, const double* scale_col) {
  if (rows <= 0 || cols <= 0) return;
  launch(c, k_copy2d, grid_for(c, rows * cols), 256, 0, rows, cols, in, ldi, out, ldo,
         scale_col);
  TTG_CHECK_LAUNCH();
}

void normalize_by_dev(Context* c, int64_t n, double* x, double* nrm) {
  if (n <= 0) return;
  launch(c, k_normalize_by, grid_for(c, n), 256, 0, n, x, nrm);
  TTG_CHECK_LAUNCH();
}

void axpby_dev(Context* c, int64_t n, double a, const double* x, const double* b, double* y) {
  if (n <= 0) return;
  launch(c, k_axpby_dev, grid_for(c, n), 256, 0, n, a, x, b, y);
  TTG_CHECK_LAUNCH();
}

void scalar_op(Context* c, int op, double* out, const double* p0, const double* p1,
               const double* p2, double k) {
  launch(c, k_scalar_op, 1, 1, 0, op, out, p0, p1, p2, k);
  TTG_CHECK_LAUNCH();
}

void first_exceeding(Context* c, int64_t nb, const double* cand, const double* den,
                     const double* thr, double* out) {
  launch(c, k_first_exceeding, 1, 1, 0, nb, cand, den, thr, out);
  TTG_CHECK_LAUNCH();
}

void collapse_flag(Context* c, int64_t k, const double* G0, int64_t ld0, const double* G1,
                   int64_t ld1, double tau, int* keep) {
  launch(c, k_collapse_flag, 1, 1, 0, k, G0, ld0, G1, ld1, tau, keep);
  TTG_CHECK_LAUNCH();
}

void orth_check(Context* c, int64_t n, const double* G, double tol, int* flag) {
  launch(c, k_orth_check, unsigned(std::min<int64_t>((n + 3) / 4, c->num_sms)), 128, 0, n, G, tol,
         flag);
  TTG_CHECK_LAUNCH();
}

void accumulate_info(Context* c, const int* info, int* err_slot) {
  launch(c, k_accumulate_info, 1, 1, 0, info, err_slot);
  TTG_CHECK_LAUNCH();
}

void randn_f64(Context* c, int64_t n, uint64_t seed, uint64_t offset, double* y) {
  if (n <= 0) return;
  launch(c, k_randn, grid_for(c, n), 256, 0, n, seed, offset, y);
  TTG_CHECK_LAUNCH();
}

}  // namespace ttg
