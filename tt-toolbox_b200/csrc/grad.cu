// Gradients of three TT functionals with respect to every core (FP64).
//
// TT-Toolbox has no derivative code.  The forward maps are its own:
//   <x, A x>  : @tt_matrix/mtimes.m:38-65 (A x) and @tt_tensor/dot.m:92-111
//   <x, b>    : @tt_tensor/dot.m:92-111 (left-to-right interface sweep)
//   X[idx_s]  : @tt_tensor/subsref.m:93-123 (an entry is the product of the
//               core slices x_k(:, i_k, :))
// A TT functional is multilinear in the cores, so the gradient with respect
// to core k is the functional with core k removed: the interfaces left and
// right of k contracted with everything that touched core k.
//
// <x, A x>: the interfaces are those of AMEn's local system (compute_next_Phi,
//   solve/amen_solve2.m:834-920, without its normalisation), L_k [bra, ket, ra]
//   from the left and R_k [ket, ra, bra] from the right.  The derivative
//   through the bra copy of x_k is the local matvec bfun3
//   (solve/amen_solve2.m:924-951) L_k x A_k x R_{k+1} applied to x_k, whose
//   first two products are those of the update of R_k: it takes one product
//   more in the right sweep.  The derivative through the ket copy, likewise,
//   is the left update's last intermediate, W2_k, times R_{k+1}.
// <x, b>:   two interface sweeps Psi_L [rx, rb], Psi_R [rx, rb]; three GEMMs
//   per core.
// sum_s (X[idx_s] - y_s)^2: per sample s, the row vector l_k(s) = product of
//   the slices left of k and the column vector rho_k(s) = 2 e_s times the
//   product of the slices right of k, e_s = X[idx_s] - y_s.  The gradient of
//   core k at slice j is sum over samples with i_k = j of l_k(s)^T rho_k(s)^T.
//   Samples are bucketed by i_k (stable counting sort, deterministic), and
//   every product becomes a gathered GEMM on the FP64 tensor cores: the CTA
//   owns 128 samples of one bucket, stages their vectors (gathered rows) and
//   the bucket's slice in shared memory and multiplies with mma.m8n8k4.  The
//   gradient is a split-K GEMM per bucket (512 samples per CTA) whose
//   partials are summed in a fixed order, so results are bitwise repeatable.
#include "grad.h"
#include "dmma.cuh"
#include "kernels.h"

namespace ttg {

namespace {

constexpr int PT = 128;          // samples per propagation tile
constexpr int PROP_THREADS = 256, GRAD_THREADS = 128, GRAD_STAGES = 3;
// Bytes of intermediates that <x, A x> keeps between its sweeps and the gradient.
constexpr int64_t KEEP_MAX = int64_t(2) << 30;
constexpr int GT = 512;          // samples per gradient (split-K) tile
constexpr int SORT_CHUNK = 1024; // samples per sorting warp
constexpr int64_t MAX_BUCKETS = 8192;

int blocks_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return int(b < 1 ? 1 : (b > 65535 * 16 ? 65535 * 16 : b));
}

// ---------------------------------------------------------------------------
// Sample bucketing (stable counting sort of one index column)
// ---------------------------------------------------------------------------

// err |= 1 when some idx[s + k*S] is outside [0, n_k).
__global__ void k_check_idx(int64_t S, int d, const int* __restrict__ idx,
                            const int64_t* __restrict__ nk, int* err) {
  const int64_t total = S * d;
  for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
       t += int64_t(gridDim.x) * blockDim.x) {
    const int v = idx[t];
    if (v < 0 || v >= nk[t / S]) atomicOr(err, 1);
  }
}

__device__ __forceinline__ int clamp_bucket(int v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// counts[j * nblk + b] = #samples of chunk b with idx = j.  One warp per chunk.
__global__ void k_bucket_count(int64_t S, const int* __restrict__ col, int n, int nblk,
                               int* __restrict__ counts) {
  extern __shared__ int sh_cnt[];
  for (int j = threadIdx.x; j < n; j += 32) sh_cnt[j] = 0;
  __syncwarp();
  const int64_t s0 = int64_t(blockIdx.x) * SORT_CHUNK;
  const int64_t s1 = min(S, s0 + SORT_CHUNK);
  for (int64_t s = s0 + threadIdx.x; s < s1; s += 32) atomicAdd(&sh_cnt[clamp_bucket(col[s], n)], 1);
  __syncwarp();
  for (int j = threadIdx.x; j < n; j += 32) counts[int64_t(j) * nblk + blockIdx.x] = sh_cnt[j];
}

// Exclusive scan of counts[j * nblk + (0..nblk-1)] in place; total[j].
__global__ void k_bucket_scan(int nblk, int* __restrict__ counts, int* __restrict__ total) {
  __shared__ int sh[256];
  __shared__ int carry;
  int* row = counts + int64_t(blockIdx.x) * nblk;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nblk; base += 256) {
    const int i = base + threadIdx.x;
    const int v = i < nblk ? row[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {  // Hillis-Steele inclusive scan
      const int add = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += add;
      __syncthreads();
    }
    if (i < nblk) row[i] = carry + sh[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 255) carry += sh[255];
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// Bucket starts and the tile tables of both tilings (one thread; n is small).
//   meta[0 .. n]            bucket start (meta[n] = S)
//   meta[n+1 .. 2n+1]       first propagation tile of each bucket (+ total)
//   meta[2n+2 .. 3n+2]      first gradient tile of each bucket (+ total)
__global__ void k_bucket_base(int n, const int* __restrict__ total, int* __restrict__ meta) {
  int s = 0, tp = 0, tg = 0;
  for (int j = 0; j < n; ++j) {
    meta[j] = s;
    meta[n + 1 + j] = tp;
    meta[2 * n + 2 + j] = tg;
    const int cnt = total[j];
    s += cnt;
    tp += (cnt + PT - 1) / PT;
    tg += (cnt + GT - 1) / GT;
  }
  meta[n] = s;
  meta[2 * n + 1] = tp;
  meta[3 * n + 2] = tg;
}

// perm[bucket_start[j] + offs[j*nblk+b] + rank] = s, stable within buckets.
__global__ void k_bucket_scatter(int64_t S, const int* __restrict__ col, int n, int nblk,
                                 const int* __restrict__ offs, const int* __restrict__ meta,
                                 int* __restrict__ perm) {
  extern __shared__ int sh_cnt[];
  for (int j = threadIdx.x; j < n; j += 32) sh_cnt[j] = 0;
  __syncwarp();
  const int lane = threadIdx.x;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t s0 = int64_t(blockIdx.x) * SORT_CHUNK;
  const int64_t s1 = min(S, s0 + SORT_CHUNK);
  for (int64_t sb = s0; sb < s1; sb += 32) {
    const int64_t s = sb + lane;
    const bool valid = s < s1;
    const int v = valid ? clamp_bucket(col[s], n) : n + lane;  // invalid lanes: own groups
    const unsigned same = __match_any_sync(0xffffffffu, v);
    const int rank = __popc(same & lt);
    const int before = valid ? sh_cnt[v] : 0;
    __syncwarp();
    if (valid) {
      perm[int64_t(meta[v]) + offs[int64_t(v) * nblk + blockIdx.x] + before + rank] = int(s);
      if (rank == 0) sh_cnt[v] = before + __popc(same);
    }
    __syncwarp();
  }
}

// Bucket j of tile t: the largest j with start[j] <= t (start has n+1 entries).
__device__ __forceinline__ int find_bucket(const int* __restrict__ start, int n, int t) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// Gathered propagation GEMM
//   forward  (BWD=false): vout[s, c] = sum_a vin[s, a] * x_k[a, j, c]
//   backward (BWD=true):  vout[s, a] = sum_c x_k[a, j, c] * vin[s, c]
// for every sample s of bucket j (i_k(s) = j).  Sample vectors are rows:
// v[s * ld + a].  CTA = 128 samples x BN outputs, eight warps of 32 x BN / 2,
// K in steps of 16 through a ring of three tiles (the pitches and copies of
// TileS).  Bound by the FP64 tensor rate next to reading and writing one
// vector per sample: 1M samples, 64 x 64 slices 279 us forward, 280 backward
// (29 TFLOP/s with 3.7 TB/s), against 493 and 426 with 64 samples a CTA, two
// stages, 8-byte copies and conflicting pitches.
// ---------------------------------------------------------------------------
struct PropP {
  const double* vin;
  int64_t ldi;
  double* vout;
  int64_t ldo;
  const double* core;
  int64_t r1, n, r2;
  int64_t K, N;
  const int* perm;
  const int* meta;  // bucket table (k_bucket_base layout)
  int vecA, vecB, vecC;  // 16-byte accesses of vin, of the slices and of vout
};

template <int BN, bool BWD>
constexpr size_t prop_smem() {
  return sizeof(double) * GRAD_STAGES *
             (TileS<PT, true, PROP_THREADS>::SIZE + TileS<BN, !BWD, PROP_THREADS>::SIZE) +
         sizeof(int64_t) * PT;
}

template <int BN, bool BWD>
__global__ void __launch_bounds__(PROP_THREADS) k_prop(PropP p) {
  using SA = TileS<PT, true, PROP_THREADS>;
  using SB = TileS<BN, !BWD, PROP_THREADS>;
  constexpr int NI = BN / 16;
  extern __shared__ __align__(16) double psm[];
  int64_t* rowoff = reinterpret_cast<int64_t*>(psm + GRAD_STAGES * (SA::SIZE + SB::SIZE));
  const int nb = int(p.n);
  const int* bstart = p.meta;
  const int* tstart = p.meta + nb + 1;
  const int t = blockIdx.x;
  if (t >= tstart[nb]) return;
  const int j = find_bucket(tstart, nb, t);
  const int64_t s0 = int64_t(bstart[j]) + int64_t(t - tstart[j]) * PT;
  const int64_t cnt = min(int64_t(PT), int64_t(bstart[j + 1]) - s0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < PT) rowoff[tid] = tid < cnt ? int64_t(p.perm[s0 + tid]) : -1;
  __syncthreads();
  const double* __restrict__ W = p.core + p.r1 * j;
  const int64_t ldw = p.r1 * p.n;
  const int64_t n0 = int64_t(blockIdx.y) * BN;
  const int64_t K = p.K, N = p.N;
  const int ktiles = int((K + TILE_K - 1) / TILE_K);

  auto load_tile = [&](int kt) {
    if (kt < ktiles) {
      double* sa = psm + (kt % GRAD_STAGES) * (SA::SIZE + SB::SIZE);
      const int64_t k0 = int64_t(kt) * TILE_K;
      // A(m, k) = vin[rowoff[m] * ldi + k]   (k contiguous)
      if (p.vecA) {
        const int k = (tid & 7) * 2, mb = tid >> 3;
        const int64_t left = K - (k0 + k);
        const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
#pragma unroll
        for (int i = 0; i < PT * 8 / PROP_THREADS; ++i) {
          const int m = mb + PROP_THREADS / 8 * i;
          const int64_t ro = rowoff[m];
          const bool ok = bytes && ro >= 0;
          cp_async16(sa + m * SA::LD + k, ok ? p.vin + ro * p.ldi + k0 + k : p.vin,
                     ok ? bytes : 0);
        }
      } else {
        const int k = tid & 15, mb = tid >> 4;
#pragma unroll
        for (int i = 0; i < PT * 16 / PROP_THREADS; ++i) {
          const int m = mb + PROP_THREADS / 16 * i;
          const int64_t ro = rowoff[m];
          const bool ok = ro >= 0 && k0 + k < K;
          cp_async8(sa + m * SA::LD + k, ok ? p.vin + ro * p.ldi + k0 + k : p.vin, ok);
        }
      }
      // forward B(k=a, n=c) = W[a + c*ldw], backward B(k=c, n=a) = W[a + c*ldw]
      SB::load(sa + SA::SIZE, W, ldw, n0, N, k0, K, p.vecB);
    }
    cp_async_commit();
  };

  double acc[4][NI][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int jj = 0; jj < NI; ++jj) acc[i][jj][0] = acc[i][jj][1] = 0.0;

  const int g = lane >> 2, tq = lane & 3;
  const int wm = (warp & 3) * 32, wn = (warp >> 2) * (BN / 2);
#pragma unroll
  for (int s = 0; s < GRAD_STAGES - 1; ++s) load_tile(s);
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_async_wait<GRAD_STAGES - 2>();
    __syncthreads();
    load_tile(kt + GRAD_STAGES - 1);
    const double* As = psm + (kt % GRAD_STAGES) * (SA::SIZE + SB::SIZE);
    const double* Bs = As + SA::SIZE;
#pragma unroll
    for (int kk = 0; kk < TILE_K / 4; ++kk) {
      double a[4], b[NI];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = SA::at(As, wm + i * 8 + g, kk * 4 + tq);
#pragma unroll
      for (int jj = 0; jj < NI; ++jj) b[jj] = SB::at(Bs, wn + jj * 8 + g, kk * 4 + tq);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int jj = 0; jj < NI; ++jj) dmma(acc[i][jj][0], acc[i][jj][1], a[i], b[jj]);
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t ro = rowoff[wm + i * 8 + g];
    if (ro < 0) continue;
    double* dst = p.vout + ro * p.ldo;
#pragma unroll
    for (int jj = 0; jj < NI; ++jj) {
      const int64_t col = n0 + wn + jj * 8 + 2 * tq;
      if (p.vecC && col + 1 < N) {
        *reinterpret_cast<double2*>(dst + col) = make_double2(acc[i][jj][0], acc[i][jj][1]);
      } else {
        if (col < N) dst[col] = acc[i][jj][0];
        if (col + 1 < N) dst[col + 1] = acc[i][jj][1];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Gradient partials: part[t][a + r1*c] = sum over the <= 512 samples s of
// gradient tile t of L[s, a] * P[s, c]   (M = r1, N = r2, K = samples)
// The same ring; 1M samples, 64 x 64: 283 us (315 before).
// ---------------------------------------------------------------------------
struct GradP {
  const double* L;
  int64_t ldl;
  const double* P;
  int64_t ldp;
  double* part;
  int64_t r1, n, r2;
  const int* perm;
  const int* meta;
  int vecA, vecB;
};

template <int BM, int BN>
constexpr size_t grad_smem() {
  return sizeof(double) * GRAD_STAGES *
             (TileS<BM, false, GRAD_THREADS>::SIZE + TileS<BN, false, GRAD_THREADS>::SIZE) +
         sizeof(int64_t) * GT;
}

// Columns x0.. of the gathered rows k0.. of v into an operand tile (zeros
// outside): s[k * LD + x] = v[rowoff[k0 + k] * ld + x0 + x].
template <int T>
__device__ __forceinline__ void load_gathered(double* s, const double* __restrict__ v, int64_t ld,
                                              const int64_t* rowoff, int64_t x0, int64_t X,
                                              int k0, int K, bool vec) {
  constexpr int LD = TileS<T, false, GRAD_THREADS>::LD;
  const int tid = threadIdx.x;
  if (vec) {
    const int x = (tid % (T / 2)) * 2, kb = tid / (T / 2);
    const int64_t left = X - (x0 + x);
    const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
#pragma unroll
    for (int i = 0; i < TILE_K * T / (2 * GRAD_THREADS); ++i) {
      const int k = kb + 2 * GRAD_THREADS / T * i;
      const bool ok = bytes && k0 + k < K;
      cp_async16(s + k * LD + x, ok ? v + rowoff[k0 + k] * ld + x0 + x : v, ok ? bytes : 0);
    }
  } else {
    const int x = tid % T, kb = tid / T;
    const bool xok = x0 + x < X;
#pragma unroll
    for (int i = 0; i < TILE_K * T / GRAD_THREADS; ++i) {
      const int k = kb + GRAD_THREADS / T * i;
      const bool ok = xok && k0 + k < K;
      cp_async8(s + k * LD + x, ok ? v + rowoff[k0 + k] * ld + x0 + x : v, ok);
    }
  }
}

template <int BM, int BN>
__global__ void __launch_bounds__(GRAD_THREADS) k_grad_tiles(GradP p) {
  using SA = TileS<BM, false, GRAD_THREADS>;
  using SB = TileS<BN, false, GRAD_THREADS>;
  constexpr int MI = BM / 16, NI = BN / 16;
  extern __shared__ __align__(16) double gtsm[];
  int64_t* rowoff = reinterpret_cast<int64_t*>(gtsm + GRAD_STAGES * (SA::SIZE + SB::SIZE));
  const int nb = int(p.n);
  const int* bstart = p.meta;
  const int* gstart = p.meta + 2 * nb + 2;
  const int t = blockIdx.x;
  if (t >= gstart[nb]) return;
  const int j = find_bucket(gstart, nb, t);
  const int64_t s0 = int64_t(bstart[j]) + int64_t(t - gstart[j]) * GT;
  const int cnt = int(min(int64_t(GT), int64_t(bstart[j + 1]) - s0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < cnt; i += GRAD_THREADS) rowoff[i] = int64_t(p.perm[s0 + i]);
  __syncthreads();
  const int64_t m0 = int64_t(blockIdx.y) * BM, n0 = int64_t(blockIdx.z) * BN;
  const int64_t M = p.r1, N = p.r2;
  const int ktiles = (cnt + TILE_K - 1) / TILE_K;

  auto load_tile = [&](int kt) {
    if (kt < ktiles) {
      double* s = gtsm + (kt % GRAD_STAGES) * (SA::SIZE + SB::SIZE);
      load_gathered<BM>(s, p.L, p.ldl, rowoff, m0, M, kt * TILE_K, cnt, p.vecA);
      load_gathered<BN>(s + SA::SIZE, p.P, p.ldp, rowoff, n0, N, kt * TILE_K, cnt, p.vecB);
    }
    cp_async_commit();
  };

  double acc[MI][NI][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int jj = 0; jj < NI; ++jj) acc[i][jj][0] = acc[i][jj][1] = 0.0;

  const int g = lane >> 2, tq = lane & 3;
  const int wm = (warp & 1) * (BM / 2), wn = (warp >> 1) * (BN / 2);
#pragma unroll
  for (int s = 0; s < GRAD_STAGES - 1; ++s) load_tile(s);
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_async_wait<GRAD_STAGES - 2>();
    __syncthreads();
    load_tile(kt + GRAD_STAGES - 1);
    const double* As = gtsm + (kt % GRAD_STAGES) * (SA::SIZE + SB::SIZE);
    const double* Bs = As + SA::SIZE;
#pragma unroll
    for (int kk = 0; kk < TILE_K / 4; ++kk) {
      double a[MI], b[NI];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i] = SA::at(As, wm + i * 8 + g, kk * 4 + tq);
#pragma unroll
      for (int jj = 0; jj < NI; ++jj) b[jj] = SB::at(Bs, wn + jj * 8 + g, kk * 4 + tq);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int jj = 0; jj < NI; ++jj) dmma(acc[i][jj][0], acc[i][jj][1], a[i], b[jj]);
    }
  }

  double* dst = p.part + int64_t(t) * (p.r1 * p.r2);
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int64_t row = m0 + wm + i * 8 + g;
    if (row >= M) continue;
#pragma unroll
    for (int jj = 0; jj < NI; ++jj) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t col = n0 + wn + jj * 8 + 2 * tq + e;
        if (col < N) dst[row + col * M] = acc[i][jj][e];
      }
    }
  }
}

// grad[a + r1*j + r1*n*c] = sum_{t in gradient tiles of bucket j} part[t][a + r1*c]
// (fixed order; empty buckets give zero slices).
__global__ void k_grad_reduce(int64_t r1, int64_t n, int64_t r2, const double* __restrict__ part,
                              const int* __restrict__ meta, double* __restrict__ grad) {
  const int64_t total = r1 * r2 * n;
  const int* gstart = meta + 2 * n + 2;
  const int64_t R = r1 * r2;
  for (int64_t id = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; id < total;
       id += int64_t(gridDim.x) * blockDim.x) {
    const int64_t ac = id % R;
    const int64_t j = id / R;
    const int64_t a = ac % r1, c = ac / r1;
    double s = 0.0;
    for (int t = gstart[j]; t < gstart[j + 1]; ++t) s += part[int64_t(t) * R + ac];
    grad[a + r1 * j + r1 * n * c] = s;
  }
}

// e = v - y; rho = 2 e.
__global__ void k_sample_residual(int64_t S, const double* __restrict__ v,
                                  const double* __restrict__ y, double* __restrict__ e,
                                  double* __restrict__ rho) {
  for (int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; s < S;
       s += int64_t(gridDim.x) * blockDim.x) {
    const double r = v[s] - y[s];
    e[s] = r;
    rho[s] = 2.0 * r;
  }
}

template <int BN, bool BWD>
void prop_launch(Context* c, int64_t tiles, const PropP& p) {
  constexpr size_t smem = prop_smem<BN, BWD>();
  ensure_smem_attr(reinterpret_cast<const void*>(k_prop<BN, BWD>), c->device, int(smem));
  dim3 grid{unsigned(tiles), unsigned((p.N + BN - 1) / BN), 1};
  k_prop<BN, BWD><<<grid, PROP_THREADS, smem, c->stream>>>(p);
  c->launches += 1;
  TTG_CHECK_LAUNCH();
}

// Outputs up to 32 take the narrow tile: the wide one would multiply padding.
template <bool BWD>
void propagate(Context* c, int64_t tiles, PropP p) {
  p.vecA = vec16(p.vin, p.ldi);
  p.vecB = vec16(p.core, p.r1);  // slices start r1 apart
  p.vecC = vec16(p.vout, p.ldo);
  if (p.N <= 32)
    prop_launch<32, BWD>(c, tiles, p);
  else
    prop_launch<64, BWD>(c, tiles, p);
}

template <int BM, int BN>
void grad_launch(Context* c, int64_t tiles, const GradP& p) {
  constexpr size_t smem = grad_smem<BM, BN>();
  ensure_smem_attr(reinterpret_cast<const void*>(k_grad_tiles<BM, BN>), c->device, int(smem));
  dim3 grid{unsigned(tiles), unsigned((p.r1 + BM - 1) / BM), unsigned((p.r2 + BN - 1) / BN)};
  k_grad_tiles<BM, BN><<<grid, GRAD_THREADS, smem, c->stream>>>(p);
  c->launches += 1;
  TTG_CHECK_LAUNCH();
}

void check_tt_vector(const ttg_tt_s* x, const char* what) {
  TTG_REQUIRE(x && !x->is_matrix, "%s must be a TT tensor", what);
  TTG_REQUIRE(x->r[0] == 1 && x->r[x->d] == 1, "%s: boundary ranks must be 1", what);
}

}  // namespace

// ---------------------------------------------------------------------------
// <x, A x>: eight products per core (three each way for the interfaces, two
// for the gradient), shared by the two sweeps two to a launch where they are
// short.  Bound by the chain of 49 dependent launches of 11-12 us: d = 12, n = 32,
// rank 64 580 us, against 1151 us with two whole local matvecs and three
// permutations per core and 696 us with one launch per product.
// ---------------------------------------------------------------------------
void grad_xAx(Context* c, const ttg_tt_s* x, const ttg_tt_s* A, double* grad, double* value) {
  check_tt_vector(x, "x");
  TTG_REQUIRE(A && A->is_matrix, "A must be a TT matrix");
  const int64_t d = x->d;
  TTG_REQUIRE(A->d == d, "A has %lld cores, x has %lld", (long long)A->d, (long long)d);
  TTG_REQUIRE(A->r[0] == 1 && A->r[d] == 1, "A: boundary ranks must be 1");
  for (int64_t k = 0; k < d; ++k)
    TTG_REQUIRE(A->n[k] == x->n[k] && A->m[k] == x->n[k],
                "core %lld: A is %lldx%lld, x has mode size %lld", (long long)k,
                (long long)A->n[k], (long long)A->m[k], (long long)x->n[k]);
  const auto& r = x->r;
  const auto& ra = A->r;
  // Interfaces L[k] [r_k, r_k, ra_k] and R[k] [r_k, ra_k, r_k], k = 0..d, and the
  // second products of every core's updates, W2 and Z2.
  std::vector<int64_t> off(d + 2, 0), woff(d + 1, 0), zoff(d + 1, 0);
  int64_t w1max = 1, z1max = 1;
  for (int64_t k = 0; k <= d; ++k) off[k + 1] = off[k] + r[k] * r[k] * ra[k];
  for (int64_t k = 0; k < d; ++k) {
    const int64_t w2 = r[k] * x->n[k] * ra[k + 1] * r[k + 1],
                  z2 = r[k] * ra[k] * x->n[k] * r[k + 1];
    woff[k + 1] = woff[k] + w2;
    zoff[k + 1] = zoff[k] + z2;
    w1max = std::max(w1max, z2);
    z1max = std::max(z1max, w2);
  }
  DBuf<double> L(c, off[d + 1]), R(c, off[d + 1]);
  DBuf<double> W1, Z1, W2, Z2;
  bool keep = false;
  auto W1p = [&] { return keep ? W1.p() : Z2.p(); };
  auto Z1p = [&] { return keep ? Z1.p() : W2.p(); };
  auto W2k = [&](int64_t k) { return W2.p() + (keep ? woff[k] : 0); };
  auto Z2k = [&](int64_t k) { return Z2.p() + (keep ? zoff[k] : 0); };
  fill_f64(c, 1, 1.0, L.p());
  fill_f64(c, 1, 1.0, R.p() + off[d]);
  // left: W1[(y,al),(j,c)] = L_k^T x, W2_c[y,(m,be)] = W1_c[y,(al,j)] A[(al,j),(m,be)],
  //       L_{k+1},be [c, e] = W2[(y,m), be, c]^T x[(y,m), e]
  // right: Z1[(y,m),(be,c)] = x R_{k+1}, Z2_c[y,(al,j)] = Z1_c[y,(m,be)] A[(al,j),(m,be)]^T,
  //       R_k[(y,al), a] = Z2[(y,al),(j,c)] x[a,(j,c)]^T
  // gradient through the bra copy: G[a,(j,c)] = L_k[a,(y,al)] Z2[(y,al),(j,c)],
  //       through the ket copy: G[(y,m), e] += W2[(y,m),(be,c)] R_{k+1}[e,(be,c)]^T
  enum { LEFT1, LEFT2, LEFT3, RIGHT1, RIGHT2, RIGHT3, BRA, KET };
  auto op = [&](int which, int64_t k) -> GemmOp {
    const int64_t r1 = r[k], r2 = r[k + 1], a1 = ra[k], a2 = ra[k + 1], n = x->n[k];
    const double* xk = x->core + x->ps[k];
    const double* Ak = A->core + A->ps[k];
    double* gk = grad + x->ps[k];
    const double* Lk = L.p() + off[k];
    const double* Rn = R.p() + off[k + 1];
    switch (which) {
      case LEFT1:
        return {true, false, r1 * a1, n * r2, r1, Lk, r1, 0, xk, r1, 0, 0.0, W1p(), r1 * a1, 0, 1};
      case LEFT2:
        return {false, false, r1, n * a2, a1 * n, W1p(), r1, r1 * a1 * n, Ak, a1 * n, 0, 0.0,
                W2k(k), r1, r1 * n * a2, r2};
      case LEFT3:
        return {true, false, r2, r2, r1 * n, W2k(k), r1 * n * a2, r1 * n, xk, r1 * n, 0, 0.0,
                L.p() + off[k + 1], r2, r2 * r2, a2};
      case RIGHT1:
        return {false, false, r1 * n, a2 * r2, r2, xk, r1 * n, 0, Rn, r2, 0, 0.0, Z1p(), r1 * n,
                0, 1};
      case RIGHT2:
        return {false, true, r1, a1 * n, n * a2, Z1p(), r1, r1 * n * a2, Ak, a1 * n, 0, 0.0,
                Z2k(k), r1, r1 * a1 * n, r2};
      case RIGHT3:
        return {false, true, r1 * a1, r1, n * r2, Z2k(k), r1 * a1, 0, xk, r1, 0, 0.0,
                R.p() + off[k], r1 * a1, 0, 1};
      case BRA:
        return {false, false, r1, n * r2, r1 * a1, Lk, r1, 0, Z2k(k), r1 * a1, 0, 0.0, gk, r1, 0,
                1};
      default:
        return {false, true, r1 * n, r2, a2 * r2, W2k(k), r1 * n, 0, Rn, r2, 0, 1.0, gk, r1 * n, 0,
                1};
    }
  };
  auto one = [&](int which, int64_t k) {
    const GemmOp o = op(which, k);
    gemm_f64(c, o.tA, o.tB, o.M, o.N, o.K, 1.0, o.A, o.lda, o.sA, o.B, o.ldb, o.sB, o.beta, o.C,
             o.ldc, o.sC, o.batch);
  };
  // Every core's W2 and Z2 are kept between the sweeps and the gradient, and
  // the sweeps then run side by side.
  auto side_by_side = [&] {
    keep = true;
    W1.reset(c, w1max);
    Z1.reset(c, z1max);
    W2.reset(c, woff[d]);
    Z2.reset(c, zoff[d]);
    for (int64_t k = 0; k < d; ++k) {
      const int64_t l = d - 1 - k;
      gemm_pair_f64(c, op(LEFT1, k), op(RIGHT1, l));
      gemm_pair_f64(c, op(LEFT2, k), op(RIGHT2, l));
      if (l > 0)
        gemm_pair_f64(c, op(LEFT3, k), op(RIGHT3, l));
      else
        one(LEFT3, k);
    }
    for (int64_t k = 0; k <= d; ++k) {  // a core's ket product follows its bra product
      if (k == 0)
        one(BRA, 0);
      else if (k < d)
        gemm_pair_f64(c, op(BRA, k), op(KET, k - 1));
      else
        one(KET, d - 1);
    }
  };
  // The right sweep follows the left one and forms W2 again: two buffers of
  // the largest core, W1 in Z2's and Z1 in W2's.
  auto one_by_one = [&] {
    keep = false;
    for (DBuf<double>* b : {&W1, &Z1, &W2, &Z2}) b->release();
    W2.reset(c, z1max);
    Z2.reset(c, w1max);
    for (int64_t k = 0; k < d; ++k)
      for (int which : {LEFT1, LEFT2, LEFT3}) one(which, k);
    for (int64_t k = d - 1; k >= 0; --k) {
      for (int which : {RIGHT1, RIGHT2, BRA}) one(which, k);
      if (k > 0) one(RIGHT3, k);
      for (int which : {LEFT1, LEFT2, KET}) one(which, k);
    }
  };
  // Side by side up to KEEP_MAX, where the device has the memory for it.
  bool done = false;
  if ((woff[d] + zoff[d]) * int64_t(sizeof(double)) <= KEEP_MAX) {
    try {
      side_by_side();
      done = true;
    } catch (const Error& e) {
      if (e.code != TTG_ERR_ALLOC) throw;
    }
  }
  if (!done) one_by_one();
  if (value) copy_f64(c, 1, L.p() + off[d], value);
}

// ---------------------------------------------------------------------------
// <x, b>
// ---------------------------------------------------------------------------
void grad_xb(Context* c, const ttg_tt_s* x, const ttg_tt_s* b, double* grad, double* value) {
  check_tt_vector(x, "x");
  check_tt_vector(b, "b");
  const int64_t d = x->d;
  TTG_REQUIRE(b->d == d, "b has %lld cores, x has %lld", (long long)b->d, (long long)d);
  for (int64_t k = 0; k < d; ++k)
    TTG_REQUIRE(b->n[k] == x->n[k], "core %lld: mode sizes differ (%lld vs %lld)", (long long)k,
                (long long)b->n[k], (long long)x->n[k]);
  const auto& r = x->r;
  const auto& rb = b->r;
  std::vector<int64_t> poff(d + 2, 0), toff(d + 1, 0);
  for (int64_t k = 0; k <= d; ++k) poff[k + 1] = poff[k] + r[k] * rb[k];
  for (int64_t k = 0; k < d; ++k) toff[k + 1] = toff[k] + r[k] * x->n[k] * rb[k + 1];
  DBuf<double> PL(c, poff[d + 1]), PR(c, poff[d + 1]), T(c, toff[d]);
  int64_t umax = 1;
  for (int64_t k = 0; k < d; ++k) umax = std::max(umax, rb[k] * x->n[k] * r[k + 1]);
  DBuf<double> U(c, umax);
  fill_f64(c, 1, 1.0, PL.p());
  fill_f64(c, 1, 1.0, PR.p() + poff[d]);
  for (int64_t k = 0; k < d; ++k) {
    const int64_t r1 = r[k], r2 = r[k + 1], q1 = rb[k], q2 = rb[k + 1], n = x->n[k];
    const double* xk = x->core + x->ps[k];
    const double* bk = b->core + b->ps[k];
    double* Tk = T.p() + toff[k];
    // T[a, (i,q)] = Psi_L[a, p] b_k[p, (i,q)]
    gemm_f64(c, false, false, r1, n * q2, q1, 1.0, PL.p() + poff[k], r1, 0, bk, q1, 0, 0.0, Tk,
             r1, 0);
    // Psi_L[k+1][c, q] = sum_{(a,i)} x_k[(a,i), c] T[(a,i), q]
    gemm_f64(c, true, false, r2, q2, r1 * n, 1.0, xk, r1 * n, 0, Tk, r1 * n, 0, 0.0,
             PL.p() + poff[k + 1], r2, 0);
  }
  for (int64_t k = d - 1; k >= 0; --k) {
    const int64_t r1 = r[k], r2 = r[k + 1], q1 = rb[k], q2 = rb[k + 1], n = x->n[k];
    const double* xk = x->core + x->ps[k];
    const double* bk = b->core + b->ps[k];
    const double* PRn = PR.p() + poff[k + 1];
    // gradient: G[(a,i), c] = sum_q T[(a,i), q] Psi_R[k+1][c, q]
    gemm_f64(c, false, true, r1 * n, r2, q2, 1.0, T.p() + toff[k], r1 * n, 0, PRn, r2, 0, 0.0,
             grad + x->ps[k], r1 * n, 0);
    if (k == 0) break;
    // U[(p,i), c] = sum_q b_k[(p,i), q] Psi_R[k+1][c, q]
    gemm_f64(c, false, true, q1 * n, r2, q2, 1.0, bk, q1 * n, 0, PRn, r2, 0, 0.0, U.p(), q1 * n,
             0);
    // Psi_R[k][a, p] = sum_{(i,c)} x_k[a, (i,c)] U[p, (i,c)]
    gemm_f64(c, false, true, r1, q1, n * r2, 1.0, xk, r1, 0, U.p(), q1, 0, 0.0,
             PR.p() + poff[k], r1, 0);
  }
  if (value) copy_f64(c, 1, PL.p() + poff[d], value);
}

// ---------------------------------------------------------------------------
// sum_s (X[idx_s] - y_s)^2
// ---------------------------------------------------------------------------
void grad_sampled(Context* c, const ttg_tt_s* x, int64_t S, const int* idx, const double* y,
                  double* grad, double* value) {
  check_tt_vector(x, "x");
  const int64_t d = x->d;
  const auto& r = x->r;
  TTG_REQUIRE(S >= 0 && S <= int64_t(0x7fffffff) - 1, "sample count %lld out of range",
              (long long)S);
  for (int64_t k = 0; k < d; ++k)
    TTG_REQUIRE(x->n[k] <= MAX_BUCKETS, "mode size %lld above %lld", (long long)x->n[k],
                (long long)MAX_BUCKETS);
  if (S == 0) {
    fill_f64(c, x->numel, 0.0, grad);
    if (value) fill_f64(c, 1, 0.0, value);
    return;
  }
  TTG_REQUIRE(idx && y, "NULL sample arrays");
  // Index range check (one read-back; the sort below clamps as well).
  {
    DBuf<int64_t> nk(c, d);
    DBuf<int> err(c, 1);
    TTG_CUDA(cudaMemcpyAsync(nk.p(), x->n.data(), d * sizeof(int64_t), cudaMemcpyHostToDevice,
                             c->stream));
    TTG_CUDA(cudaMemsetAsync(err.p(), 0, sizeof(int), c->stream));
    k_check_idx<<<blocks_for(S * d), 256, 0, c->stream>>>(S, int(d), idx, nk.p(), err.p());
    c->launches += 1;
    TTG_CHECK_LAUNCH();
    int h = 0;
    TTG_CUDA(cudaMemcpyAsync(&h, err.p(), sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TTG_CUDA(cudaStreamSynchronize(c->stream));
    TTG_REQUIRE(h == 0, "sample index out of range (idx is 0-based, column k in [0, n_k))");
  }
  // Bucketing of every index column.
  const int nblk = int((S + SORT_CHUNK - 1) / SORT_CHUNK);
  int64_t nmax = 1;
  std::vector<int64_t> moff(d + 1, 0);
  for (int64_t k = 0; k < d; ++k) {
    nmax = std::max(nmax, x->n[k]);
    moff[k + 1] = moff[k] + 3 * x->n[k] + 3;
  }
  DBuf<int> perm(c, size_t(S) * d), meta(c, moff[d]), counts(c, size_t(nmax) * nblk),
      total(c, nmax);
  std::vector<int> hmeta(moff[d]);
  for (int64_t k = 0; k < d; ++k) {
    const int n = int(x->n[k]);
    const int* col = idx + k * S;
    k_bucket_count<<<nblk, 32, n * sizeof(int), c->stream>>>(S, col, n, nblk, counts.p());
    k_bucket_scan<<<n, 256, 0, c->stream>>>(nblk, counts.p(), total.p());
    k_bucket_base<<<1, 1, 0, c->stream>>>(n, total.p(), meta.p() + moff[k]);
    k_bucket_scatter<<<nblk, 32, n * sizeof(int), c->stream>>>(S, col, n, nblk, counts.p(),
                                                                meta.p() + moff[k],
                                                                perm.p() + k * S);
    c->launches += 4;
    TTG_CHECK_LAUNCH();
  }
  // Tile counts per core sized the grids; read them once.
  TTG_CUDA(cudaMemcpyAsync(hmeta.data(), meta.p(), moff[d] * sizeof(int), cudaMemcpyDeviceToHost,
                           c->stream));
  TTG_CUDA(cudaStreamSynchronize(c->stream));
  // Left vectors l_k [S x r_k], k = 0..d (l_0 = 1, l_d = the sampled entries).
  std::vector<int64_t> loff(d + 2, 0);
  int64_t rmax = 1;
  for (int64_t k = 0; k <= d; ++k) {
    loff[k + 1] = loff[k] + S * r[k];
    rmax = std::max(rmax, r[k]);
  }
  int64_t partmax = 1;
  for (int64_t k = 0; k < d; ++k) {
    const int n = int(x->n[k]);
    partmax = std::max(partmax, int64_t(hmeta[moff[k] + 3 * n + 2]) * r[k] * r[k + 1]);
  }
  DBuf<double> Lv(c, loff[d + 1]), rho0(c, S * rmax), rho1(c, S * rmax), e(c, S),
      part(c, partmax);
  fill_f64(c, S, 1.0, Lv.p());
  for (int64_t k = 0; k < d; ++k) {
    const int n = int(x->n[k]);
    const int ntiles = hmeta[moff[k] + 2 * n + 1];
    if (ntiles == 0) continue;
    propagate<false>(c, ntiles,
                     PropP{Lv.p() + loff[k], r[k], Lv.p() + loff[k + 1], r[k + 1],
                           x->core + x->ps[k], r[k], x->n[k], r[k + 1], r[k], r[k + 1],
                           perm.p() + k * S, meta.p() + moff[k], 0, 0, 0});
  }
  double* rho = rho0.p();
  double* rho_next = rho1.p();
  k_sample_residual<<<blocks_for(S), 256, 0, c->stream>>>(S, Lv.p() + loff[d], y, e.p(), rho);
  c->launches += 1;
  TTG_CHECK_LAUNCH();
  if (value) dot_f64(c, S, e.p(), nullptr, value);
  for (int64_t k = d - 1; k >= 0; --k) {
    const int n = int(x->n[k]);
    const int ngt = hmeta[moff[k] + 3 * n + 2];
    const int64_t r1 = r[k], r2 = r[k + 1];
    GradP gp{Lv.p() + loff[k], r1, rho, r2, part.p(), r1, x->n[k], r2, perm.p() + k * S,
             meta.p() + moff[k], vec16(Lv.p() + loff[k], r1), vec16(rho, r2)};
    // narrow tiles for ranks up to 32
    if (r1 <= 32 && r2 <= 32)
      grad_launch<32, 32>(c, ngt, gp);
    else if (r1 <= 32)
      grad_launch<32, 64>(c, ngt, gp);
    else if (r2 <= 32)
      grad_launch<64, 32>(c, ngt, gp);
    else
      grad_launch<64, 64>(c, ngt, gp);
    k_grad_reduce<<<blocks_for(r1 * r2 * x->n[k]), 256, 0, c->stream>>>(
        r1, x->n[k], r2, part.p(), meta.p() + moff[k], grad + x->ps[k]);
    c->launches += 1;
    TTG_CHECK_LAUNCH();
    if (k == 0) break;
    const int ntiles = hmeta[moff[k] + 2 * n + 1];
    propagate<true>(c, ntiles,
                    PropP{rho, r2, rho_next, r1, x->core + x->ps[k], r1, x->n[k], r2, r2, r1,
                          perm.p() + k * S, meta.p() + moff[k], 0, 0, 0});
    std::swap(rho, rho_next);
  }
}

}  // namespace ttg
