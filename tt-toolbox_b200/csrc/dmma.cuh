// FP64 tensor-core (DMMA) and cp.async helpers shared by the FP64 kernels.
#pragma once
#include <cstdint>

namespace ttg {

// 8-byte async global->shared copy; pred == false writes zeros.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool pred) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  int bytes = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
// 16-byte async global->shared copy of the first `bytes` (0, 8 or 16), zeros
// in the rest; both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// {c0,c1} += a * b for one 8x8x4 FP64 tile fragment (row.col).
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int TILE_K = 16;  // k extent of the FP64 operand tiles

// One operand tile of T rows (of C) by TILE_K in shared memory, filled by NT
// threads in the order of its global layout: k contiguous (KC) as rows of
// TILE_K + 4, else k slices of T + 4.  Either pitch is 4 mod 16 doubles, which puts the 16 doubles that a
// half-warp reads for an mma fragment (4 of k by 4 rows) in different banks.
template <int T, bool KC, int NT>
struct TileS {
  static constexpr int LD = KC ? TILE_K + 4 : T + 4;
  static constexpr int SIZE = KC ? T * LD : TILE_K * LD;
  static __device__ __forceinline__ double at(const double* s, int r, int k) {
    return KC ? s[r * LD + k] : s[k * LD + r];
  }
  // Rows r0.. of R, k0.. of K of the operand g (element (r, k) at
  // g[k + r ld] or g[r + k ld]); zeros outside.
  static __device__ __forceinline__ void load(double* s, const double* __restrict__ g, int64_t ld,
                                              int64_t r0, int64_t R, int64_t k0, int64_t K,
                                              bool vec) {
    const int tid = threadIdx.x;
    if (KC) {
      if (vec) {
        const int k = (tid & 7) * 2, rb = tid >> 3;
        const int64_t left = K - (k0 + k);
        const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
#pragma unroll
        for (int i = 0; i < TILE_K * T / (2 * NT); ++i) {
          const int r = rb + NT / (TILE_K / 2) * i;
          const bool ok = bytes && r0 + r < R;
          cp_async16(s + r * LD + k, ok ? g + (k0 + k) + (r0 + r) * ld : g, ok ? bytes : 0);
        }
      } else {
        const int k = tid & 15, rb = tid >> 4;
        const bool kok = k0 + k < K;
#pragma unroll
        for (int i = 0; i < TILE_K * T / NT; ++i) {
          const int r = rb + NT / TILE_K * i;
          const bool ok = kok && r0 + r < R;
          cp_async8(s + r * LD + k, ok ? g + (k0 + k) + (r0 + r) * ld : g, ok);
        }
      }
    } else {
      if (vec) {
        const int r = (tid % (T / 2)) * 2, kb = tid / (T / 2);
        const int64_t left = R - (r0 + r);
        const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
#pragma unroll
        for (int i = 0; i < TILE_K * T / (2 * NT); ++i) {
          const int k = kb + 2 * NT / T * i;
          const bool ok = bytes && k0 + k < K;
          cp_async16(s + k * LD + r, ok ? g + (r0 + r) + (k0 + k) * ld : g, ok ? bytes : 0);
        }
      } else {
        const int r = tid % T, kb = tid / T;
        const bool rok = r0 + r < R;
#pragma unroll
        for (int i = 0; i < TILE_K * T / NT; ++i) {
          const int k = kb + NT / T * i;
          const bool ok = rok && k0 + k < K;
          cp_async8(s + k * LD + r, ok ? g + (r0 + r) + (k0 + k) * ld : g, ok);
        }
      }
    }
  }
};

// An operand whose columns (or rows, k contiguous) all start on 16 bytes.
inline bool vec16(const double* p, int64_t ld, int64_t stride = 0, int64_t batch = 1) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 2 == 0 &&
         (batch == 1 || stride % 2 == 0);
}

}  // namespace ttg
