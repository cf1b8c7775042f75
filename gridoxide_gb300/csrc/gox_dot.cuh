// Interpreter of the dot-product programs (gox_dot.hpp).
//
// What bounds it: the top is a chain of some 400 ticks each way (2,000 buses),
// a tick the latency of a sum (header, its loads, up to 8 dependent
// multiply-adds, for a pivot a reciprocal, 441 cycles in FP64) plus a CTA
// barrier (78 cycles for 32 warps); the bins are bound by the latency of
// their loads and by instructions (about 75 per sum).  Why sums instead of the
// streams' columns: a column's pivot and its L entries run on as many warps
// at once (2.8k cycles per tick with 128 groups against 4.0k per level), no
// ring has to be kept (values are found in the L1: a hit costs 67 cycles, as
// much as an own copy in shared memory would with its bookkeeping), and the
// bottom's columns spread over every SM instead of the group's.
// Why the touches: without them the tail's loads miss the L1 (the top of 128
// groups FP32 takes 1.04 ms, with them 0.70 ms).
// Refactor with both substitutions, streams -> programs, ms: 2,000 buses, 128
// groups FP32 2.15 -> 1.71, 47 groups FP64 5.94 -> 2.26, one group FP32 2.07 ->
// 1.07; 10,000 buses, 128 groups FP32 9.4 -> 6.0; 20,000 buses, one group FP32
// 9.5 -> 4.3; 118 buses, one group FP64 0.41 -> 0.22.
#pragma once
#include "gox_dot.hpp"
#include "gox_kernels.cuh"

namespace gox {

template <typename T>
__device__ __forceinline__ T dot_ld(const char* base, uint32_t row) {
  return *reinterpret_cast<const T*>(base + (size_t)row * (32u * sizeof(T)));
}

// M products at q: every load before the first multiply
template <typename T, int M>
__device__ __forceinline__ void dot_terms(const uint4* q, const char* A, const char* B, T& v) {
  T a[M], b[M];
#pragma unroll
  for (int t = 0; t < M; t += 2) {
    const uint4 e = q[t / 2];
    a[t] = dot_ld<T>(A, e.x);
    b[t] = dot_ld<T>(B, e.y);
    if (t + 1 < M) {
      a[t + 1] = dot_ld<T>(A, e.z);
      b[t + 1] = dot_ld<T>(B, e.w);
    }
  }
#pragma unroll
  for (int t = 0; t < M; t++) v -= a[t] * b[t];
}

// four values into the L1: asynchronous copies (cached at every level) into a
// row of shared memory that nobody reads
template <typename T>
__device__ __forceinline__ void dot_touch(const char* base, const uint4& q, uint32_t sink) {
  const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int t = 0; t < 4; t++)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sink), "l"(base + (size_t)r[t] * (32u * sizeof(T))),
                 "n"((int)sizeof(T)) : "memory");
}

// One warp runs one stream.  win: 64 quads of shared memory, the chunk being
// run and the next one; the third is in registers.  TOP: with barriers (all
// warps of the CTA, and the mid barriers between a column's pivot and its L
// entries, whose reciprocal goes through sinv).
template <typename T, bool TOP>
__device__ __forceinline__ void dot_run(const uint4* __restrict__ gs, uint4* win, const SchedDev& S,
                                        const BatchDev& D, int g, T* sinv, T* sink_row) {
  const int lane = threadIdx.x & 31;
  const size_t lb = (size_t)lane * sizeof(T);
  char* LU = (char*)D.lu + (size_t)g * S.n_slots * 32u * sizeof(T) + lb;
  char* X = (char*)D.sol + (size_t)g * S.n_u * 32u * sizeof(T) + lb;
  const char* R = (const char*)D.rhs + (size_t)g * S.n_u * 32u * sizeof(T) + lb;
  const float ptol = D.piv_tol;
  const uint32_t sink = TOP ? smem_u32(sink_row + lane) : 0u;
  bool bad = false, tiny = false;
  T v = (T)0, inv = (T)0, piv = (T)0;
  gs += lane;
  win[lane] = __ldg(gs);
  win[32 + lane] = __ldg(gs + 32);
  uint4 pre = __ldg(gs + 64);
  gs += 96;
  __syncwarp();
  int half = 0;
  const uint4* p = win;
  for (;;) {
    const uint4 h = *p++;
    const uint32_t op = h.x & 15u;
    if (op <= (TOP ? DOT_TOUCH : DOT_SKIP)) {
      if (op == DOT_END) break;
      if (TOP && op == DOT_TOUCH) {
        for (uint32_t i = 0; i < h.y; i++) dot_touch<T>(LU, *p++, sink);
        for (uint32_t i = 0; i < h.z; i++) dot_touch<T>(X, *p++, sink);
        continue;
      }
      if (op == DOT_SKIP) {
        __syncwarp();
        win[half + lane] = pre;
        pre = __ldg(gs);
        gs += 32;
        half ^= 32;
        p = win + half;
        __syncwarp();
        continue;
      }
      if (TOP)
        for (uint32_t i = 0; i < h.y; i++) __syncthreads();
      continue;
    }
    const bool row = op >= DOT_Y;
    char* B = row ? X : LU;
    if (!(h.x & DOT_CIN)) v = dot_ld<T>((h.x & DOT_FIRST) ? R : B, h.y);
    T d = (T)1;
    if (op == DOT_B) d = dot_ld<T>(LU, h.z);
    const int n = (int)((h.x >> 12) & 15u);
    switch (n) {
      case 1: dot_terms<T, 1>(p, LU, B, v); break;
      case 2: dot_terms<T, 2>(p, LU, B, v); break;
      case 3: dot_terms<T, 3>(p, LU, B, v); break;
      case 4: dot_terms<T, 4>(p, LU, B, v); break;
      case 5: dot_terms<T, 5>(p, LU, B, v); break;
      case 6: dot_terms<T, 6>(p, LU, B, v); break;
      case 7: dot_terms<T, 7>(p, LU, B, v); break;
      case 8: dot_terms<T, 8>(p, LU, B, v); break;
      default: break;
    }
    p += (n + 1) >> 1;
    if (h.x & DOT_COUT) continue;
    T out = v;
    switch (op) {
      case DOT_D:
        piv = fabs(v);
        bad |= v == (T)0;
        tiny |= ptol > 0.0f && (float)piv < ptol * (float)piv;
        inv = rcp_rn(v);
        if (TOP) {
          const uint32_t id = (h.x >> 8) & 15u;
          if (id) {
            sinv[((h.z >> 16) * 2 + 0) * 32 + lane] = inv;
            sinv[((h.z >> 16) * 2 + 1) * 32 + lane] = piv;
            asm volatile("barrier.cta.arrive %0, %1;\n" ::"r"(id), "r"(h.z & 0xffffu) : "memory");
          }
        }
        break;
      case DOT_LH:
        if (TOP) {
          asm volatile("barrier.cta.sync %0, %1;\n" ::"r"((h.x >> 8) & 15u), "r"(h.z & 0xffffu) : "memory");
          inv = sinv[((h.z >> 16) * 2 + 0) * 32 + lane];
          piv = sinv[((h.z >> 16) * 2 + 1) * 32 + lane];
        }
        // fallthrough: scaled as an L entry
      case DOT_L:
        tiny |= ptol > 0.0f && (float)piv < ptol * (float)fabs(v);
        out = v * inv;
        break;
      case DOT_B:
        out = v / d;
        bad |= !isfinite(out);
        break;
      default: break;
    }
    *reinterpret_cast<T*>(B + (size_t)h.y * (32u * sizeof(T))) = out;
    if (TOP && (h.x & DOT_BARF)) __syncthreads();
  }
  if (TOP) asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (bad) D.sing[g * 32 + lane] = 1;
  if (tiny) D.piv_flag[g * 32 + lane] = 1;
}

constexpr int kDotBinWarps = 8;  // streams per CTA of the bin launches
enum : int { DOT_BOTTOM = 0, DOT_PREP = 1, DOT_BACK = 2 };

template <typename T>
__device__ __forceinline__ void dot_bins_body(const DotDev& P, const SchedDev& S, const BatchDev& D, int which,
                                              int BX, int g) {
  __shared__ uint4 win[kDotBinWarps][64];
  if (!D.gact[g]) return;
  const int warp = threadIdx.x >> 5, b = BX * kDotBinWarps + warp;
  const int n = which == DOT_BOTTOM ? P.n_bottom : which == DOT_PREP ? P.n_prep : P.n_back;
  const int32_t* start = which == DOT_BOTTOM ? P.bottom : which == DOT_PREP ? P.prep : P.back;
  if (b >= n) return;
  dot_run<T, false>(P.words + start[b], win[warp], S, D, g, (T*)nullptr, (T*)nullptr);
}
template <typename T>
__global__ void __launch_bounds__(32 * kDotBinWarps) k_dot_bins(DotDev P, SchedDev S, BatchDev D, int which) {
  dot_bins_body<T>(P, S, D, which, blockIdx.x, blockIdx.y);
}

template <typename T, int NT>
__device__ __forceinline__ void dot_top_body(const DotDev& P, const SchedDev& S, const BatchDev& D, int g) {
  __shared__ uint4 win[NT][64];
  __shared__ T sinv[kDotMaxMid * 2 * 32];
  __shared__ T sink[32];
  if (!D.gact[g]) return;
  const int warp = threadIdx.x >> 5;
  dot_run<T, true>(P.words + P.top[warp], win[warp], S, D, g, sinv, sink);
}
template <typename T, int NT>
__global__ void __launch_bounds__(32 * NT, 1) k_dot_top(DotDev P, SchedDev S, BatchDev D) {
  dot_top_body<T, NT>(P, S, D, blockIdx.x);
}

// The same over a list of jobs (their CTAs: kDotBinWarps streams each, group by
// group; the top: one per group).
__device__ __host__ __forceinline__ int dot_blocks(int streams) {
  return (streams + kDotBinWarps - 1) / kDotBinWarps;
}
template <typename T>
__global__ void __launch_bounds__(32 * kDotBinWarps) k_dot_bins_multi(const MultiJob* __restrict__ jobs,
                                                                       MultiList L, int which) {
  __shared__ __align__(16) MultiJob J;
  const int b = enter_job(J, jobs, L);
  const int n = which == DOT_BOTTOM ? J.dot.n_bottom : which == DOT_PREP ? J.dot.n_prep : J.dot.n_back;
  const int nb = dot_blocks(n);
  dot_bins_body<T>(J.dot, J.S, J.D, which, b % nb, b / nb);
}
template <typename T, int NT>
__global__ void __launch_bounds__(32 * NT, 1) k_dot_top_multi(const MultiJob* __restrict__ jobs, MultiList L) {
  __shared__ __align__(16) MultiJob J;
  const int b = enter_job(J, jobs, L);
  dot_top_body<T, NT>(J.dot, J.S, J.D, b);
}

}  // namespace gox
