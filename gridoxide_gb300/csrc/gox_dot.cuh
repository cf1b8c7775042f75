// Interpreter of the dot-product programs (gox_dot.hpp).
//
// What bounds it: the top is a chain of some 400 ticks forward (2,000 buses), a
// tick the latency of a sum (header and dispatch about 100 cycles, up to 8
// products about 300, for a pivot a reciprocal: 83 cycles, in FP64 441) plus
// a CTA barrier (78 cycles for 32 warps); its backward rows are a chain as
// long; the bins are bound by the latency of their loads and by instructions.
// Why sums instead of the streams' columns: a column's pivot and its L entries
// run on as many warps at once (1.7k cycles per tick against 4.0k per level),
// no ring has to be kept (values are found in the L1: a hit costs 67 cycles),
// and the bottom's columns spread over every SM instead of the group's.
// Why the touches: without them the tail's loads miss the L1 (the top of 128
// groups FP32 took 1.04 ms, with them 0.70 ms).
// Why packs: most sums of the bottom have no more than 3 products, and a unit of
// its own costs about 75 instructions (4 sums of 2 in a pack: about 75 too);
// with one finish per column and packs the 2,000-bus bottom of 256 bins went
// from 0.42 to 0.31 ms (128 groups FP32), at 64 registers instead of 40, with a
// kernel per launch (40 again) to 0.26 ms.
// Why chains: a backward row of the tail took about 950 cycles, the loads of
// the next row now run under it (2,000 buses, 128 groups FP32: 1.62 -> 1.45 ms
// with the kernels split by launch).
// Why the mid stage: a group's top ran on one SM, its early ticks 10 to 20k
// cycles wide, while with few groups the other SMs were idle.  Its second prep
// runs in ticks because a top column's U entries along a path of mid columns
// depend on each other (20,000 buses, one warp per column 0.35 ms, depth by
// depth over a CTA 0.35, with the sums' leading parts in earlier ticks 0.17).
// Refactor with both substitutions, streams -> programs without -> with the mid
// stage, ms: 2,000 buses, 128 groups FP32 2.15 -> 1.32 (none), 47 groups FP64
// 5.94 -> 2.07 -> 1.74, one group FP32 2.07 -> 0.95 -> 0.67; 10,000 buses, 128
// groups FP32 9.4 -> 4.9 (none); 20,000 buses, one group FP32 9.5 -> 3.8 -> 1.52;
// 118 buses, one group FP64 0.41 -> 0.19 -> 0.156.
#pragma once
#include "gox_dot.hpp"
#include "gox_kernels.cuh"

namespace gox {

// A value's address.  O32: base is the group's and the lane's value lies at a
// 32-bit offset from it (the base is the same for the whole grid row, so an
// address is one 32-bit multiply-add and no 64-bit one); else base is the
// lane's.  Measured (2,000 buses, 128 groups FP32, ms, 64-bit -> O32): top .604
// -> .561, back .125 -> .100; the bottom and prep get slower (.256 -> .283, .217
// -> .233: 48 registers, or 40 with fewer loads in flight), the top's backward
// rows too (.236 -> .254).
template <typename T, bool O32>
__device__ __forceinline__ size_t dot_at(uint32_t row) {
  if constexpr (O32) return (size_t)(row * (uint32_t)(32u * sizeof(T)) + (threadIdx.x & 31u) * (uint32_t)sizeof(T));
  return (size_t)row * (32u * sizeof(T));
}
template <typename T, bool O32 = false>
__device__ __forceinline__ T dot_ld(const char* base, uint32_t row) {
  return *reinterpret_cast<const T*>(base + dot_at<T, O32>(row));
}

template <typename T, bool O32 = false>
__device__ __forceinline__ void dot_st(char* base, uint32_t row, T v) {
  *reinterpret_cast<T*>(base + dot_at<T, O32>(row)) = v;
}

// M products at q: every load before the first multiply
template <typename T, int M, bool O32 = false>
__device__ __forceinline__ void dot_terms(const uint4* q, const char* A, const char* B, T& v) {
  T a[M], b[M];
#pragma unroll
  for (int t = 0; t < M; t += 2) {
    const uint4 e = q[t / 2];
    a[t] = dot_ld<T, O32>(A, e.x);
    b[t] = dot_ld<T, O32>(B, e.y);
    if (t + 1 < M) {
      a[t + 1] = dot_ld<T, O32>(A, e.z);
      b[t + 1] = dot_ld<T, O32>(B, e.w);
    }
  }
#pragma unroll
  for (int t = 0; t < M; t++) v -= a[t] * b[t];
}

// n products (0 to 8) at p.  Comparisons, not a jump table: an indirect branch
// costs more (one per unit over all units: the 2,000-bus top of one group FP32
// .346 -> .385 ms; a switch over n as a table against this tree .346 / .330).
template <typename T, bool O32 = false>
__device__ __forceinline__ void dot_sum(int n, const uint4* p, const char* A, const char* B, T& v) {
  if (n <= 4) {
    if (n <= 2) {
      if (n == 2) dot_terms<T, 2, O32>(p, A, B, v);
      else if (n == 1) dot_terms<T, 1, O32>(p, A, B, v);
    } else {
      if (n == 3) dot_terms<T, 3, O32>(p, A, B, v);
      else dot_terms<T, 4, O32>(p, A, B, v);
    }
  } else if (n <= 6) {
    if (n == 5) dot_terms<T, 5, O32>(p, A, B, v);
    else dot_terms<T, 6, O32>(p, A, B, v);
  } else {
    if (n == 7) dot_terms<T, 7, O32>(p, A, B, v);
    else dot_terms<T, 8, O32>(p, A, B, v);
  }
}

// Four sums of M products each at q (a quad of a's, then one of b's per product)
template <typename T, int M, bool O32 = false>
__device__ __forceinline__ void dot_pack(const uint4* q, const char* A, const char* B, T* v) {
  T a[M][4], b[M][4];
#pragma unroll
  for (int t = 0; t < M; t++) {
    const uint4 x = q[2 * t], y = q[2 * t + 1];
    a[t][0] = dot_ld<T, O32>(A, x.x);
    a[t][1] = dot_ld<T, O32>(A, x.y);
    a[t][2] = dot_ld<T, O32>(A, x.z);
    a[t][3] = dot_ld<T, O32>(A, x.w);
    b[t][0] = dot_ld<T, O32>(B, y.x);
    b[t][1] = dot_ld<T, O32>(B, y.y);
    b[t][2] = dot_ld<T, O32>(B, y.z);
    b[t][3] = dot_ld<T, O32>(B, y.w);
  }
#pragma unroll
  for (int t = 0; t < M; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] -= a[t][i] * b[t][i];
}

// Backward rows one after the other (a chain of the tail): a row's loads are
// issued while the row before it is summed, whose x it takes from a register.
template <typename T>
struct DotRow {
  uint32_t k, n;
  T v, d, a[dot_chain_terms(sizeof(T))], b[dot_chain_terms(sizeof(T))];
};
template <typename T>
__device__ __forceinline__ const uint4* dot_row_open(const uint4* p, const char* LU, const char* X, DotRow<T>& r) {
  const uint4 h = *p++;
  r.k = h.x;
  r.n = h.z;
  r.v = dot_ld<T>(X, h.x);
  r.d = dot_ld<T>(LU, h.y);
  const int n = (int)(h.z & 0xffffu);
#pragma unroll
  for (int t = 0; t < dot_chain_terms(sizeof(T)); t += 2)
    if (t < n) {
      const uint4 e = p[t / 2];
      r.a[t] = dot_ld<T>(LU, e.x);
      r.b[t] = dot_ld<T>(X, e.y);
      r.a[t + 1] = dot_ld<T>(LU, e.z);  // (an odd row's last product again: not summed)
      r.b[t + 1] = dot_ld<T>(X, e.w);
    }
  return p + ((n + 1) >> 1);
}
template <typename T, int M>
__device__ __forceinline__ void dot_row_sum(const DotRow<T>& r, T b0, T& v) {
#pragma unroll
  for (int t = 0; t < M; t++) v -= r.a[t] * (t == 0 ? b0 : r.b[t]);
}
template <typename T>
__device__ __forceinline__ T dot_row_run(const DotRow<T>& r, T x, char* X, bool& bad) {
  const int n = (int)(r.n & 0xffffu);
  T v = r.v;
  const T b0 = (r.n & DOT_NEXT) ? x : r.b[0];
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int t = 0; t < dot_chain_terms(sizeof(T)); t++)
      if (t < n) v -= r.a[t] * (t == 0 ? b0 : r.b[t]);
  } else {  // (a predicated FP64 multiply-add takes its time also where it is off)
    switch (n) {
      case 1: dot_row_sum<T, 1>(r, b0, v); break;
      case 2: dot_row_sum<T, 2>(r, b0, v); break;
      case 3: dot_row_sum<T, 3>(r, b0, v); break;
      case 4: dot_row_sum<T, 4>(r, b0, v); break;
      case 5: dot_row_sum<T, 5>(r, b0, v); break;
      case 6: dot_row_sum<T, 6>(r, b0, v); break;
      case 7: dot_row_sum<T, 7>(r, b0, v); break;
      case 8: dot_row_sum<T, 8>(r, b0, v); break;
      default: break;
    }
  }
  v = v / r.d;
  bad |= !isfinite(v);
  dot_st<T>(X, r.k, v);
  return v;
}
template <typename T>
__device__ __forceinline__ const uint4* dot_chain(const uint4* p, int rows, const char* LU, char* X, bool& bad) {
  DotRow<T> r, s;
  T x = (T)0;
  p = dot_row_open<T>(p, LU, X, r);
  for (;;) {
    if (rows > 1) p = dot_row_open<T>(p, LU, X, s);
    x = dot_row_run<T>(r, x, X, bad);
    if (--rows == 0) break;
    if (rows > 1) p = dot_row_open<T>(p, LU, X, r);
    x = dot_row_run<T>(s, x, X, bad);
    if (--rows == 0) break;
  }
  return p;
}

// four values into the L1: asynchronous copies (cached at every level) into a
// row of shared memory that nobody reads
template <typename T, bool O32 = false>
__device__ __forceinline__ void dot_touch(const char* base, const uint4& q, uint32_t sink) {
  const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int t = 0; t < 4; t++)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sink), "l"(base + dot_at<T, O32>(r[t])),
                 "n"((int)sizeof(T)) : "memory");
}

// What a launch's streams hold: only those units are compiled into it.
enum : int { DOT_BOTTOM = 0, DOT_PREP = 1, DOT_BACK = 2, DOT_TOP = 3, DOT_TOPBACK = 4 };

// One warp runs one stream.  win: 64 quads of shared memory, the chunk being
// run and the next one; the third is in registers.  The top's launches have
// barriers (all warps of the CTA, and the mid barriers between a column's
// pivot and its L entries, whose reciprocal goes through sinv) and touches.
template <typename T, int WHICH>
__device__ __forceinline__ void dot_run(const uint4* __restrict__ gs, uint4* win, const SchedDev& S,
                                        const BatchDev& D, int g, T* sinv, T* sink_row) {
  constexpr bool BAR = WHICH == DOT_TOP || WHICH == DOT_TOPBACK;  // ticks
  constexpr bool FWD = WHICH != DOT_BACK && WHICH != DOT_TOPBACK;
  const int lane = threadIdx.x & 31;
  constexpr bool O32 = WHICH == DOT_TOP || WHICH == DOT_BACK;
  const size_t lb = O32 ? 0 : (size_t)lane * sizeof(T);
  char* LU = (char*)D.lu + (size_t)g * S.n_slots * 32u * sizeof(T) + lb;
  char* X = (char*)D.sol + (size_t)g * S.n_u * 32u * sizeof(T) + lb;
  const char* R = (const char*)D.rhs + (size_t)g * S.n_u * 32u * sizeof(T) + lb;
  const float ptol = D.piv_tol;
  const uint32_t sink = BAR ? smem_u32(sink_row + lane) : 0u;
  bool bad = false, tiny = false;
  T v = (T)0;
  gs += lane;
  static_assert(kDotAhead >= 2, "two chunks in shared memory and one in registers");
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
    if (op < DOT_U) {
      if (FWD && op == DOT_PACK) {
        const uint4 e = *p++;
        char* B = (h.x & DOT_ROW) ? X : LU;
        const char* F = (h.x & DOT_FIRST) ? R : B;
        T x[4] = {dot_ld<T, O32>(F, e.x), dot_ld<T, O32>(F, e.y), dot_ld<T, O32>(F, e.z), dot_ld<T, O32>(F, e.w)};
        switch ((h.x >> 12) & 15u) {
          case 1: dot_pack<T, 1, O32>(p, LU, B, x); p += 2; break;
          case 2: dot_pack<T, 2, O32>(p, LU, B, x); p += 4; break;
          case 3: dot_pack<T, 3, O32>(p, LU, B, x); p += 6; break;
          default: break;
        }
        dot_st<T, O32>(B, e.x, x[0]);
        dot_st<T, O32>(B, e.y, x[1]);
        dot_st<T, O32>(B, e.z, x[2]);
        dot_st<T, O32>(B, e.w, x[3]);
      } else if (FWD && op == DOT_FIN) {
        char* C = LU + (size_t)h.y * (32u * sizeof(T));
        const T d = dot_ld<T, O32>(C, 0);
        const T r = rcp_rn(d), pa = fabs(d);
        T m = pa;
        const int z = (int)h.z;
        for (int i = 1; i <= z; i += 4) {  // (the last entry again where fewer than four are left)
          const int i1 = min(i + 1, z), i2 = min(i + 2, z), i3 = min(i + 3, z);
          const T x0 = dot_ld<T, O32>(C, i), x1 = dot_ld<T, O32>(C, i1), x2 = dot_ld<T, O32>(C, i2), x3 = dot_ld<T, O32>(C, i3);
          if (sizeof(T) == 4) m = fmax(fmax(m, fmax(fabs(x0), fabs(x1))), fmax(fabs(x2), fabs(x3)));
          dot_st<T, O32>(C, i, x0 * r);
          // (in FP64 a multiply costs more than a branch)
          if (sizeof(T) == 4 || i1 != i) dot_st<T, O32>(C, i1, x1 * r);
          if (sizeof(T) == 4 || i2 != i1) dot_st<T, O32>(C, i2, x2 * r);
          if (sizeof(T) == 4 || i3 != i2) dot_st<T, O32>(C, i3, x3 * r);
        }
        bad |= d == (T)0;
        tiny |= ptol > 0.0f && (float)pa < ptol * (float)m;
      } else if (WHICH == DOT_TOPBACK && op == DOT_CHAIN) {
        p = dot_chain<T>(p, (int)h.y, LU, X, bad);
      } else if (op == DOT_SKIP) {
        __syncwarp();
        win[half + lane] = pre;
        pre = __ldg(gs);
        gs += 32;
        half ^= 32;
        p = win + half;
        __syncwarp();
        continue;
      } else if (BAR && op == DOT_TOUCH) {
        for (uint32_t i = 0; i < h.y; i++) dot_touch<T, O32>(LU, *p++, sink);
        for (uint32_t i = 0; i < h.z; i++) dot_touch<T, O32>(X, *p++, sink);
        continue;
      } else if (BAR && op == DOT_BAR) {
        for (uint32_t i = 0; i < h.y; i++) __syncthreads();
        continue;
      } else {
        break;  // DOT_END
      }
    } else {
      if (FWD && (h.x & DOT_PLAIN)) {  // the most frequent unit: no other flag to look at
        const int n = (int)((h.x >> 12) & 15u);
        T s = dot_ld<T, O32>(LU, h.y);
        dot_sum<T, O32>(n, p, LU, LU, s);
        dot_st<T, O32>(LU, h.y, s);
        p += (n + 1) >> 1;
        if (BAR && (h.x & DOT_BARF)) __syncthreads();
        continue;
      }
      const bool row = !FWD || op >= DOT_Y;
      char* B = row ? X : LU;
      if (!(h.x & DOT_CIN)) v = dot_ld<T, O32>(FWD && (h.x & DOT_FIRST) ? R : B, h.y);
      T d = (T)1;
      if (!FWD) d = dot_ld<T, O32>(LU, h.z);
      const int n = (int)((h.x >> 12) & 15u);
      dot_sum<T, O32>(n, p, LU, B, v);
      p += (n + 1) >> 1;
      if (h.x & DOT_COUT) continue;
      T out = v;
      if (!FWD) {  // DOT_B
        out = v / d;
        bad |= !isfinite(out);
      } else if (WHICH == DOT_TOP && op == DOT_D) {
        const T inv = rcp_rn(v);
        T* q = sinv + (h.z >> 16) * 64 + lane;
        q[0] = inv;
        q[32] = v;
        asm volatile("barrier.cta.arrive %0, %1;\n" ::"r"((h.x >> 8) & 15u), "r"(h.z & 0xffffu) : "memory");
        bad |= v == (T)0;
        tiny |= ptol > 0.0f && (float)fabs(v) < ptol * (float)fabs(v);
      } else if (WHICH == DOT_TOP && op == DOT_LH) {
        asm volatile("barrier.cta.sync %0, %1;\n" ::"r"((h.x >> 8) & 15u), "r"(h.z & 0xffffu) : "memory");
        const T* q = sinv + (h.z >> 16) * 64 + lane;
        const T inv = q[0], piv = q[32];
        tiny |= ptol > 0.0f && (float)fabs(piv) < ptol * (float)fabs(v);
        out = v * inv;
      }
      dot_st<T, O32>(B, h.y, out);
    }
    if (BAR && (h.x & DOT_BARF)) __syncthreads();
  }
  if (BAR) asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (bad) D.sing[g * 32 + lane] = 1;
  if (tiny) D.piv_flag[g * 32 + lane] = 1;
}

constexpr int kDotBinWarps = 8;  // streams per CTA of the bin launches
// CTAs of an SM: 40 registers in FP32 and for the backward rows, 64 in FP64 (72
// and 88 where the compiler may: 2,000 buses, 128 groups FP32, the whole
// refactor 1.47 ms against 1.33)
constexpr int dot_bin_ctas(size_t elem, int which) { return elem == 4 || which == DOT_BACK ? 6 : 4; }

template <typename T, int WHICH>
__device__ __forceinline__ void dot_bins_body(const DotDev& P, const SchedDev& S, const BatchDev& D, int BX,
                                              int g) {
  __shared__ uint4 win[kDotBinWarps][64];
  if (!D.gact[g]) return;
  const int warp = threadIdx.x >> 5, b = BX * kDotBinWarps + warp;
  const int n = WHICH == DOT_BOTTOM ? P.n_bottom : WHICH == DOT_PREP ? P.n_prep : P.n_back;
  const int32_t* start = WHICH == DOT_BOTTOM ? P.bottom : WHICH == DOT_PREP ? P.prep : P.back;
  if (b >= n) return;
  dot_run<T, WHICH>(P.words + start[b], win[warp], S, D, g, (T*)nullptr, (T*)nullptr);
}
template <typename T, int WHICH>
__global__ void __launch_bounds__(32 * kDotBinWarps, dot_bin_ctas(sizeof(T), WHICH))
    k_dot_bins(DotDev P, SchedDev S, BatchDev D) {
  dot_bins_body<T, WHICH>(P, S, D, blockIdx.x, blockIdx.y);
}

// The launches of the tick kernels, and a group's CTAs in each.
enum : int { DOT_IN_TOP = 0, DOT_IN_MID = 1, DOT_IN_PREP2 = 2 };
__device__ __host__ __forceinline__ int dot_ctas(const DotDev& P, int stage) {
  return stage == DOT_IN_MID ? P.n_mid : stage == DOT_IN_PREP2 ? P.n_prep2 : 1;
}

template <typename T, int NT>
__device__ __forceinline__ void dot_top_body(const DotDev& P, const SchedDev& S, const BatchDev& D, int stage,
                                             int BX, int g) {
  __shared__ uint4 win[NT][64];
  __shared__ T sinv[kDotMaxMid * 2 * 32];
  __shared__ T sink[32];
  if (!D.gact[g]) return;
  const int warp = threadIdx.x >> 5;
  const int32_t* start = stage == DOT_IN_MID ? P.mid : stage == DOT_IN_PREP2 ? P.prep2 : P.top;
  dot_run<T, DOT_TOP>(P.words + start[BX * NT + warp], win[warp], S, D, g, sinv, sink);
}
template <typename T, int NT>
__global__ void __launch_bounds__(32 * NT, 1) k_dot_top(DotDev P, SchedDev S, BatchDev D, int stage) {
  dot_top_body<T, NT>(P, S, D, stage, blockIdx.x, blockIdx.y);
}
template <typename T>
__device__ __forceinline__ void dot_topback_body(const DotDev& P, const SchedDev& S, const BatchDev& D, int stage,
                                                 int BX, int g) {
  __shared__ uint4 win[kDotBackWarps][64];
  __shared__ T sink[32];
  if (!D.gact[g]) return;
  const int warp = threadIdx.x >> 5;
  dot_run<T, DOT_TOPBACK>(P.words + (stage == DOT_IN_MID ? P.midback : P.tback)[BX * kDotBackWarps + warp], win[warp], S, D, g,
                          (T*)nullptr, sink);
}
template <typename T>
__global__ void __launch_bounds__(32 * kDotBackWarps, 1) k_dot_topback(DotDev P, SchedDev S, BatchDev D, int stage) {
  dot_topback_body<T>(P, S, D, stage, blockIdx.x, blockIdx.y);
}

// The same over a list of jobs (their CTAs: kDotBinWarps streams each, group by
// group; the top's: one per group, the mid stage's: n_mid per group).
__device__ __host__ __forceinline__ int dot_blocks(int streams) {
  return (streams + kDotBinWarps - 1) / kDotBinWarps;
}
template <typename T, int WHICH>
__global__ void __launch_bounds__(32 * kDotBinWarps, dot_bin_ctas(sizeof(T), WHICH))
    k_dot_bins_multi(const MultiJob* __restrict__ jobs, MultiList L) {
  __shared__ __align__(16) MultiJob J;
  const int b = enter_job(J, jobs, L);
  const int n = WHICH == DOT_BOTTOM ? J.dot.n_bottom : WHICH == DOT_PREP ? J.dot.n_prep : J.dot.n_back;
  const int nb = dot_blocks(n);
  dot_bins_body<T, WHICH>(J.dot, J.S, J.D, b % nb, b / nb);
}
template <typename T, int NT>
__global__ void __launch_bounds__(32 * NT, 1) k_dot_top_multi(const MultiJob* __restrict__ jobs, MultiList L,
                                                                   int stage) {
  __shared__ __align__(16) MultiJob J;
  const int b = enter_job(J, jobs, L), nb = dot_ctas(J.dot, stage);
  dot_top_body<T, NT>(J.dot, J.S, J.D, stage, b % nb, b / nb);
}
template <typename T>
__global__ void __launch_bounds__(32 * kDotBackWarps, 1) k_dot_topback_multi(const MultiJob* __restrict__ jobs,
                                                                              MultiList L, int stage) {
  __shared__ __align__(16) MultiJob J;
  const int b = enter_job(J, jobs, L), nb = stage == DOT_IN_MID ? J.dot.n_midback : 1;
  dot_topback_body<T>(J.dot, J.S, J.D, stage, b % nb, b / nb);
}

}  // namespace gox
