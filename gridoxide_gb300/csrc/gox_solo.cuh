// Interpreter of the solo programs (gox_solo.hpp).
//
// What bounds it: a chain of as many ticks forward as the elimination has
// levels and as many back (2,000 buses: 414 + 414), each the latency of a
// unit: its words from shared memory, its values, four multiply-adds, for a
// column a shuffle and a reciprocal, a store and a CTA barrier.  A sum per lane
// puts what the dot programs spread over 32 warps on two or three, so a tick
// has few instructions and the FP64 pipe has one multiply-add where it had up
// to 32 on idle lanes.
// Why shared memory: values in the L1 instead cost a tag lookup per lane and
// load, 9 loads a unit (2,000 buses FP32, one scenario: 0.95 ms against 0.54).
// Why the next unit's words are loaded under this one's values: a tick is
// mostly dependent instructions, and what need not follow the barrier is moved
// out of the chain (118 buses FP64 0.145 -> 0.104 ms, FP32 0.060 -> 0.049).
// Eight warps: with 16 the copies of the streams take the room of values (118
// buses: the same time).
// Refactor of one scenario with both substitutions, dot program -> solo, ms:
// 118 buses FP64 0.156 -> 0.104; 2,000 buses FP32 0.67 -> 0.37, FP64 1.27 -> 0.74;
// 20,000 buses FP32 1.52 -> 0.74.  152 scenarios of 2,000 buses FP32 0.69 -> 0.47;
// 600 of 118 buses FP64 0.19 -> 0.12.
#pragma once
#include "gox_kernels.cuh"
#include "gox_solo.hpp"

namespace gox {

struct SoloDev {
  const uint4* words;
  const uint32_t* lists;
  const SoloCta* cta[4];
  int ctas[4], bytes[4];  // per launch: CTAs, shared memory of one
  int stride;             // from a scenario's value to its next (32; 1: a batch of one by itself)
};

// One launch of a program: a CTA per part and scenario.
template <typename T>
__global__ void __launch_bounds__(32 * kSoloWarps)
    k_solo(SoloDev P, SchedDev S, BatchDev D, int which) {
  extern __shared__ __align__(16) unsigned char solo_smem[];
  const int g = blockIdx.y >> 5, l = blockIdx.y & 31, s = blockIdx.y;
  if (!D.gact[g]) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SoloCta* C = P.cta[which] + blockIdx.x;
  uint4* ring = reinterpret_cast<uint4*>(solo_smem) + warp * kSoloDepth * kSoloQuads + lane;
  char* c = reinterpret_cast<char*>(solo_smem) + kSoloRingBytes;
  const uint4* gs = P.words + (size_t)C->stream[warp] * kSoloQuads + lane;
  auto fetch = [&](int slot) {
#pragma unroll
    for (int i = 0; i < 3; i++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(ring + slot * kSoloQuads + 32 * i)),
                   "l"(gs + 32 * i)
                   : "memory");
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    gs += kSoloQuads;
  };
#pragma unroll
  for (int i = 0; i < kSoloDepth; i++) fetch(i);
  const size_t stride = (size_t)P.stride;
  T* lu = (T*)D.lu + (size_t)g * S.n_slots * 32 + l;
  T* sol = (T*)D.sol + (size_t)g * S.n_u * 32 + l;
  const T* rhs = (const T*)D.rhs + (size_t)g * S.n_u * 32 + l;
  const int n_load = C->n_load, n_store = C->n_store;
  const uint32_t *load = P.lists + C->load, *store = P.lists + C->store;
  T* values = reinterpret_cast<T*>(c);
#pragma unroll 4
  for (int i = threadIdx.x; i < n_load; i += 32 * kSoloWarps) {
    const uint32_t x = __ldg(load + i), w = x & SOLO_WHERE;
    values[i] = (w == SOLO_LU ? lu : w == SOLO_RHS ? rhs : sol)[(x & ~SOLO_WHERE) * stride];
  }
  if (threadIdx.x == 0) values[n_load] = (T)0;
  __syncthreads();
  const float ptol = D.piv_tol;
  bool bad = false, tiny = false;
  T v = (T)0;
  auto at = [&](uint32_t off) -> T& { return *reinterpret_cast<T*>(c + off); };
  int slot = 0;
  uint4 q0, q1, q2;
  // a unit's words: a lane reads only what it copied itself
  auto words = [&]() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kSoloDepth - 1) : "memory");
    const uint4* u = ring + slot * kSoloQuads;
    q0 = u[0];
    q1 = u[32];
    q2 = u[64];
  };
  // on to the next unit's, in the shadow of this one's loads
  auto next = [&]() {
    fetch(slot);
    slot = slot == kSoloDepth - 1 ? 0 : slot + 1;
    words();
  };
  // the products of the lane that the unit's longest sum has (in FP64 each one
  // left out saves 65 cycles; in FP32 a test costs more than it saves)
  auto sum = [&](uint32_t n, T a0, T b0, T a1, T b1, T a2, T b2, T a3, T b3) {
    if (sizeof(T) == 4) {
      v -= a0 * b0;
      v -= a1 * b1;
      v -= a2 * b2;
      v -= a3 * b3;
    } else if (n > 0) {
      v -= a0 * b0;
      if (n > 1) {
        v -= a1 * b1;
        if (n > 2) {
          v -= a2 * b2;
          if (n > 3) v -= a3 * b3;
        }
      }
    }
  };
  words();
  while (!(q2.w & (SOLO_DIV | SOLO_END))) {
    const uint32_t f = q2.w, info = q2.y, to = q0.x;
    const T a0 = at(q0.y), b0 = at(q0.z), a1 = at(q0.w), b1 = at(q1.x), a2 = at(q1.y), b2 = at(q1.z),
            a3 = at(q1.w), b3 = at(q2.x), v0 = at(to);
    next();
    v = (f & SOLO_CIN) ? v : v0;
    sum((f >> 4) & 7u, a0, b0, a1, b1, a2, b2, a3, b3);
    if (f & SOLO_COL) {
      const T piv = __shfl_sync(0xffffffffu, v, info & SOLO_SRC);
      const T r = rcp_rn(piv);
      if (info & SOLO_STORE) at(to) = (info & SOLO_SCALE) ? v * r : v;
      const bool in_col = (info & (SOLO_PIVOT | SOLO_SCALE)) != 0;
      bad |= in_col && piv == (T)0;
      tiny |= in_col && ptol > 0.0f && (float)fabs(piv) < ptol * (float)fabs(v);
    } else if (info & SOLO_STORE) {
      at(to) = v;
    }
    for (uint32_t n = f >> 8; n > 0; n--) __syncthreads();
  }
  while (!(q2.w & SOLO_END)) {
    const uint32_t f = q2.w, info = q2.y, to = q0.x;
    const T a0 = at(q0.y), b0 = at(q0.z), a1 = at(q0.w), b1 = at(q1.x), a2 = at(q1.y), b2 = at(q1.z),
            a3 = at(q1.w), b3 = at(q2.x), v0 = at(to), d = at(q2.z);
    next();
    v = (f & SOLO_CIN) ? v : v0;
    sum((f >> 4) & 7u, a0, b0, a1, b1, a2, b2, a3, b3);
    if (!(f & SOLO_COUT)) {
      const T out = v / d;
      if (info & SOLO_STORE) {
        at(to) = out;
        bad |= !isfinite(out);
      }
    }
    for (uint32_t n = f >> 8; n > 0; n--) __syncthreads();
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  for (int i = threadIdx.x; i < n_store; i += 32 * kSoloWarps) {
    const uint2 x = *reinterpret_cast<const uint2*>(store + 2 * i);
    ((x.x & SOLO_WHERE) == SOLO_LU ? lu : sol)[(x.x & ~SOLO_WHERE) * stride] = values[x.y];
  }
  if (bad) D.sing[s] = 1;
  if (tiny) D.piv_flag[s] = 1;
}

}  // namespace gox
