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
// 118 buses FP64 0.156 -> 0.104; 2,000 buses FP32 0.67 -> 0.31, FP64 1.27 -> 0.69;
// 20,000 buses FP32 1.52 -> 0.59.  152 scenarios of 2,000 buses FP32 0.69 -> 0.47;
// 600 of 118 buses FP64 0.19 -> 0.12.
#pragma once
#include "gox_kernels.cuh"
#include "gox_solo.hpp"

namespace gox {

struct SoloDev {
  const uint4* words;
  const uint32_t* lists;
  const SoloCta* cta[4];
  int ctas[4], bytes[4];  // per launch: CTAs, bytes of a CTA's values
  int stride;             // from a scenario's value to its next (32; 1: a batch of one by itself)
};

// Scenario s's part in CTA `part` of a launch; DEPTH: units of a warp in shared
// memory.
template <typename T, int DEPTH>
__device__ __forceinline__ void solo_body(const SoloDev& P, const SchedDev& S, const BatchDev& D, int which, int part,
                                          int s) {
  extern __shared__ __align__(16) unsigned char solo_smem[];
  const int g = s >> 5, l = s & 31;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SoloCta* C = P.cta[which] + part;
  uint4* ring = reinterpret_cast<uint4*>(solo_smem) + warp * DEPTH * kSoloQuads + lane;
  char* c = reinterpret_cast<char*>(solo_smem) + kSoloWarps * DEPTH * kSoloQuads * 16;
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
  for (int i = 0; i < DEPTH; i++) fetch(i);
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
    asm volatile("cp.async.wait_group %0;\n" ::"n"(DEPTH - 1) : "memory");
    const uint4* u = ring + slot * kSoloQuads;
    q0 = u[0];
    q1 = u[32];
    q2 = u[64];
  };
  // on to the next unit's, in the shadow of this one's loads
  auto next = [&]() {
    fetch(slot);
    slot = slot == DEPTH - 1 ? 0 : slot + 1;
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

// One launch of a program: a CTA per part and scenario.
template <typename T, int DEPTH>
__global__ void __launch_bounds__(32 * kSoloWarps) k_solo(SoloDev P, SchedDev S, BatchDev D, int which) {
  if (D.gact[blockIdx.y >> 5]) solo_body<T, DEPTH>(P, S, D, which, blockIdx.x, blockIdx.y);
}

// Task t's Jacobian entries of one scenario (out: it has a branch out)
template <typename T>
__device__ __forceinline__ void solo_fill(const SchedDev& S, const BatchDev& D, int g, int lane, int s, bool out, int t) {
  const int4 dst = __ldg(S.ft_dst + t), bus = __ldg(S.ft_bus + t);
  T G, B;
  if constexpr (sizeof(T) == 4) {
    const float2 y = __ldg(S.ft_yf + t);
    G = y.x;
    B = y.y;
  } else {
    const double2 y = __ldg(S.ft_y + t);
    G = y.x;
    B = y.y;
  }
  const size_t gb = (size_t)g * S.n_bus * 32u + lane, xi = gb + (size_t)bus.x * 32u, xk = gb + (size_t)bus.y * 32u;
  const bool dg = bus.w != 0;
  const T *eT = (const T*)D.eT, *fT = (const T*)D.fT, *ivT = (const T*)D.ivT;
  const T v[5] = {eT[xi], fT[xi], dg ? ivT[xi] : eT[xk], dg ? ((const T*)D.pT)[xi] : fT[xk],
                  dg ? ((const T*)D.qT)[xi] : ivT[xk]};
  if (out) {
    for (int c = 0; c < 4; c++)
      if (D.o_slot[4 * s + c] == bus.z) {  // (the first of equal slots, as the batch kernel)
        const double2 y = __ldg(S.ft_y + t);
        G = (T)(y.x + D.o_dre[4 * s + c]);
        B = (T)(y.y + D.o_dim[4 * s + c]);
        break;
      }
  }
  T h, nn, m, l;
  fill_entries<T>(dg, v, G, B, h, nn, m, l);
  T* LU = (T*)D.lu + (size_t)g * S.n_slots * 32u;
  T* OFF = (T*)D.off + (size_t)g * S.n_off * 32u;
  fill_store(LU, OFF, S.n_slots, dst.x, lane, h);
  fill_store(LU, OFF, S.n_slots, dst.y, lane, nn);
  fill_store(LU, OFF, S.n_slots, dst.z, lane, m);
  fill_store(LU, OFF, S.n_slots, dst.w, lane, l);
}

// A scenario's whole Newton loop on its CTA (programs of one CTA): the
// batch kernels' steps with a thread per bus, per Y entry and per slot, and
// CTA barriers between them.  Seven launches, a copy and a wait on the host
// per iteration took some 50 us of a small grid's iteration, as much as its
// refactor.  Measured, whole solves: 118 buses FP64, one scenario .741 -> .565
// ms (mixed .513 -> .347), 75 load cases of 300 buses .631 -> .542.
// (kSoloDepth units: with kSoloDeep the 75 cases took .567 ms.)  EXTRA: the batch
// has outages or voltage-dependent loads.
template <typename T, bool EXTRA>
__global__ void __launch_bounds__(32 * kSoloWarps, 4) k_solo_newton(SoloDev P, SchedDev S, BatchDev D, int max_iter) {
  constexpr int NTH = 32 * kSoloWarps;
  __shared__ unsigned long long red[kSoloWarps];
  __shared__ int go;
  const int s = blockIdx.x, g = s >> 5, l = s & 31, tid = threadIdx.x;
  int obf = -1, obt = -1;
  if (EXTRA && D.o_bf) {
    obf = D.o_bf[s];
    obt = D.o_bt[s];
  }
  for (int it = 0; it < max_iter; it++) {
    for (int i = tid; i < S.n_bus; i += NTH) update_one<T>(S, D, it, 0, g, i, l);
    const bool active = D.status[s] == ST_RUNNING && !(it > 0 && D.sing[s] != 0);
    __syncthreads();
    unsigned long long mx = 0ull;
    for (int i = tid; i < S.n_bus; i += NTH)
      inject_one<T, EXTRA, EXTRA>(S, D, g, i, l, s, active, obf, obt, it == 0 ? D.st0 : nullptr, mx);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((tid & 31) == 0) red[tid >> 5] = mx;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < kSoloWarps; w++) mx = max(mx, red[w]);
      go = decide_one(D, it, 0, s, active ? mx : 0ull);
    }
    __syncthreads();
    if (!go) return;
    for (int t = tid; t < S.n_ftask; t += NTH) solo_fill<T>(S, D, g, l, s, EXTRA && obf >= 0, t);
    T* LU = (T*)D.lu + (size_t)g * S.n_slots * 32u + l;
    for (int z = tid; z < S.n_fzero; z += NTH) LU[(size_t)__ldg(S.fz_slot + z) * 32u] = (T)0;
    __syncthreads();
    solo_body<T, kSoloDepth>(P, S, D, 2, 0, s);
    __syncthreads();
  }
  for (int i = tid; i < S.n_bus; i += NTH) update_one<T>(S, D, max_iter, 1, g, i, l);
  __syncthreads();
  if (tid == 0) decide_one(D, max_iter, 1, s, 0ull);
}

}  // namespace gox
