// Solo programs: the refactor of one scenario with both substitutions, the
// lanes of a warp on different sums.
//
// The dot programs (gox_dot.hpp) run a sum on a warp, a lane per scenario; a
// batch of one leaves 31 lanes idle.  Here a warp runs 32 sums at once, on the
// scenario's values in shared memory.  The sums, their order and their rounding
// are the dot programs'; a sum with fewer products than its warp's longest is
// filled up with products of a zero (v - 0 * 0 is v, bit for bit, for every v).
//
// A CTA loads the values it uses from the batch's interleaved ones, runs its
// sums in ticks that only read values of earlier ticks, a CTA barrier between
// them, and stores what later launches read.  One CTA runs everything where
// its values fit in shared memory; else columns in independent parts go to
// several CTAs, the leading products of the remaining columns that the parts
// allow run next, a few columns per CTA, then one CTA runs the rest and its
// backward rows, then the parts' CTAs theirs.
#pragma once
#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "gox_engine.hpp"

namespace gox {

// A unit: 12 words per lane, as three 16-byte quads of 32 lanes.  Values are
// byte offsets in the CTA's shared memory.
//   0        the lane's value
//   1 .. 8   four products a, b
//   9        SOLO_SRC: the lane of its column's pivot | SOLO_STORE ... (on a sum's
//            last unit)
//   10       backward rows: the pivot
//   11       the warp's flags | most products of a lane << 4 | barriers after the
//            unit << 8
enum : uint32_t {
  SOLO_SRC = 31u,
  SOLO_STORE = 1u << 5,  // the lane's value is stored after the unit
  SOLO_PIVOT = 1u << 6,  // it is its column's pivot
  SOLO_SCALE = 1u << 7   // an L entry: times the pivot's reciprocal
};
enum : uint32_t {
  SOLO_CIN = 1u,   // the sums go on from the unit before
  SOLO_COUT = 2u,  // ... and on to the next
  SOLO_COL = 4u,   // lanes with columns' entries
  SOLO_DIV = 8u,   // backward rows: divided by the pivot
  SOLO_END = 128u  // after the stream's last unit
};
constexpr int kSoloTerms = 4;              // products of a unit, per lane
constexpr int kSoloQuads = 3 * 32;         // quads of a unit
constexpr int kSoloWarps = 8;
// Units of a warp in shared memory, the one run and the next ones, while every
// scenario's CTA finds a place with kSoloDeep, else kSoloDepth (a unit's words come from
// the L2 and are wanted 300 to 500 cycles later; ms per refactor with 2 / 3 / 4 / 5
// / 6 units: 2,000 buses FP32, 16 CTAs .53 / .39 / .324 / .310 / .316, 20,000 buses
// .97 / .735 / .645 / .594 / .592; 600 scenarios of 118 buses FP64, which fit the
// chip with 3 only, .119 with 3 and .197 with 5).
constexpr int kSoloDepth = 3, kSoloDeep = 5;
constexpr int kSoloAhead = kSoloDeep - 1;  // units that are read past the one run (a program ends in as many)
static_assert(kSoloDeep >= kSoloDepth, "the deeper ring is the one that reads further");
constexpr int solo_ring_bytes(int depth) { return kSoloWarps * depth * kSoloQuads * 16; }
constexpr int kSoloSmem = 226 * 1024;  // of a CTA (1 KB is left for the kernel's own)
constexpr int kSoloMaxBytes = kSoloSmem - solo_ring_bytes(kSoloDepth);  // a CTA's values

// A CTA: its warps' streams (first unit of each), its values and what it stores
// (positions in lists: SOLO_LU, SOLO_RHS or SOLO_SOL and the slot or row, a
// stored one followed by its place among the values).
struct SoloCta {
  int32_t stream[kSoloWarps];
  int32_t load, n_load, store, n_store;
};
enum : uint32_t { SOLO_LU = 0u, SOLO_RHS = 1u << 30, SOLO_SOL = 2u << 30, SOLO_WHERE = 3u << 30 };

struct SoloPlan {
  int elem = 4;  // bytes of a value
  int ctas = 0;  // CTAs of the parts (0: one CTA runs everything)
  int cols = 4;  // columns of a CTA of the launch after them
};

struct SoloProgram {
  SoloPlan plan;
  std::vector<uint32_t> words, lists;
  // the launches' CTAs: the parts, the leading products of the rest, the rest
  // with its backward rows, the parts' backward rows
  std::vector<SoloCta> launch[4];
  int max_values[4] = {0, 0, 0, 0};  // of a CTA, the zero included
  int ctas() const { return std::max<int>(1, (int)launch[0].size()); }
};

// Compiles a plan: false where it cannot be (a schedule without the fused
// forward substitution, values that do not fit).
bool build_solo(const Schedule& sc, const SoloPlan& plan, SoloProgram& out);
// The program for a batch of one (wide) or for as many scenarios as possible:
// the parts' CTAs that measured best, or as few as fit.
bool build_solo_default(const Schedule& sc, int elem, bool wide, SoloProgram& out);
// Scenarios that a program of the schedule could run at most, by the sizes alone
// (more: none is compiled for them).
int solo_most(const Schedule& sc, int elem);
// Scenarios whose CTAs find a place on the chip at once by their shared memory,
// with `depth` units of a warp in it (0: its values leave no room for them).
// Registers are not counted: of k_solo_newton's CTAs (64 a thread) four fit on an SM,
// of k_solo's (40, FP64 47) six and five, so that of a grid of up to 60 buses more
// are let in than run at once.  They are still faster than the dot program (ms,
// 640 to 760 scenarios here / 800 there: 20 buses mixed .374 / .465, FP64 .48 / .53;
// 700 / 1,000: 50 buses .49 / .55, .66 / .68).
int solo_scenarios(const SoloProgram& p, int depth);

// Host interpreter for one scenario in FP64, with the checks of run_dot_host:
// indices in range, values final when read and not written in the tick (or, by
// another CTA, in the launch) they are used in, equal barrier counts, every
// sum complete and in order.  Returns an empty string or the first violation.
std::string run_solo_host(const Schedule& sc, const SoloProgram& p, std::vector<double>& lu,
                          const std::vector<double>& rhs, std::vector<double>& X, bool& singular);

}  // namespace gox
