// Dot-product programs for the batched refactor.
//
// Every value of the factor and of the two substitutions is one ordered sum
// of products: an entry (i, k) of L or U is its A value minus the L(i, j)
// U(j, k) in KLU's update order (an L entry then times the pivot's
// reciprocal), y_k is b_k minus the L(k, j) y_j, x_k is y_k minus the U(k, j)
// x_j, divided by the pivot.  A program may run the sums in any order of
// values, and a sum in pieces, as long as each value's own products stay in
// order: the result is the stream form's (gox_stream.hpp) bit for bit.
//
// Five to eight launches run a refactor with both substitutions:
//   bottom    columns in independent parts of the elimination forest, whole
//             parts assigned to bins; one warp runs a bin's sums in order and
//             needs no barrier, since it wrote every value it reads
//   prep      one warp per remaining column or two: the leading part of each
//             of its sums that only needs bottom columns
//   mid       (few groups) columns in independent parts of what is left, dealt
//             out to a few CTAs per group: the sums as units of up to 8 products
//             spread over the warps, in ticks that only read values of earlier
//             ticks, with a CTA barrier after each
//   prep 2    the leading parts of the remaining sums that the mid columns
//             allow, a few columns per CTA, in ticks
//   top       the rest of the columns, one CTA per group, in ticks
//   top back  their backward rows, one CTA per group, in ticks too
//   mid back  the mid columns' backward rows, CTA by CTA, in ticks
//   back      the backward rows of the bottom columns, bin by bin
#pragma once
#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "gox_engine.hpp"

namespace gox {

// A stream is a list of 16-byte quads in chunks of 32.  A unit is one header
// quad, then its products (a, b), two per quad, all in one chunk:
//   x = op | barrier after << 4 | first << 5 | carry in << 6 | carry out << 7 |
//       mid << 8 | n << 12 | row << 16 | plain << 17 (U without a carry)
//   y = the value's slot (U, D, LH) or row (Y, B); BAR: how many
//   z = D, LH: threads of the mid barrier | shared index << 16;  B: pivot slot
// a and b are LU slots (U, D, LH), or an LU slot and a row (Y, B).  A sum of
// more than 8 products is carried from unit to unit in a register.
enum : uint32_t {
  DOT_END = 0,
  DOT_BAR = 1,   // y CTA barriers
  DOT_SKIP = 2,  // on to the next chunk
  DOT_TOUCH = 3, // y quads of LU slots, then z quads of rows: values a later
                 // unit needs, loaded into the SM's L1 and dropped
  DOT_PACK = 4,  // four U or (DOT_ROW) Y sums of n <= 3 products each: one quad of
                 // values, then per product a quad of a's and one of b's
  DOT_FIN = 5,   // a column's pivot in slot y and the z L entries after it, all
                 // sums done: reciprocal, L entries scaled
  DOT_CHAIN = 6, // y backward rows, one after the other: per row a quad k, pivot
                 // slot, n | DOT_NEXT, 0, then its products; DOT_NEXT: the first
                 // one's x is the row before's
  DOT_U = 7,     // U(j, k), or a leading part of any LU entry's sum
  DOT_D = 8,     // pivot: its reciprocal to shared memory, for the LH units
  DOT_LH = 9,    // L(i, k): its sum first, then the mid barrier, then scaled
  DOT_Y = 10,    // y_k (first: starts from the right-hand side, else from y)
  DOT_B = 11     // x_k
};
constexpr uint32_t DOT_BARF = 1u << 4, DOT_FIRST = 1u << 5, DOT_CIN = 1u << 6, DOT_COUT = 1u << 7,
                   DOT_ROW = 1u << 16, DOT_NEXT = 1u << 16, DOT_PLAIN = 1u << 17;
constexpr int kDotTerms = 8;    // products of a unit
constexpr int kDotBackWarps = 16;  // warps of the top's backward CTA
// products of a chain's row (two rows in registers)
constexpr int dot_chain_terms(int elem) { return elem == 4 ? 10 : 8; }
constexpr int kDotChunk = 32;   // quads of a chunk: one 16-byte load per lane
constexpr int kDotAhead = 3;    // chunks that a stream ends in (two are read past the one run)
constexpr int kDotMaxMid = 14;  // mid barriers of one tick (ids 1..14)

struct DotPlan {
  int bins = 0;        // bins of the bottom (0: every column is in the top)
  int top_warps = 16;
  double cap = 1.0;    // largest part, of a bin's even share
  int mid = 0;         // CTAs of the mid stage (0: none)
  double mid_cap = 1.0;  // largest part, of such a CTA's even share
  int prep_cols = 4;   // columns of a CTA of the prep after it
  int chain = 8;       // longest rows of a chain
  int pack = 3;        // longest sums that are packed by fours (0: none)
  int ahead = 2;       // ticks by which values are touched before their use (0: not)
  int keep = 700;      // values touched since, after which one is taken to have left the L1
};

struct DotProgram {
  DotPlan plan;
  std::vector<uint32_t> words;                   // all streams, 4 words per quad
  std::vector<int32_t> bottom, prep, mid, prep2, top, tback, midback, back;  // per bin / warp: first quad of its stream
  bool with_subst = false;                       // forward and backward substitution included
};

// Programs address a group's values by 32-bit byte offsets: a matrix with more
// slots (some 16 million, an 800,000-bus grid) keeps the streams.
inline bool dot_fits(const Schedule& sc) { return (int64_t)std::max(sc.n_slots, sc.n_u) * 256 < ((int64_t)1 << 32); }

// The plan taken where nothing is timed, for `groups` groups of scenarios, and
// the plans the autotuner times.
DotPlan dot_default(const Schedule& sc, int elem, int groups);
std::vector<DotPlan> dot_candidates(const Schedule& sc, int elem, int groups);
// Whether a plan made for few groups is the one to run `groups` groups with: an
// SM for each CTA of the mid stage (three of them at least, the fewest that pay).
bool dot_few(const DotPlan& p, int groups);

// Compiles the refactor of a schedule (with both substitutions when the
// schedule fuses the forward one).
void build_dot(const Schedule& sc, const DotPlan& plan, DotProgram& out);

// Host interpreter of a program for one scenario in FP64, with the checks
// that make the device's order of execution irrelevant: every index in
// range, every value final when it is read and written by the same warp
// earlier or in an earlier tick or launch (reads checked when the device
// issues them), no two warps on one value in one tick, equal barrier counts,
// every sum complete and in order.  Returns an empty string or the first
// violation.
std::string run_dot_host(const Schedule& sc, const DotProgram& p, std::vector<double>& lu,
                         const std::vector<double>& rhs, std::vector<double>& X, bool& singular);

}  // namespace gox
