// sliced.hpp -- host-side layouts of the block-per-instance sparse LDL^T
// (ldl_sliced.cu): the substitution and residual pages and the factorisation
// op pages of one prepared instance.
//
// Every sparse sum of the kernels (a row of L, a column of L, a row of K, the
// updates of one factor entry) is a segment of a stream: the level's (for K:
// the matrix's) terms in a fixed order.  The order of additions of a segment
// follows from its place in the stream alone: the stream is cut into chunks
// of 32 lanes of R terms (R = 4, ops 2); the terms of a segment inside one lane
// (a run) are added in turn, the lanes' sums by a doubling scan, and the sum
// up to a chunk's end is the first term of the segment's part in the next
// chunk (a carry).  Keeping that order fixed makes results independent of how
// the sums are spread over warps.
//
// A page gives one lane to each run: 32 lanes of R terms whose segments are
// whole parts (all lanes of a part side by side), in any order, from any
// chunk of the level.  So every lane adds at most R terms, straight-line, and a
// page's scan only takes the steps its widest part needs.
//
// The substitutions and the residual run in stages of up to kSlStagePages
// pages of one level, one page per warp, every stage ending with a meeting of
// the block; only a stage's used lanes are stored (narrow levels fill one page
// in part).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "setup.hpp"

namespace clgpu {

constexpr int kSlWarps = 4;       // warps per instance (one block)
constexpr int kSlStagePages = 3;  // pages of a stage: the fourth warp copies
constexpr int kSlStage = 32 * kSlStagePages;
constexpr int kSlRun = 4;         // terms per lane of a substitution page
constexpr int kSlPage = 32 * kSlRun;
constexpr int kSlOpRun = 2;       // ops per lane of an op page
constexpr int kSlOpWords = 4 * 32;  // words of an op page
constexpr uint16_t kSlNone = 0xffff;

// Stage words, uint4 per lane, low halves: 8 * the gathered slots of the
// lane's terms (byte offsets of one vector); high halves:
//   .x  target slot of the part (on its last lane; else N)
//   .y  reach (lanes back the scan adds, bits 0..4), bit 5: instead of the
//       scan, the previous lane's scanned sum is added at the end
//   .z  slot of the run's first addend (a carry; else N)
//   .w  the page's control, the same on every lane: scan steps (bits 0..2),
//       bit 3: some lane has a carry, bit 4: some lane adds the previous
//       lane's sum
// Slots: [0, N) the vector, N zero, above: carries.  A part whose target is a
// carry stores its sum there; else the sum is the segment's.

// Op pages, uint4 per lane: 14-bit fields a0 b0 k0 a1 b1 k1 t ini (bits 0..111
// of the four words in little-endian order), reach (5 bits), bit 117: add the
// previous lane's sum, scan steps (3 bits), level ends after the page (7
// bits).  A term is M[a] M[b] M[k]; positions: the diagonal [0, N), the factor's
// entries [N, N + nl), zero at N + nl, carries above.
constexpr int kSlOpMaxWait = 127;
constexpr int kSlOpPositions = 1 << 14;

// One warp's op pages: count[w] from first[w] after skip[w] level ends.
struct SlRange {
  int first[kSlWarps], count[kSlWarps], skip[kSlWarps];
};

struct SlicedPlan {
  int N = 0, nl = 0, nlev = 0;
  int ncarry = 0, nopcarry = 0;   // carry slots
  int nstage[3] = {0, 0, 0}, olevels = 0;  // forward, backward, residual
  std::vector<uint8_t> used;      // stored lanes of every stage, pass by pass
  std::vector<uint32_t> ent;      // four words per stored lane
  // substitutions: factor entry of every stored value (kSlNone: zero)
  std::vector<uint16_t> lpos;
  // residual: the stored position of every CSR entry of K, and the work
  // position a stored value initialises in the factorisation (kSlNone: the
  // upper triangle, padding)
  std::vector<int> kslot;
  std::vector<uint16_t> kdst;
  // factorisation: op pages; the nodes of the first level (no updates; every
  // other node's pivot follows the last update of its diagonal); the expected
  // pivot signs; entry -> column
  std::vector<uint32_t> ops;
  SlRange op;
  std::vector<uint16_t> leaf, ecol;
  std::vector<signed char> sign;
};

// whether the instance takes this factorisation (else the block kernels with
// global scratch, or the supernodal one)
inline bool sl_fits(const Prepared &p) {
  const long long nl = (long long)p.Li.size();
  return !p.supernodal && p.N > 0 && (long long)p.N * 8 <= 48 * 1024 &&
         (p.N + nl) * 8 + 4096 <= 96 * 1024 && (long long)p.Kj.size() < (1 << 22);
}
// vgroup: consecutive terms a lane reads in one 16-byte load of values (2 for
// FP64, 4 for FP32).  False: a field is out of range (the instance then takes
// the block kernels).
bool sl_build(const Prepared &p, int vgroup, SlicedPlan &s);

// position of (term r, lane) inside a stage of `used` lanes that hold groups of v
// consecutive terms side by side
inline int sl_at(int r, int lane, int v, int used) {
  return (r / v) * used * v + lane * v + r % v;
}

// field f (14 bits) of an op page's lane words
inline unsigned sl_op_field(const uint32_t *w, int bit, int width) {
  const unsigned long long lo = w[bit / 32], hi = bit / 32 + 1 < 4 ? w[bit / 32 + 1] : 0;
  return (unsigned)(((lo | (hi << 32)) >> (bit % 32)) & ((1ull << width) - 1));
}

}  // namespace clgpu
