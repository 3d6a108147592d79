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
constexpr int kSlRing = 3;    // stages copied ahead of use
constexpr int kSlOpRing = 4;  // op pages of a warp
constexpr int kSlSmemMax = 224 * 1024;  // dynamic shared memory of a block

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

// Op pages, uint4 per lane (bits of the four words in little-endian order): a0 b0
// (15 bits each), k0 (13), a1 b1 (15 each), k1 (13), t (15), ini (11), reach (5),
// bit 117: add the previous lane's sum, scan steps (3 bits), level ends after the
// page (7 bits).  A term is M[a] M[b] M[k]; positions: the diagonal [0, N), the
// factor's entries [N, N + nl), zero at N + nl, carries above.  k is a diagonal
// position, ini counts from zero's.  Padding has a = b = zero and the k of the
// lane's first term, or node 0, which is a leaf: values that are final.
struct SlOpField {
  int bit, width;
};
constexpr SlOpField kSlOpA[2] = {{0, 15}, {43, 15}}, kSlOpB[2] = {{15, 15}, {58, 15}},
                    kSlOpK[2] = {{30, 13}, {73, 13}}, kSlOpT = {86, 15}, kSlOpIni = {101, 11};
constexpr int kSlOpMaxWait = 127;

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

// whether the instance may take this factorisation (else the block kernels with
// global scratch, or the supernodal one): positions within the op fields and V in
// a block's shared memory.  Up to that limit this wins, also with one block per SM:
// MPC problems of n = 1200 to 2000 (14 to 23 k positions), 8 iterations, alone
// 5.7-8.1 ms against 45-58 by the block kernels, 512 of them 20-31 against 90-111;
// three semidefinite blocks of side 12 (20 k), alone 28 against 59, 256 of them
// 43 against 90.
inline bool sl_fits(const Prepared &p) {
  const long long nl = (long long)p.Li.size();
  return !p.supernodal && p.N > 0 && (long long)p.N * 8 <= 48 * 1024 &&
         p.N + nl < (1 << kSlOpT.width) && (p.N + nl) * 8 <= kSlSmemMax &&
         (long long)p.Kj.size() < (1 << 22);
}
// vgroup: consecutive terms a lane reads in one 16-byte load of values (2 for
// FP64, 4 for FP32).  False: a field is out of range, or a block's shared memory
// too small (the instance then takes the block kernels).
bool sl_build(const Prepared &p, int vgroup, SlicedPlan &s);

// Dynamic shared memory of an instance's blocks: solves with one and two sides, the
// factorisation in FP64 and in FP32.
struct SlNeed {
  long long solve[2], factor[2];
};
SlNeed sl_need(const SlicedPlan &p);

// position of (term r, lane) inside a stage of `used` lanes that hold groups of v
// consecutive terms side by side
inline int sl_at(int r, int lane, int v, int used) {
  return (r / v) * used * v + lane * v + r % v;
}

// `width` bits from `bit` on of an op page's lane words
inline unsigned sl_op_field(const uint32_t *w, int bit, int width) {
  const unsigned long long lo = w[bit / 32], hi = bit / 32 + 1 < 4 ? w[bit / 32 + 1] : 0;
  return (unsigned)(((lo | (hi << 32)) >> (bit % 32)) & ((1ull << width) - 1));
}
inline unsigned sl_op_field(const uint32_t *w, SlOpField f) {
  return sl_op_field(w, f.bit, f.width);
}

}  // namespace clgpu
