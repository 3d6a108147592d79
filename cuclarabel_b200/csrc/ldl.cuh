// ldl.cuh -- batched sparse LDL^T of the quasi-definite KKT systems.
//
// Stands in for the reference's cuDSS calls (src/kktsolvers/gpu/
// directldl_cudss.jl:30-59 and directldl_mixed_cudss.jl:42-78), which are not
// available in this environment.  The host computes a fill-reducing ordering
// and the symbolic factorisation once per instance (setup.cpp); the device
// refactors every IPM iteration and solves with iterative refinement
// (kktsolver_directldl_gpu.jl:300-409).
#pragma once
#include "common.cuh"

namespace clgpu {

struct SnExec;

// blocks per SM the register budgets of the class-1 kernels aim at
constexpr int kSlSolveBlocks = 5;
constexpr int kSlFactorBlocks = 6;

// One class-1 instance: sizes, and where its part of each array begins.
struct SlWarp {  // one warp's op pages (from the instance's first)
  int opage, nop, oskip;
};
struct SlInst {
  int N, nl, nk;        // dimension, entries of L, of K
  int voff;             // vectors
  int stage0;           // stage table
  int nf, nb, nr;       // stages of the forward, backward, residual pass
  int lane0;            // words
  int vlane0, nvlane;   // factor values
  int kx0, nkx;         // stored K values
  int opage0, nops;     // op stream, its words
  int nleaf;            // nodes of the first level
  int ecol0;
  int ncarry, nopcarry; // carry slots
  SlWarp w[4];
};
// launches of one kind: instances of similar shared-memory need together
struct SlGroup {
  int first, count, smem, smem2;
};
struct SlGroups {
  int n;
  SlGroup g[4];
};

struct KKTDev {
  int B;
  const int *N;     // [B] KKT dimension of each instance
  const int *voff;  // [B+1] offsets of per-instance vectors (sum of N)
  const int *poff;  // [B]   offsets into the (N+1)-long pointer arrays
  // permuted full KKT (both triangles), CSR with global positions
  const int *Kp, *Kj;
  double *Kx;
  const int *Kdiag;          // [sum N] position of the diagonal of each row
  const signed char *Dsign;  // [sum N] +1 / -1
  const int *gsrc;           // [sum N] rhs gather / solution scatter codes
  // factor L (strict lower, CSC with global positions) and D
  const int *Lp, *Li;
  void *Lx, *D, *Dinv;  // double or float (mixed precision)
  // row pattern of L: for column j the list (k, pos of L(j,k))
  const int *Rp, *Rk, *Rpos;
  // elimination-tree levels: nodes of level l of instance i are
  // lvl_nodes[voff[i] + lvl_ptr[lvl_off[i] + l] .. lvl_ptr[lvl_off[i] + l + 1])
  const int *lvl_off, *nlev, *lvl_ptr, *lvl_nodes;
  // substitution schedules, one int4 per node:
  //   fsched[voff[i] + t] = {node, Rp[node], Rp[node+1], 0} in level order
  //     (leaves first);
  //   bsched[voff[i] + t] = {node, Lp[node], Lp[node+1], 0} in backward order
  //     (root level first: level l occupies [N - lvl_ptr[l+1], N - lvl_ptr[l]))
  const int4 *fsched, *bsched;
  // copy of L's values in row-pattern order (LxR[r] = Lx[Rpos[r]]), written at
  // the end of every factorisation so the forward substitution reads L rows
  // contiguously; same element type as Lx
  void *LxR;
  // Block-per-instance factorisation and solves (class 1, ldl_sliced.cu): the
  // instances' layouts (sliced.hpp) concatenated.  Their K values are stored
  // in the residual's page order (every position map points there).
  const SlInst *sl;                // [B]
  const uint16_t *sl_kdst;         // per stored K value of the batch
  const uint8_t *sl_used;          // stage tables: stored lanes of each stage
  const uint32_t *sl_ent, *sl_ops;
  const uint16_t *sl_lpos, *sl_leaf, *sl_ecol;
  const signed char *sl_sign;      // [sum N] expected pivot signs
  const int *sl_kdiag;             // [sum N] stored position of K's diagonal
  void *sl_val;                    // double or float: factor values, page order
  const int *sl_solve_inst, *sl_factor_inst;  // launch order (largest first)
  SlGroups sl_solve, sl_factor;
  // profiling only (else null): per instance, algorithmic bytes moved by the
  // factorisations [0, B), the one-side solves [B, 2B) and the two-side
  // solves [2B, 3B) of the profiled solve
  double *prof_bytes;
  // [B] kernel class: 1 = one block with everything in shared memory (the
  // layouts above), 2 = block kernels with global scratch, 3 = supernodal
  // (sn below; no scalar factor structures)
  const int *cls;
  // supernodal factorisation of the class-3 instances (host object; null
  // when there are none)
  SnExec *sn;
  int has_large;  // some class-2 instance
  // scratch (global, per instance, sum N each)
  double *w;       // dense factor accumulator (large instances)
  double *yf;      // substitution work vector (large instances)
  // FP32-stored factor only (null otherwise): the FP64 factor values and
  // pivots the factorisation itself runs on; the solves read the FP32 copy
  double *Lacc;
  double *Dacc;
  // solve scratch per instance (sum N each): right-hand side b, accepted
  // iterate x and residual e of the first and the second side
  double *b, *x, *e, *b2, *x2, *e2;
  double *dx;
};

// Right-hand sides of one solve launch: side r gathers its rhs from rx[r] /
// rz[r] and scatters its solution to lx[r] / lz[r] (either may be null).
template <int NR>
struct SolveIO {
  const double *rx[NR], *rz[NR];
  double *lx[NR], *lz[NR];
};

struct LDLParams {
  int static_reg;
  double static_c, static_prop;
  int dyn_reg;
  double dyn_eps, dyn_delta;
  int ir_enable, ir_maxiter;
  double ir_reltol, ir_abstol, ir_stopratio;
};

// numeric refactorisation of every instance with run[i] != 0; sets
// ok[i] = 0 if a pivot is not finite; eps_out[i] receives the static
// regulariser used (diagonal_regularizer of the reference).  fp32 stores the
// factor in FP32; arith32 (with fp32) also eliminates in FP32 arithmetic,
// otherwise the elimination is FP64.
void ldl_factor(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
                int *ok, double *eps_out, cudaStream_t st, bool arith32 = false);
// solve K [lx; lz; *] = [rx; rz; 0] with iterative refinement for every
// instance with run[i] != 0.  rx/lx are indexed by global x index, rz/lz by
// global s/z row; lx or lz may be null.  ok[i] cleared on non-finite results.
void ldl_solve(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
               const double *rx, const double *rz, double *lx, double *lz,
               int *ok, cudaStream_t st);
// two right-hand sides with the same factor in one launch: side 0 (rx0, rz0)
// -> (lx0, lz0), side 1 likewise; each result is exactly that of ldl_solve
void ldl_solve2(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
                const double *rx0, const double *rz0, double *lx0, double *lz0,
                const double *rx1, const double *rz1, double *lx1, double *lz1, int *ok,
                cudaStream_t st);

// the same for the class-1 instances only (ldl_sliced.cu)
void sl_factor(const KKTDev &k, bool fp32, bool arith32, const LDLParams &p, const int *run,
               int *ok, double *eps_out, cudaStream_t st);
void sl_solve(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
              const SolveIO<1> &io, int *ok, cudaStream_t st);
void sl_solve2(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
               const SolveIO<2> &io, int *ok, cudaStream_t st);

}  // namespace clgpu
