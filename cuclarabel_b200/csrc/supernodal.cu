// supernodal.cu -- numeric supernodal (multifrontal) LDL^T and solves.
//
// Plays cuDSS's numeric role for the large problems: refactor! every IPM
// iteration (src/kktsolvers/gpu/directldl_cudss.jl:37-46; FP32 for
// :cudssmixed, directldl_mixed_cudss.jl:42-60) and solve! with the FP64
// iterative refinement of kktsolver_directldl_gpu.jl:349-410.  The plan
// (front layout, maps, per-level launch lists) comes from supernodal.cpp.
//
// Factorisation, level by level from the leaves (every task list of a
// level is one launch):
//   small fronts  one block assembles the front in shared memory (original
//                 entries, children's Schur complements), eliminates its
//                 pivots and writes L, D and the Schur complement back;
//   blocked       k_sn_assemble zeroes and assembles column ranges of the
//   fronts        front (a task owns its columns, so children are added in a
//                 fixed order without atomics), then per panel of K <= 128
//                 pivots: k_sn_diag factors the K x K diagonal block,
//                 k_sn_trsm solves every 128-row tile below by triangular
//                 substitution (W = A L11^-T, L = W D^-1), and
//                 k_sn_update_* subtracts L W^T from every lower tile of the
//                 trailing matrix.  FP64 tiles run on the tensor cores (DMMA,
//                 mma.sync m8n8k4), FP32 tiles (mixed form) on FMA units;
//                 both stage their operands with cp.async.
// Solve: forward substitution leaves first (small fronts one warp each,
// blocked fronts one block per row tile, the panels' solutions handed on
// through flags), D^-1, backward substitution roots first.
// Every reduction runs in a fixed order: results do not depend on timing.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "common.cuh"
#include "ldl.cuh"
#include "sn_exec.cuh"
#include "pinned.hpp"

namespace clgpu {

namespace {

// trailing update tiles: 128 rows x kUpdCols columns, k in chunks of kUpdKC
constexpr int kUpdCols = 64;
constexpr int kUpdKC = 16;
constexpr int kUpdStages = 3;
constexpr int kUpdLdA = kSnNB + 4;     // shared row strides (elements): 4 mod 16 (FP64
constexpr int kUpdLdB = kUpdCols + 4;  // banks), so DMMA fragment loads are conflict-free
static_assert(kSnKPad % kUpdKC == 0, "panel widths are whole update chunks");
constexpr int kDiagThreads = 256;
constexpr int kTrsmThreads = 256;
constexpr int kAsmThreads = 256;
constexpr int kSmallThreads = 128;

// two consecutive elements of a front (8- or 16-byte aligned pairs)
template <typename T>
struct Pair {
  T x, y;
};
__device__ __forceinline__ Pair<double> load_pair(const double *p) {
  const double2 w = *reinterpret_cast<const double2 *>(p);
  return {w.x, w.y};
}
__device__ __forceinline__ Pair<float> load_pair(const float *p) {
  const float2 w = *reinterpret_cast<const float2 *>(p);
  return {w.x, w.y};
}
__device__ __forceinline__ void store_pair(double *p, Pair<double> w) {
  *reinterpret_cast<double2 *>(p) = make_double2(w.x, w.y);
}
__device__ __forceinline__ void store_pair(float *p, Pair<float> w) {
  *reinterpret_cast<float2 *>(p) = make_float2(w.x, w.y);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
// D(8x8) += A(8x4) B(4x8), FP64 tensor cores.  Fragments: a = A[lane/4][lane%4],
// b = B[lane%4][lane/4], (c0, c1) = C[lane/4][2 (lane%4) + {0, 1}].
__device__ __forceinline__ void dmma884(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// dynamic regularisation (QDLDL's Dsigns rule, kktsolver_directldl.jl:224-229)
__device__ __forceinline__ double sn_pivot(double dj, int sg, const LDLParams &prm) {
  if (prm.dyn_reg && double(sg) * dj <= prm.dyn_eps) dj = prm.dyn_delta * double(sg);
  return dj;
}
__device__ __forceinline__ int pivot_sign(const KKTDev &k, int g) {
  return g >= 0 ? int(k.Dsign[g]) : 1;
}

// ------------------------------------------------------------------ eps
// static regulariser per instance: c + prop * max |diag(K)|
// (_compute_regularizer, kktsolver_directldl.jl:299-313)
__global__ void k_sn_eps(SnDev d, KKTDev k, LDLParams prm, const int *insts, const int *run,
                         double *eps_out) {
  const int inst = insts[blockIdx.x];
  if (!run[inst]) return;
  __shared__ double red[kAsmThreads / 32];
  double mx = 0;
  if (prm.static_reg)
    for (int v = k.voff[inst] + threadIdx.x; v < k.voff[inst + 1]; v += kAsmThreads)
      mx = fmax(mx, fabs(k.Kx[k.Kdiag[v]]));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kAsmThreads / 32; ++w) mx = fmax(mx, red[w]);
    mx = fmax(mx, red[0]);
    const double eps = prm.static_reg ? prm.static_c + prm.static_prop * mx : 0.0;
    d.eps[inst] = eps;
    if (eps_out) eps_out[inst] = eps;
  }
}

// --------------------------------------------------------- small fronts
// One block per front of at most kSnSmallMax rows: assemble in shared
// memory, eliminate the ncol pivots (right-looking), write back.
template <typename T>
__global__ void __launch_bounds__(kSmallThreads) k_sn_small(SnDev d, KKTDev k, LDLParams prm,
                                                           int base, const int *run, int *ok) {
  const int s = d.tasks[base + blockIdx.x].x, inst = d.inst[s];
  if (!run[inst]) return;
  extern __shared__ __align__(16) unsigned char sraw[];
  const int ld = d.ld[s], nc = d.ncol[s], tid = threadIdx.x;
  T *f = reinterpret_cast<T *>(sraw);
  T *col = f + ld * ld;
  for (int i = tid; i < ld * ld; i += kSmallThreads) f[i] = T(0);
  __syncthreads();
  const int2 *am = d.amap;
  for (int q = d.acol[d.cbase[s]] + tid; q < d.acol[d.cbase[s] + nc]; q += kSmallThreads)
    f[am[q].y] = T(k.Kx[am[q].x]);
  __syncthreads();
  const double eps = d.eps[inst];
  for (int c = tid; c < nc; c += kSmallThreads) {
    const int g = d.col0g[s] + c;
    f[c * ld + c] += T(k.Dsign[g] > 0 ? eps : -eps);
  }
  __syncthreads();
  const T *F = reinterpret_cast<const T *>(d.F);
  for (int a = d.ch_ptr[s]; a < d.ch_ptr[s + 1]; ++a) {
    const int c = d.ch[a], cn = d.nrow[c], cld = d.ld[c], cu = d.u0[c];
    const int *rel = d.rel + d.rel_off[c];
    const T *cf = F + d.foff[c];
    for (int q = 0; q < cn; ++q) {
      const int pc = rel[q];
      for (int r = q + tid; r < cn; r += kSmallThreads)
        f[pc * ld + rel[r]] += cf[(long long)(cu + q) * cld + cu + r];
    }
    __syncthreads();
  }
  bool bad = false;
  for (int j = 0; j < nc; ++j) {
    const int g = d.col0g[s] + j;
    const T dj = T(sn_pivot(double(f[j * ld + j]), k.Dsign[g], prm));
    for (int i = j + 1 + tid; i < ld; i += kSmallThreads) col[i] = f[j * ld + i];
    __syncthreads();
    {
      // rank-1 update of the trailing lower triangle: 16 x 8 threads
      const int tx = tid & 15, ty = tid >> 4;
      for (int r = j + 1 + ty; r < ld; r += kSmallThreads / 16) {
        const T cr = col[r];
        for (int i = j + 1 + tx; i < ld; i += 16)
          if (i >= r) f[r * ld + i] -= (col[i] / dj) * cr;
      }
    }
    for (int i = j + 1 + tid; i < ld; i += kSmallThreads) f[j * ld + i] = col[i] / dj;
    if (tid == 0) {
      f[j * ld + j] = dj;
      const double di = 1.0 / double(dj);
      d.Dinv[g] = di;
      if (!isfinite(di) || !isfinite(double(dj))) bad = true;
    }
    __syncthreads();
  }
  T *out = reinterpret_cast<T *>(d.F) + d.foff[s];
  for (int i = tid; i < ld * ld; i += kSmallThreads) {
    const int c = i / ld, r = i % ld;
    if (r >= c) out[i] = f[i];
  }
  if (bad) ok[inst] = 0;
}

// ------------------------------------------------------- blocked fronts
// Assembly of columns [ca, cb) of a blocked front: zero (rows c..ld), the
// original entries (+ static regularisation), unit dummy pivots, then the
// Schur complements of the children that touch these columns, in child
// order (the plan lists them per 8-column chunk with their entry ranges).
template <typename T>
__global__ void __launch_bounds__(kAsmThreads) k_sn_assemble(SnDev d, KKTDev k, int base,
                                                            const int *run) {
  const int4 t = d.tasks[base + blockIdx.x];
  const int s = t.x, ca = t.y, cb = t.z, inst = d.inst[s];
  if (!run[inst]) return;
  const long long ld = d.ld[s];
  const int nc = d.ncol[s], u0 = d.u0[s], tid = threadIdx.x;
  T *f = reinterpret_cast<T *>(d.F) + d.foff[s];
  for (int c = ca; c < cb; ++c)
    for (long long r = c + tid; r < ld; r += kAsmThreads) f[c * ld + r] = T(0);
  __syncthreads();
  const double eps = d.eps[inst];
  const int ce = min(cb, nc);
  if (ca < ce) {
    const int2 *am = d.amap;
    for (int q = d.acol[d.cbase[s] + ca] + tid; q < d.acol[d.cbase[s] + ce]; q += kAsmThreads) {
      const int2 e = am[q];
      double v = k.Kx[e.x];
      const int c = e.y / (int)ld, r = e.y - c * (int)ld;
      if (r == c) v += k.Dsign[d.col0g[s] + c] > 0 ? eps : -eps;
      f[e.y] = T(v);
    }
  }
  for (int c = max(ca, nc) + tid; c < min(cb, u0); c += kAsmThreads) f[c * ld + c] = T(1);
  __syncthreads();
  const T *F = reinterpret_cast<const T *>(d.F);
  // the children touching columns [ca, cb), in child order (plan)
  for (int a = d.cl_ptr[t.w]; a < d.cl_ptr[t.w + 1]; ++a) {
    const int4 cq = d.clist[a];
    const int c = cq.x, qa = cq.y, qb = cq.z, cn = d.nrow[c], cu = d.u0[c];
    const long long cld = d.ld[c];
    const int *rel = d.rel + d.rel_off[c];
    const T *cf = F + d.foff[c];
    for (int q = qa; q < qb; ++q) {
      const long long pc = rel[q];
      const T *src = cf + (cu + q) * cld + cu;
      // four rows per thread per round, their loads issued before any add
      // (the parent positions of one column are distinct)
      for (int r0 = q + tid; r0 < cn; r0 += 4 * kAsmThreads) {
        int rr[4];
        T sv[4], fv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int r = r0 + u * kAsmThreads;
          rr[u] = r < cn ? rel[r] : 0;
          sv[u] = r < cn ? src[r] : T(0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (r0 + u * kAsmThreads < cn) fv[u] = f[pc * ld + rr[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (r0 + u * kAsmThreads < cn) f[pc * ld + rr[u]] = fv[u] + sv[u];
      }
    }
    __syncthreads();
  }
}

// Diagonal block of a panel: factor the K x K block (the static shift was
// applied at assembly), write L11 and D to the front and 1/d to the
// workspace.  Blocked right-looking LDL^T in 32-column blocks, every column
// kept unscaled until the end (L(:, j) = a(:, j) / d_j is written last):
//   1. one warp factors the 32 x 32 diagonal block (lane i owns row i; step
//      j subtracts a(i, j) (a(k, j) / d_j) from a(i, k), j < k <= i), with
//      the pivot rule applied to each pivot as it becomes final;
//   2. every row below the block (one thread each, the row in registers)
//      takes the same 32 steps against the block's columns;
//   3. the trailing lower triangle -= X D^-1 X^T over the block's 32
//      columns, 6 x 6 outputs per thread.
// Three barriers per column block instead of one per pivot.  Pivot signs
// and D's global positions are staged first.
// The block width is a template argument (32, or 16 for the last block): with a
// run-time width every multiply-add carried its own guard and waited for its own
// shared load (38 cycles each; a 128-pivot block took 106 us, now 42).
constexpr int kDiagNB = 32;
template <typename T, int NB>
__device__ __forceinline__ void diag_block(T *blk, T *wsc, double *dinv, T *dd, const int *sgn,
                                           const LDLParams &prm, int b0, int K) {
  const int tid = threadIdx.x;
  // 1. the diagonal block, one warp, a row per lane in registers.  Column j goes
  // through shared memory for the other lanes, except the one entry that the
  // next pivot waits for (a shuffle).
  if (tid < 32) {
    const int i = tid;
    T x[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) x[j] = blk[(b0 + j) * K + b0 + min(i, NB - 1)];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      T *cj = blk + (b0 + j) * K + b0;
      const T dj = T(sn_pivot(double(__shfl_sync(0xffffffffu, x[j], j)), sgn[b0 + j], prm));
      const double di = 1.0 / double(dj);
      if (i == 0) {
        dd[b0 + j] = dj;
        dinv[b0 + j] = di;
      }
      if (i > j && i < NB) cj[i] = x[j];
      const T li = x[j] * T(di);
      if (j + 1 < NB) x[j + 1] -= li * __shfl_sync(0xffffffffu, x[j], (j + 1) & 31);
      __syncwarp();
#pragma unroll
      for (int q = j + 2; q < NB; ++q) x[q] -= li * cj[q];
    }
  }
  __syncthreads();
  const int rb = b0 + NB, m = K - rb;  // rows below the block
  if (m <= 0) return;
  // 2. the rows below, one thread each
  if (tid < m) {
    const int r = rb + tid;
    T x[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) x[j] = blk[(b0 + j) * K + r];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const T lj = x[j] * T(dinv[b0 + j]);
      wsc[j * kSnNB + tid] = lj;
#pragma unroll
      for (int q = j + 1; q < NB; ++q) x[q] -= lj * blk[(b0 + j) * K + b0 + q];
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) blk[(b0 + j) * K + r] = x[j];
  }
  __syncthreads();
  // 3. trailing lower triangle: a(r, c) -= sum_j x(r, j) (x(c, j) / d_j), the
  // lower 16 x 16 blocks only; rows and columns beyond m read whatever lies there
  // and are not stored
  const int tx = tid & 15, ty = tid >> 4;
  T acc[6][6];
#pragma unroll
  for (int u = 0; u < 6; ++u)
#pragma unroll
    for (int v = 0; v <= u; ++v) acc[u][v] = T(0);
#pragma unroll 4
  for (int j = 0; j < NB; ++j) {
    T xa[6], wb[6];
#pragma unroll
    for (int u = 0; u < 6; ++u) {
      xa[u] = blk[(b0 + j) * K + rb + tx + 16 * u];
      wb[u] = wsc[j * kSnNB + ty + 16 * u];
    }
#pragma unroll
    for (int u = 0; u < 6; ++u)
      if (16 * u < m) {
#pragma unroll
        for (int v = 0; v <= u; ++v) acc[u][v] += xa[u] * wb[v];
      }
  }
#pragma unroll
  for (int u = 0; u < 6; ++u)
#pragma unroll
    for (int v = 0; v <= u; ++v) {
      const int rr = tx + 16 * u, cc = ty + 16 * v;
      if (rr < m && cc <= rr) blk[(rb + cc) * K + rb + rr] -= acc[u][v];
    }
  __syncthreads();
}
template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_sn_diag(SnDev d, KKTDev k, LDLParams prm,
                                                         int base, const int *run, int *ok) {
  const int4 t = d.tasks[base + blockIdx.x];
  const int s = t.x, k0 = t.y & 0xffff, K = t.y >> 16, inst = d.inst[s];
  if (!run[inst]) return;
  extern __shared__ __align__(16) unsigned char sraw[];
  T *blk = reinterpret_cast<T *>(sraw);       // K x K, column-major, stride K
  T *wsc = blk + kSnNB * kSnNB;               // scaled block columns, [kDiagNB][kSnNB]
  __shared__ double dinv[kSnNB];
  __shared__ T dd[kSnNB];
  __shared__ int gix[kSnNB], sgn[kSnNB];
  const long long ld = d.ld[s];
  T *f = reinterpret_cast<T *>(d.F) + d.foff[s];
  T *ws = reinterpret_cast<T *>(d.W) + d.woff[s];
  const int *fi = d.fidx + d.fix_off[s];
  const int tid = threadIdx.x;
  // stage the block by row pairs (16-byte loads for FP64), a fixed trip
  // count so that many loads are in flight; the strict upper part is not
  // read by the factorisation below
#pragma unroll 8
  for (int it = 0; it < kSnNB * kSnNB / 2 / kDiagThreads; ++it) {
    const int p = tid + it * kDiagThreads, c = p >> 6, r = (p & 63) * 2;
    if (c < K && r < K) store_pair(blk + c * K + r, load_pair(f + (k0 + c) * ld + k0 + r));
  }
  for (int j = tid; j < K; j += kDiagThreads) {
    const int g = fi[k0 + j];
    gix[j] = g;
    sgn[j] = pivot_sign(k, g);
  }
  __syncthreads();
  for (int b0 = 0; b0 < K; b0 += kDiagNB) {
    if (K - b0 >= kDiagNB)  // K is a multiple of 16
      diag_block<T, kDiagNB>(blk, wsc, dinv, dd, sgn, prm, b0, K);
    else
      diag_block<T, 16>(blk, wsc, dinv, dd, sgn, prm, b0, K);
  }
#pragma unroll 8
  for (int it = 0; it < kSnNB * kSnNB / kDiagThreads; ++it) {
    const int p = tid + it * kDiagThreads, c = p >> 7, r = p & (kSnNB - 1);
    if (c < K && r < K && r >= c)
      f[(k0 + c) * ld + k0 + r] = r > c ? blk[c * K + r] * T(dinv[c]) : dd[c];
  }
  bool bad = false;
  for (int j = tid; j < kSnNB; j += kDiagThreads) {
    if (j < K) {
      const double di = dinv[j];
      if (gix[j] >= 0) d.Dinv[gix[j]] = di;
      ws[j] = T(di);
      if (!isfinite(di) || !isfinite(double(dd[j]))) bad = true;
    } else {
      ws[j] = T(0);
    }
  }
  if (bad) ok[inst] = 0;
}

// row q of the packed strict lower triangle: rows padded to even lengths, so that
// every row starts on a pair
__device__ __forceinline__ int lrow(int q) { return q * q / 2; }

// one column block of the TRSM below: (a) then (b), NB columns from b0
template <typename T, int NB>
__device__ __forceinline__ void trsm_block(T *X, const T *Lr, int b0, int K, int m, int half) {
  if (half == 0) {
    T x[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) x[j] = X[(b0 + j) * kSnNB + m];
#pragma unroll
    for (int j = 0; j < NB - 1; ++j)
#pragma unroll
      for (int q = j + 1; q < NB; ++q) x[q] -= x[j] * Lr[lrow(b0 + q) + b0 + j];
#pragma unroll
    for (int j = 0; j < NB; ++j) X[(b0 + j) * kSnNB + m] = x[j];
  }
  __syncthreads();
  if (b0 + NB < K) {
    T x[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) x[j] = X[(b0 + j) * kSnNB + m];
    // four columns at a time: their sums are independent chains
    constexpr int H = kTrsmThreads / kSnNB;
    for (int q0 = b0 + NB + half; q0 < K; q0 += 4 * H) {
      T acc[4] = {T(0), T(0), T(0), T(0)};
      const T *lq[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = min(q0 + u * H, K - 1);
        lq[u] = Lr + lrow(q) + b0;
      }
#pragma unroll
      for (int j = 0; j < NB; j += 2)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const Pair<T> l = load_pair(lq[u] + j);
          acc[u] += x[j] * l.x;
          acc[u] += x[j + 1] * l.y;
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q0 + u * H < K) X[(q0 + u * H) * kSnNB + m] -= acc[u];
    }
  }
  __syncthreads();
}

// TRSM of a panel's row tile: rows r0..r0+127 of panel [k0, k0+K),
// W = A L11^-T by substitution, then L = W D^-1: L overwrites A in the
// front, W goes to the workspace for the trailing update.  Blocked by 32
// columns: (a) each row (one thread) solves the block's 32 columns in
// registers against the block's unit lower triangle (row-oriented: w(m, q)
// = a(m, q) - sum_{j<q} w(m, j) L11(q, j)); (b) the later columns of the
// row take the block's contribution, sum_j w(m, j) L11(q, j), the two
// halves of the thread block splitting the columns.  Two barriers per
// column block.  The tile (K x 128, column-major) and the strict lower triangle
// of L11 packed by rows sit in shared memory.
template <typename T>
__global__ void __launch_bounds__(kTrsmThreads) k_sn_trsm(SnDev d, int base, const int *run) {
  const int4 t = d.tasks[base + blockIdx.x];
  const int s = t.x, k0 = t.y & 0xffff, K = t.y >> 16, r0 = t.z;
  if (!run[d.inst[s]]) return;
  extern __shared__ __align__(16) unsigned char sraw[];
  T *X = reinterpret_cast<T *>(sraw);  // column q of the tile at X + q kSnNB
  T *Lr = X + K * kSnNB;               // L11(q, j), j < q, at Lr[lrow(q) + j]
  const long long ld = d.ld[s];
  T *f = reinterpret_cast<T *>(d.F) + d.foff[s];
  const T *ws = reinterpret_cast<const T *>(d.W) + d.woff[s];
  T *wr = reinterpret_cast<T *>(d.W) + d.woff[s] + kSnNB + t.w * ld;
  const int tid = threadIdx.x;
  // the tile by cp.async, then L11 by row pairs, fixed trip counts (many 16-byte
  // loads in flight)
  constexpr int E = 16 / (int)sizeof(T), per = kSnNB / E;
#pragma unroll 8
  for (int it = 0; it < kSnNB * per / kTrsmThreads; ++it) {
    const int p = tid + it * kTrsmThreads, q = p / per, m = (p % per) * E;
    if (q < K) cp_async16(X + q * kSnNB + m, f + (k0 + q) * ld + r0 + m);
  }
  cp_async_commit();
#pragma unroll 8
  for (int it = 0; it < kSnNB * kSnNB / 2 / kTrsmThreads; ++it) {
    const int p = tid + it * kTrsmThreads, j = p >> 6, q = (p & 63) * 2;
    if (j < K && q + 1 > j && q < K) {
      const Pair<T> w = load_pair(f + (k0 + j) * ld + k0 + q);
      if (q > j) Lr[lrow(q) + j] = w.x;
      Lr[lrow(q + 1) + j] = w.y;  // q + 1 > j
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  const int m = tid & (kSnNB - 1), half = tid / kSnNB;
  for (int b0 = 0; b0 < K; b0 += 32) {
    // K is a multiple of 16, so a block has 32 or 16 columns
    if (K - b0 >= 32)
      trsm_block<T, 32>(X, Lr, b0, K, m, half);
    else
      trsm_block<T, 16>(X, Lr, b0, K, m, half);
  }
#pragma unroll 8
  for (int it = 0; it < kSnNB * kSnNB / 2 / kTrsmThreads; ++it) {
    const int p = tid + it * kTrsmThreads, q = p >> 6, mm = (p & 63) * 2;
    if (q < K) {
      const Pair<T> w = load_pair(X + q * kSnNB + mm);
      const T di = ws[q];
      store_pair(wr + (long long)q * ld + r0 + mm, w);
      store_pair(f + (k0 + q) * ld + r0 + mm, Pair<T>{w.x * di, w.y * di});
    }
  }
}

// Large fronts take their panels in pairs (see the plan), K up to 256: a tile is
// loaded and stored, and its pipeline filled, once per pair (a dimension-86 000
// KKT system's updates 92 -> 85 ms, 28 -> 30 TF/s; 37 is the DMMA rate).
// Trailing update of the blocked fronts, one 128 x 64 tile per block:
// front tile (r0, c0) -= L(r0.., panel) W(c0.., :)^T, entries on or below
// the diagonal only (r0 + m >= c0 + n).  K (a multiple of kSnKPad = 16) is
// streamed in chunks of kUpdKC through a kUpdStages-deep cp.async pipeline.
// FP64: 8 warps as 4 (rows) x 2 (columns), warp tile 32 x 32 of m8n8k4
// DMMA; 120 registers, so two blocks (16 warps) are resident per SM and
// one block's prologue and epilogue overlap the other's main loop.  The
// accumulators start from the front tile itself (its loads are issued
// before the operand pipeline fills, so their latency is hidden) and the
// products are subtracted as they come (W fragments negated), so the
// epilogue only stores.
constexpr int kUpdThreads = 256;
__global__ void __launch_bounds__(kUpdThreads, 2) k_sn_update_f64(SnDev d, int base, const int *run) {
  const int4 t = d.tasks[base + blockIdx.x];
  const int s = t.x, k0 = t.y & 0xffff, K = t.y >> 16, r0 = t.z, c0 = t.w;
  if (!run[d.inst[s]]) return;
  const long long ld = d.ld[s];
  double *f = reinterpret_cast<double *>(d.F) + d.foff[s];
  const double *Ag = f + k0 * ld + r0;
  const double *Bg = reinterpret_cast<const double *>(d.W) + d.woff[s] + kSnNB + c0;
  extern __shared__ __align__(16) unsigned char sraw[];
  double *sm = reinterpret_cast<double *>(sraw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 3, wn = warp >> 2;
  // accumulator (mi, ni, h) is front entry (r0 + m, c0 + n); the whole
  // tile lies inside the front (entries above the diagonal are read and
  // left unchanged)
  double acc[4][4][2];
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        acc[mi][ni][h] = f[(long long)(c0 + wn * 32 + ni * 8 + 2 * (lane & 3) + h) * ld + r0 +
                           wm * 32 + mi * 8 + (lane >> 2)];
  const int nchunks = K / kUpdKC;
  constexpr int kStage = kUpdKC * (kUpdLdA + kUpdLdB);
  auto load = [&](int chunk, int stage) {
    double *As = sm + stage * kStage, *Bs = As + kUpdKC * kUpdLdA;
    // A: kUpdKC columns x 64 pieces of 16 B; B: kUpdKC x 32
    for (int p = tid; p < kUpdKC * 64; p += kUpdThreads) {
      const int q = p >> 6, m = (p & 63) * 2;
      cp_async16(As + q * kUpdLdA + m, Ag + ((long long)chunk * kUpdKC + q) * ld + m);
    }
    for (int p = tid; p < kUpdKC * 32; p += kUpdThreads) {
      const int q = p >> 5, n = (p & 31) * 2;
      cp_async16(Bs + q * kUpdLdB + n, Bg + ((long long)chunk * kUpdKC + q) * ld + n);
    }
  };
#pragma unroll
  for (int st = 0; st < kUpdStages - 1; ++st) {
    if (st < nchunks) load(st, st);
    cp_async_commit();
  }
  for (int c = 0; c < nchunks; ++c) {
    cp_async_wait<kUpdStages - 2>();
    __syncthreads();
    const int nx = c + kUpdStages - 1;
    if (nx < nchunks) load(nx, nx % kUpdStages);
    cp_async_commit();
    const double *As = sm + (c % kUpdStages) * kStage;
    const double *Bs = As + kUpdKC * kUpdLdA;
#pragma unroll
    for (int kk = 0; kk < kUpdKC; kk += 4) {
      const int q = kk + (lane & 3);
      double a[4], b[4];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) a[mi] = As[q * kUpdLdA + wm * 32 + mi * 8 + (lane >> 2)];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) b[ni] = -Bs[q * kUpdLdB + wn * 32 + ni * 8 + (lane >> 2)];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma884(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
    }
  }
  cp_async_wait<0>();
  const bool diag = r0 < c0 + 64;  // the tile reaches above the diagonal
#pragma unroll
  for (int mi = 0; mi < 4; ++mi) {
    const int m = wm * 32 + mi * 8 + (lane >> 2);
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = wn * 32 + ni * 8 + 2 * (lane & 3) + h;
        if (!diag || r0 + m >= c0 + n) f[(long long)(c0 + n) * ld + r0 + m] = acc[mi][ni][h];
      }
  }
}

// FP32 form: 16 x 8 threads, each 8 x 8 outputs (rows ty*4 + {0..3} and
// 64 + ty*4 + {0..3}; columns tx*4 + {0..3} and 32 + tx*4 + {0..3}), FMA units.
__global__ void __launch_bounds__(128, 2) k_sn_update_f32(SnDev d, int base, const int *run) {
  const int4 t = d.tasks[base + blockIdx.x];
  const int s = t.x, k0 = t.y & 0xffff, K = t.y >> 16, r0 = t.z, c0 = t.w;
  if (!run[d.inst[s]]) return;
  const long long ld = d.ld[s];
  float *f = reinterpret_cast<float *>(d.F) + d.foff[s];
  const float *Ag = f + k0 * ld + r0;
  const float *Bg = reinterpret_cast<const float *>(d.W) + d.woff[s] + kSnNB + c0;
  extern __shared__ __align__(16) unsigned char sraw[];
  float *sm = reinterpret_cast<float *>(sraw);
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  // accumulators start from the front tile (as in the FP64 kernel)
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      acc[i][j] = f[(long long)(c0 + (j < 4 ? 0 : 32) + tx * 4 + (j & 3)) * ld + r0 +
                    (i < 4 ? 0 : 64) + ty * 4 + (i & 3)];
  const int nchunks = K / kUpdKC;
  constexpr int kStage = kUpdKC * (kUpdLdA + kUpdLdB);
  auto load = [&](int chunk, int stage) {
    float *As = sm + stage * kStage, *Bs = As + kUpdKC * kUpdLdA;
    for (int p = tid; p < kUpdKC * 32; p += 128) {  // 16 B = 4 floats
      const int q = p >> 5, m = (p & 31) * 4;
      cp_async16(As + q * kUpdLdA + m, Ag + ((long long)chunk * kUpdKC + q) * ld + m);
    }
    for (int p = tid; p < kUpdKC * 16; p += 128) {
      const int q = p >> 4, n = (p & 15) * 4;
      cp_async16(Bs + q * kUpdLdB + n, Bg + ((long long)chunk * kUpdKC + q) * ld + n);
    }
  };
#pragma unroll
  for (int st = 0; st < kUpdStages - 1; ++st) {
    if (st < nchunks) load(st, st);
    cp_async_commit();
  }
  for (int c = 0; c < nchunks; ++c) {
    cp_async_wait<kUpdStages - 2>();
    __syncthreads();
    const int nx = c + kUpdStages - 1;
    if (nx < nchunks) load(nx, nx % kUpdStages);
    cp_async_commit();
    const float *As = sm + (c % kUpdStages) * kStage;
    const float *Bs = As + kUpdKC * kUpdLdA;
#pragma unroll
    for (int q = 0; q < kUpdKC; ++q) {
      const float4 a0 = *reinterpret_cast<const float4 *>(As + q * kUpdLdA + ty * 4);
      const float4 a1 = *reinterpret_cast<const float4 *>(As + q * kUpdLdA + 64 + ty * 4);
      const float4 b0 = *reinterpret_cast<const float4 *>(Bs + q * kUpdLdB + tx * 4);
      const float4 b1 = *reinterpret_cast<const float4 *>(Bs + q * kUpdLdB + 32 + tx * 4);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(-a[i], b[j], acc[i][j]);
    }
  }
  cp_async_wait<0>();
  const bool diag = r0 < c0 + 64;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = (i < 4 ? 0 : 64) + ty * 4 + (i & 3);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = (j < 4 ? 0 : 32) + tx * 4 + (j & 3);
      if (!diag || r0 + m >= c0 + n) f[(long long)(c0 + n) * ld + r0 + m] = acc[i][j];
    }
  }
}

// ------------------------------------------------------------------ solves
// vector index of plan entry g (global vector index)
__device__ __forceinline__ int vix(const SnDev &d, int g) { return g - d.vbase; }

// small fronts, one warp each: forward substitution
template <typename T>
__global__ void __launch_bounds__(256) k_sn_fwd_small(SnDev d, int base, int count) {
  __shared__ double vs[8][kSnSmallMax];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ti = blockIdx.x * 8 + w;
  if (ti >= count) return;
  const int s = d.tasks[base + ti].x;
  if (!d.srun[d.inst[s]]) return;
  const int ld = d.ld[s], nc = d.ncol[s];
  double *v = vs[w];
  double *y = d.y;
  for (int i = lane; i < ld; i += 32) v[i] = i < nc ? y[vix(d, d.col0g[s] + i)] : 0.0;
  __syncwarp();
  for (int a = d.ch_ptr[s]; a < d.ch_ptr[s + 1]; ++a) {
    const int c = d.ch[a], cn = d.nrow[c];
    const int *rel = d.rel + d.rel_off[c];
    const double *u = d.U + d.uoff[c];
    for (int q = lane; q < cn; q += 32) v[rel[q]] += u[q];
    __syncwarp();
  }
  const T *f = reinterpret_cast<const T *>(d.F) + d.foff[s];
  // lane holds rows lane + 32 r (ld <= 128); column j + 1 is loaded while
  // column j is applied, so the dependent chain waits on shared memory only
  double cur[4], nxt[4];
  auto column = [&](int j, double (&o)[4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = lane + 32 * r;
      o[r] = (j < nc && i > j && i < ld) ? double(f[j * ld + i]) : 0.0;
    }
  };
  column(0, cur);
  for (int j = 0; j < nc; ++j) {
    column(j + 1, nxt);
    const double vj = v[j];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = lane + 32 * r;
      if (i > j && i < ld) v[i] -= cur[r] * vj;
      cur[r] = nxt[r];
    }
    __syncwarp();
  }
  for (int i = lane; i < nc; i += 32) y[vix(d, d.col0g[s] + i)] = v[i];
  double *uo = d.U + d.uoff[s];
  for (int q = lane; q < ld - nc; q += 32) uo[q] = v[nc + q];
}

// small fronts, one warp each: backward substitution
template <typename T>
__global__ void __launch_bounds__(256) k_sn_bwd_small(SnDev d, int base, int count) {
  __shared__ double vs[8][kSnSmallMax];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ti = blockIdx.x * 8 + w;
  if (ti >= count) return;
  const int s = d.tasks[base + ti].x;
  if (!d.srun[d.inst[s]]) return;
  const int ld = d.ld[s], nc = d.ncol[s];
  const int *fi = d.fidx + d.fix_off[s];
  double *v = vs[w];
  double *y = d.y;
  for (int i = lane; i < ld; i += 32) v[i] = y[vix(d, fi[i])];
  __syncwarp();
  const T *f = reinterpret_cast<const T *>(d.F) + d.foff[s];
  // column j - 1 is loaded while column j's dot product runs
  double cur[4], nxt[4];
  auto column = [&](int j, double (&o)[4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = lane + 32 * r;
      o[r] = (j >= 0 && i > j && i < ld) ? double(f[j * ld + i]) : 0.0;
    }
  };
  column(nc - 1, cur);
  for (int j = nc - 1; j >= 0; --j) {
    column(j - 1, nxt);
    double t = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = lane + 32 * r;
      if (i > j && i < ld) t += cur[r] * v[i];
      cur[r] = nxt[r];
    }
    t = warp_sum(t);
    if (lane == 0) v[j] -= t;
    __syncwarp();
  }
  for (int i = lane; i < nc; i += 32) y[vix(d, d.col0g[s] + i)] = v[i];
}

// Blocked fronts: one block per row tile (forward) or panel (backward), all
// fronts of a level in one launch.  Rows and panels share one partition (tile
// 0 has u0 mod kSnNB rows when that is nonzero, every other tile kSnNB).
//   forward   tile t sums its rows from y and the children's vectors, subtracts
//             L(t, j) x_j for the panels j < t as they are published, solves
//             its own triangle (pivot tiles) and publishes x_t;
//   backward  panel t subtracts L(i, t)^T x_i for the tiles i > t (the update
//             rows first, then the panels from the last down), solves, publishes.
// What bounds a pass is the chain over a front's panels, so everything that does
// not depend on the chain is done ahead of it: L streams through a ring of
// chunks (32 columns forward, 32 rows backward; cp.async) and the diagonal block
// is staged while the block waits.  A link of the chain is then the 128 steps of
// one warp with x in registers; 32 values are handed on as soon as they are
// final.  A value is its own flag: the published vectors hold kSubEmpty until a
// value is written, so it travels in one store and one polled load; each
// direction empties the other's vector.  (Two launches per panel and direction,
// each staging its block after the launch: 24 us a panel.  A pass over 2 000
// second-order cones' 22 panels in 7 levels: 1.5 ms before, 0.33 ms now.)
// Every sum is in an order that does not depend on the split: the children in
// order; per panel four interleaved column sums forward; per tile and column a
// balanced tree over the rows, and four interleaved sums over the tiles in
// ascending order, backward.
// The update rows' part of a backward panel needs nothing from the front's other
// panels; above kSubOwn tiles it is given to blocks of its own, a few tiles each,
// which publish their tile sums (one block streamed 16 tiles in 38 us: a level's
// backward launch 51 us on average, 26 now).
// Tasks are taken in list order (a ticket per launch), a task waits only for
// earlier ones, so the waits end whatever is resident; a bounded wait that runs
// out makes the solution NaN, which the caller reports as a failed solve.
constexpr int kSubThreads = 256;
constexpr int kSubCols = 32;   // columns (rows) of a chunk, columns of a block column
constexpr int kSubRing = 3;
constexpr int kSubSpin = 1 << 21;  // polls, about a second
constexpr int kSubNear = 36;  // tile sums of a backward panel kept on chip
constexpr int kSubB = kSnNB / kSubCols;  // block columns of a diagonal block
template <typename T>
struct Sub {
  static constexpr int pad = 16 / (int)sizeof(T);  // columns stay 16-byte aligned
  static constexpr int ldc = kSnNB + pad;          // a chunk's columns forward
  static constexpr int ldr = kSubCols + pad;       // and backward: no bank conflicts
  static constexpr int stage = kSnNB * ldr;        // the larger of the two chunks
  static_assert(stage >= kSubCols * ldc, "a stage holds either chunk");
  static constexpr int ldb(int b) { return kSnNB - kSubCols * b + pad; }
  // block column b of the diagonal block: rows 32 b .. 127
  static constexpr int boff(int b) {
    return kSubCols * (b * (kSnNB + pad) - kSubCols * (b * (b - 1) / 2));
  }
  static constexpr int ring = kSubRing * stage, l11 = boff(kSubB);
  static constexpr int aux = kSubNear * kSnNB;  // gathered values and column sums; tile sums
  static constexpr size_t bytes =
      (ring + l11) * sizeof(T) + (aux + kSnNB + 2 * kSubCols + 2 * kSnNB) * sizeof(double);
};
// one value of a published vector; a NaN when the wait runs out, and at once
// for the rest of a block that has given up
constexpr unsigned long long kSubEmpty = 0xfff8dead00000001ull;
__device__ __forceinline__ double sub_wait(const double *p, bool &lost) {
  unsigned long long v = kSubEmpty;
  for (int it = lost ? kSubSpin : 0; v == kSubEmpty && it < kSubSpin; ++it)
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  lost = v == kSubEmpty;
  return lost ? CUDART_NAN : __longlong_as_double((long long)v);
}
__device__ __forceinline__ void sub_publish(double *p, double x) {
  unsigned long long v = (unsigned long long)__double_as_longlong(x);
  if (v == kSubEmpty) v = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}
struct SubTiles {  // the partition of a front
  int first, np;   // rows of tile 0 (0: none shorter), panels
  __device__ SubTiles(int u0) : first(u0 % kSnNB), np((u0 + kSnNB - 1) / kSnNB) {}
  __device__ int start(int t) const { return first ? (t ? first + (t - 1) * kSnNB : 0) : t * kSnNB; }
  __device__ int rows(int t) const { return first && t == 0 ? first : kSnNB; }
};
// columns [col, col + w), rows r0 .. r0 + 127 into a ring stage (forward)
template <typename T>
__device__ __forceinline__ void sub_copy(T *dst, const T *f, long long ld, int r0, int col, int w) {
  constexpr int E = 16 / (int)sizeof(T), per = kSnNB / E;
#pragma unroll
  for (int it = 0; it < kSubCols * per / kSubThreads; ++it) {
    const int e = threadIdx.x + it * kSubThreads, c = e / per, r = (e % per) * E;
    if (c < w) cp_async16(dst + c * Sub<T>::ldc + r, f + (long long)(col + c) * ld + r0 + r);
  }
}
// rows r0 .. r0 + 31, columns [col, col + w) (backward)
template <typename T>
__device__ __forceinline__ void sub_copy_rows(T *dst, const T *f, long long ld, int r0, int col,
                                              int w) {
  constexpr int E = 16 / (int)sizeof(T), per = kSubCols / E;
#pragma unroll
  for (int it = 0; it < kSnNB * per / kSubThreads; ++it) {
    const int e = threadIdx.x + it * kSubThreads, c = e / per, r = (e % per) * E;
    if (c < w) cp_async16(dst + c * Sub<T>::ldr + r, f + (long long)(col + c) * ld + r0 + r);
  }
}
// the block columns of the diagonal block at (k0, k0), h rows; zeros beyond h
template <typename T>
__device__ __forceinline__ void sub_copy_diag(T *L, const T *f, long long ld, int k0, int h) {
  constexpr int E = 16 / (int)sizeof(T), per = kSnNB / E;
  for (int e = threadIdx.x; e < kSnNB * per; e += kSubThreads) {
    const int c = e / per, r = (e % per) * E, b = c / kSubCols;
    if (r + E <= b * kSubCols) continue;
    T *dst = L + Sub<T>::boff(b) + (c - b * kSubCols) * Sub<T>::ldb(b) + r - b * kSubCols;
    if (c < h && r < h) {  // h is a multiple of 16
      cp_async16(dst, f + (long long)(k0 + c) * ld + k0 + r);
    } else {
#pragma unroll
      for (int k = 0; k < E; ++k) dst[k] = T(0);
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(kSubThreads) k_sn_fwd_front(SnDev d, int base) {
  extern __shared__ __align__(16) unsigned char sraw[];
  T *ring = reinterpret_cast<T *>(sraw), *L = ring + Sub<T>::ring;
  double *aux = reinterpret_cast<double *>(L + Sub<T>::l11);
  double *vs = aux + Sub<T>::aux, *xs = vs + kSnNB;
  __shared__ unsigned ticket;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) ticket = atomicAdd(d.tickets + d.tasks[base].z, 1u);
  __syncthreads();
  const int4 tk = d.tasks[base + ticket];
  const int s = tk.x, t = tk.y;
  if (!d.srun[d.inst[s]]) return;
  const SubTiles P(d.u0[s]);
  const int np = P.np, r0 = P.start(t), h = P.rows(t), nc = d.ncol[s];
  const long long ld = d.ld[s];
  const T *f = reinterpret_cast<const T *>(d.F) + d.foff[s];
  double *v = d.S + d.soff[s];  // published here; then the backward vector
  const bool pivot = t < np;
  // chunks: panel 0 has n0 of them, the others kSubB
  const int k0 = P.rows(0), n0 = (k0 + kSubCols - 1) / kSubCols, last = min(t, np);
  const int G = last > 0 ? n0 + (last - 1) * kSubB : 0;
  auto issue = [&](int g) {
    if (g < G) {
      const int col = g < n0 ? kSubCols * g : k0 + kSubCols * (g - n0);
      sub_copy(ring + (g % kSubRing) * Sub<T>::stage, f, ld, r0, col,
               g < n0 ? min(kSubCols, k0 - col) : kSubCols);
    }
    cp_async_commit();
  };
  if (pivot) sub_copy_diag(L, f, ld, r0, h);
  cp_async_commit();
  issue(0);
  issue(1);
  if (pivot && tid < h)
    reinterpret_cast<unsigned long long *>(v)[d.u0[s] + r0 + tid] = kSubEmpty;
  if (pivot) {  // and the helpers' tile sums
    const int nu = (int)(ld - d.u0[s]) / kSnNB;
    unsigned long long *q = reinterpret_cast<unsigned long long *>(v) + 2LL * d.u0[s] +
                            ((long long)t * (np + nu) + np - t - 1) * kSnNB;
    for (int e = tid; nu > kSubOwn && e < nu * kSnNB; e += kSubThreads) q[e] = kSubEmpty;
  }
  // own rows: y plus the children's contributions in child order; the tile's
  // lists are one run, gathered by all threads and summed by a thread per row
  {
    const int *gp = d.gptr + d.gath0[s] + r0;
    const int first = gp[0], end = gp[h], rb = tid < h ? gp[tid] : 0, re = tid < h ? gp[tid + 1] : 0;
    double a = tid < h && r0 + tid < nc ? d.y[vix(d, d.col0g[s] + r0 + tid)] : 0.0;
    for (int w = first; w < end; w += Sub<T>::aux) {
      const int we = min(end, w + Sub<T>::aux);
#pragma unroll 8
      for (int q = w + tid; q < we; q += kSubThreads) aux[q - w] = d.U[d.gidx[q]];
      __syncthreads();
      for (int q = max(rb, w); q < min(re, we); ++q) a += aux[q - w];
      __syncthreads();
    }
    if (tid < kSnNB) vs[tid] = a;
  }
  // rows 2 rp, 2 rp + 1, columns q4, q4 + 4, ... of a panel; its four sums are
  // added when the next chunk's barrier has passed
  auto subtract = [&](int j) {
    const double *q = aux + (j & 1) * 4 * kSnNB + tid;
    if (tid < kSnNB) vs[tid] -= (q[0] + q[kSnNB]) + (q[2 * kSnNB] + q[3 * kSnNB]);
  };
  const int rp = tid & 63, q4 = tid >> 6;
  double a0 = 0, a1 = 0;
  bool lost = false;
  for (int g = 0; g < G; ++g) {
    const int col = g < n0 ? kSubCols * g : k0 + kSubCols * (g - n0);
    const int w = g < n0 ? min(kSubCols, k0 - col) : kSubCols;
    double *x = xs + (g & 1) * kSubCols;  // the other half may still be read
    if (warp == 0 && lane < w) x[lane] = sub_wait(v + col + lane, lost);
    cp_async_wait<1>();
    __syncthreads();
    issue(g + 2);  // into the stage of chunk g - 1, which everyone has left
    if (g >= n0 && (g - n0) % kSubB == 0) subtract((g - n0) / kSubB);
    const T *A = ring + (g % kSubRing) * Sub<T>::stage + 2 * rp;
#pragma unroll
    for (int q = 0; q < kSubCols / 4; ++q) {
      const int c = q4 + 4 * q;
      if (c < w) {
        const Pair<T> l = load_pair(A + c * Sub<T>::ldc);
        a0 += double(l.x) * x[c];
        a1 += double(l.y) * x[c];
      }
    }
    if (g == n0 - 1 || (g >= n0 && (g - n0) % kSubB == kSubB - 1)) {  // panel j is done
      const int j = g < n0 ? 0 : 1 + (g - n0) / kSubB;
      double *q = aux + ((j & 1) * 4 + q4) * kSnNB + 2 * rp;
      q[0] = a0;
      q[1] = a1;
      a0 = a1 = 0;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (last > 0) subtract(last - 1);
  if (!pivot) {
    const int q = r0 - d.u0[s] + tid;
    if (tid < kSnNB && q < d.nrow[s]) d.U[d.uoff[s] + q] = vs[tid];
    return;
  }
  // one warp: lane owns rows lane + 32 r; x_j is final when step j starts and is
  // broadcast from its owner
  __syncthreads();
  if (warp != 0) return;
  double xr[kSubB];
#pragma unroll
  for (int r = 0; r < kSubB; ++r) xr[r] = vs[lane + kSubCols * r];
#pragma unroll
  for (int b = 0; b < kSubB; ++b) {
    if (kSubCols * b >= h) break;
    const T *Lb = L + Sub<T>::boff(b) - kSubCols * b + lane;
#pragma unroll
    for (int jj = 0; jj < kSubCols; ++jj) {
      const double xj = __shfl_sync(0xffffffffu, xr[b], jj);
#pragma unroll
      for (int r = b; r < kSubB; ++r)
        if (r > b || lane > jj) xr[r] -= double(Lb[jj * Sub<T>::ldb(b) + kSubCols * r]) * xj;
    }
    const int r = kSubCols * b + lane;
    if (r < h) {
      sub_publish(v + r0 + r, xr[b]);
      if (r0 + r < nc) d.y[vix(d, d.col0g[s] + r0 + r)] = xr[b];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kSubThreads) k_sn_bwd_front(SnDev d, int base) {
  extern __shared__ __align__(16) unsigned char sraw[];
  T *ring = reinterpret_cast<T *>(sraw), *L = ring + Sub<T>::ring;
  double *aux = reinterpret_cast<double *>(L + Sub<T>::l11);
  double *vs = aux + Sub<T>::aux, *xs = vs + kSnNB, *red = xs + 2 * kSubCols;
  __shared__ unsigned ticket;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) ticket = atomicAdd(d.tickets + d.tasks[base].z, 1u);
  __syncthreads();
  const int4 tk = d.tasks[base + ticket];
  const int s = tk.x, t = tk.y;
  if (!d.srun[d.inst[s]]) return;
  const SubTiles P(d.u0[s]);
  const int np = P.np, k0 = P.start(t), K = P.rows(t), u0 = d.u0[s];
  const long long ld = d.ld[s];
  const int nt = np + (int)(ld - u0) / kSnNB;
  const int *fi = d.fidx + d.fix_off[s];
  const T *f = reinterpret_cast<const T *>(d.F) + d.foff[s];
  double *v = d.S + d.soff[s] + u0;  // published here; the forward vector is before it
  // tiles [i0, i1) of the update rows first, then (unless the task is only these)
  // the panels from the last down
  const bool helped = nt - np > kSubOwn, helper = tk.w != 0;
  const int i0 = helper ? tk.w & 0xffff : np, i1 = helper ? tk.w >> 16 : helped ? np : nt;
  auto tile = [&](int m) { return m < i1 - i0 ? i0 + m : np - 1 - (m - (i1 - i0)); };
  constexpr int nr = kSnNB / kSubCols;  // chunks of a tile, taken from its last rows up
  const int M = i1 - i0 + (helper ? 0 : np - 1 - t), G = M * nr;
  auto row = [&](int g) { return P.start(tile(g / nr)) + kSubCols * (nr - 1 - g % nr); };
  auto issue = [&](int g) {
    if (g < G) sub_copy_rows(ring + (g % kSubRing) * Sub<T>::stage, f, ld, row(g), k0, K);
    cp_async_commit();
  };
  if (!helper) sub_copy_diag(L, f, ld, k0, K);
  cp_async_commit();
  issue(0);
  issue(1);
  if (tid < kSnNB && !helper) {
    const int g = tid < K ? fi[k0 + tid] : -1;
    vs[tid] = g >= 0 ? d.y[vix(d, g)] : 0.0;
    if (tid < K) reinterpret_cast<unsigned long long *>(v)[k0 + tid - u0] = kSubEmpty;
  }
  // Column cl; of each chunk's 16 row pairs the even ones (odd = 0) or the odd
  // ones.  Per tile and column the sum is a tree: row pairs 16 apart (chunks 3
  // and 2, 1 and 0), then 8, 4 and 2 apart in the thread, 1 apart across the two
  // threads, then the tile's two halves.
  const int cl = tid & (kSnNB - 1), odd = tid / kSnNB;
  double pr[8], hi = 0, lo = 0;
  // tile sums: the nearest tiles in shared memory, others in the workspace
  double *far = d.S + d.soff[s] + 2LL * u0 + (long long)t * nt * kSnNB + cl;
  auto slot = [&](int i) -> double & {
    const int k = i - t - 1;
    return k < kSubNear ? aux[k * kSnNB + cl] : far[(long long)k * kSnNB];
  };
  auto finish = [&](int i) {
    const double p = (lo + red[cl]) + (hi + red[kSnNB + cl]);
    if (odd) return;
    if (helper)
      sub_publish(far + (long long)(i - t - 1) * kSnNB, p);
    else
      slot(i) = p;
  };
  double ahead = 0;
  bool lost = false;
  int pos = -1;
  if (warp == 0) {
    const int p = G > 0 && row(0) >= u0 ? fi[row(0) + lane] : -1;
    pos = G > 1 && row(1) >= u0 ? fi[row(1) + lane] : -1;
    ahead = p >= 0 ? d.y[vix(d, p)] : 0.0;
  }
  if (helped && !helper) {  // the helpers' sums, while the chain gets here
    for (int b = np + odd; b < nt; b += 16) {
      double p[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        p[k] = b + 2 * k < nt ? __ldcg(far + (long long)(b + 2 * k - t - 1) * kSnNB) : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int i = b + 2 * k;
        if (i < nt) {
          if (__double_as_longlong(p[k]) == (long long)kSubEmpty)
            p[k] = sub_wait(far + (long long)(i - t - 1) * kSnNB, lost);
          if (i - t - 1 < kSubNear) aux[(i - t - 1) * kSnNB + cl] = p[k];
        }
      }
    }
  }
  for (int g = 0; g < G; ++g) {
    const int r = row(g);
    double *x = xs + (g & 1) * kSubCols;  // the other half may still be read
    if (warp == 0) x[lane] = r >= u0 ? ahead : sub_wait(v + r + lane, lost);
    cp_async_wait<1>();
    __syncthreads();
    issue(g + 2);  // into the stage of chunk g - 1, which everyone has left
    if (warp == 0) {  // the next chunk's values and the positions of the one after
      ahead = g + 1 < G && row(g + 1) >= u0 && pos >= 0 ? d.y[vix(d, pos)] : 0.0;
      pos = g + 2 < G && row(g + 2) >= u0 ? fi[row(g + 2) + lane] : -1;
    }
    const int c = nr - 1 - g % nr;  // chunk of the tile
    if (c == nr - 1 && g > 0) finish(tile(g / nr - 1));
    const T *A = ring + (g % kSubRing) * Sub<T>::stage + cl * Sub<T>::ldr + 2 * odd;
    const double *xo = x + 2 * odd;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const Pair<T> l = load_pair(A + 4 * q);
      const double p = double(l.x) * xo[4 * q] + double(l.y) * xo[4 * q + 1];
      pr[q] = (c & 1) ? p : p + pr[q];
    }
    if (!(c & 1)) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < o; ++q) pr[q] += pr[q + o];
      if (c) hi = pr[0];
      else lo = pr[0];
      if (odd && c == 0) {
        red[cl] = lo;
        red[kSnNB + cl] = hi;
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (G > 0) finish(tile(M - 1));
  if (helper) return;
  __syncthreads();
  // four interleaved sums over the tiles in ascending order, two per thread
  {
    double a[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll 4
      for (int i = t + 1 + 2 * odd + u; i < nt; i += 4)
        a[u] += i - t - 1 < kSubNear ? slot(i) : __ldcg(&slot(i));
    __syncthreads();
    if (odd) {
      red[cl] = a[0];
      red[kSnNB + cl] = a[1];
    }
    __syncthreads();
    if (!odd) vs[cl] = cl < K ? vs[cl] - ((((0.0 + a[0]) + a[1]) + red[cl]) + red[kSnNB + cl]) : 0.0;
    __syncthreads();
  }
  // one warp: lane owns x_j, j = lane + 32 r; x_i is final when step i (descending)
  // starts, is broadcast from its owner, and L(i, j) x_i leaves every x_j, j < i
  if (warp != 0) return;
  double xr[kSubB];
#pragma unroll
  for (int r = 0; r < kSubB; ++r) xr[r] = vs[lane + kSubCols * r];
#pragma unroll
  for (int b = kSubB - 1; b >= 0; --b) {
    if (kSubCols * b >= K) continue;
#pragma unroll
    for (int ii = kSubCols - 1; ii >= 0; --ii) {
      const double xi = __shfl_sync(0xffffffffu, xr[b], ii);
#pragma unroll
      for (int r = 0; r <= b; ++r)
        if (r < b || lane < ii)
          xr[r] -= double(L[Sub<T>::boff(r) + lane * Sub<T>::ldb(r) + kSubCols * (b - r) + ii]) * xi;
    }
    const int j = kSubCols * b + lane;
    if (j < K) {
      sub_publish(v + k0 + j, xr[b]);
      const int g = fi[k0 + j];
      if (g >= 0) d.y[vix(d, g)] = xr[b];
    }
  }
}

// y <- D^-1 y over the plan's running instances; the substitution launches'
// tickets are given back on the way
__global__ void k_sn_dscale(SnDev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = i; k < d.ntickets; k += gridDim.x * blockDim.x) d.tickets[k] = 0;
  if (i >= d.vcount) return;
  const int inst = d.vinst[i];
  if (inst < 0 || !d.srun[inst]) return;
  d.y[i] *= d.Dinv[d.vbase + i];
}

// ------------------------------------------------------------- refinement
__device__ __forceinline__ void nrm_max(unsigned long long *a, double v) {
  if (!(v >= 0.0)) v = CUDART_INF;  // NaN counts as infinite
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// b, y from the right-hand side (rx by x index, rz by z row; gsrc codes);
// |b|_inf; zeroes |e|_inf
__global__ void k_sn_rhs(SnDev d, KKTDev k, const double *rx, const double *rz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.vcount) return;
  const int inst = d.vinst[i];
  if (inst < 0 || !d.srun[inst]) return;
  const int g = k.gsrc[d.vbase + i];
  const double v = g >= 0 ? rx[g] : (g == -1 ? 0.0 : rz[-g - 2]);
  d.b[i] = v;
  d.y[i] = v;
  nrm_max(d.nrm + 2 * inst, fabs(v));
}

// e = b - K xs, |e|_inf (K with its true diagonal)
__global__ void k_sn_resid(SnDev d, KKTDev k, const double *xs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.vcount) return;
  const int inst = d.vinst[i];
  if (inst < 0 || !d.srun[inst]) return;
  const int vb = k.voff[inst], r = d.vbase + i - vb;
  const int *kp = k.Kp + k.poff[inst];
  double t = 0;
  for (int p = kp[r]; p < kp[r + 1]; ++p) t += k.Kx[p] * xs[vb + k.Kj[p] - d.vbase];
  const double e = d.b[i] - t;
  d.e[i] = e;
  nrm_max(d.nrm + 2 * inst + 1, fabs(e));
}

__global__ void k_sn_zero_nrm(SnDev d, int which, int B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B && d.srun[i]) d.nrm[2 * i + which] = 0ull;
}

// mode 0: x = y; 1: y = e; 2: xn = x + y; 3: x = xn
__global__ void k_sn_vec(SnDev d, int mode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.vcount) return;
  const int inst = d.vinst[i];
  if (inst < 0 || !d.srun[inst]) return;
  switch (mode) {
    case 0: d.x[i] = d.y[i]; break;
    case 1: d.y[i] = d.e[i]; break;
    case 2: d.xn[i] = d.x[i] + d.y[i]; break;
    default: d.x[i] = d.xn[i]; break;
  }
}

// solution scatter (permuted -> x index / z row)
__global__ void k_sn_out(SnDev d, KKTDev k, double *lx, double *lz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.vcount) return;
  const int inst = d.vinst[i];
  if (inst < 0 || !d.srun[inst]) return;
  const int g = k.gsrc[d.vbase + i];
  if (g >= 0) {
    if (lx) lx[g] = d.x[i];
  } else if (g <= -2) {
    if (lz) lz[-g - 2] = d.x[i];
  }
}

__global__ void k_sn_flags(const int *insts, int n, const int *run, const int *ok, int *flags) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < n) flags[a] = (run[insts[a]] && ok[insts[a]]) ? 1 : 0;
}

__global__ void k_sn_clear_ok(const int *insts, const int *bad, int n, int *ok) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < n && bad[a]) ok[insts[a]] = 0;
}

inline int nb256(long long n) { return n <= 0 ? 1 : (int)((n + 255) / 256); }

template <typename T>
size_t diag_smem() {  // the block and the scaled columns of one column block
  return (size_t)kSnNB * kSnNB * sizeof(T) + (size_t)kDiagNB * kSnNB * sizeof(T);
}
template <typename T>
size_t trsm_smem() {  // the tile (kSnNB x kSnNB) and the packed strict lower L11
  return (size_t)kSnNB * kSnNB * sizeof(T) + (size_t)kSnNB * kSnNB / 2 * sizeof(T);
}
template <typename T>
size_t gemm_smem() {
  return (size_t)kUpdStages * kUpdKC * (kUpdLdA + kUpdLdB) * sizeof(T);
}

template <typename T>
void set_sn_attrs() {
  static bool done = false;
  if (done) return;
  cudaFuncSetAttribute(k_sn_diag<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)diag_smem<T>());
  cudaFuncSetAttribute(k_sn_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)((kSnSmallMax * kSnSmallMax + kSnSmallMax) * sizeof(T)));
  cudaFuncSetAttribute(k_sn_trsm<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_smem<T>());
  cudaFuncSetAttribute(k_sn_fwd_front<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Sub<T>::bytes);
  cudaFuncSetAttribute(k_sn_bwd_front<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Sub<T>::bytes);
  if (sizeof(T) == 8)
    cudaFuncSetAttribute(k_sn_update_f64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)gemm_smem<double>());
  else
    cudaFuncSetAttribute(k_sn_update_f32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)gemm_smem<float>());
  done = true;
}

// profiling: an event pair around one launch
void prof_begin(SnExec &ex, const SnLaunch &L, cudaStream_t st) {
  if (!ex.prof.on) return;
  auto &P = ex.prof;
  const size_t k = P.kinds.size();
  while (P.pool.size() < 2 * k + 2) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) {
      P.on = false;
      return;
    }
    P.pool.push_back(e);
  }
  P.kinds.push_back(L.kind);
  P.flops[L.kind] += L.flops;
  P.calls[L.kind]++;
  cudaEventRecord(P.pool[2 * k], st);
}
void prof_end(SnExec &ex, cudaStream_t st) {
  if (!ex.prof.on || ex.prof.kinds.empty()) return;
  cudaEventRecord(ex.prof.pool[2 * ex.prof.kinds.size() - 1], st);
}
// sum the recorded pairs (waits for the last one)
void prof_collect(SnExec &ex) {
  auto &P = ex.prof;
  if (!P.on || P.kinds.empty()) return;
  cudaEventSynchronize(P.pool[2 * P.kinds.size() - 1]);
  for (size_t k = 0; k < P.kinds.size(); ++k) {
    float t = 0.f;
    if (cudaEventElapsedTime(&t, P.pool[2 * k], P.pool[2 * k + 1]) == cudaSuccess)
      P.ms[P.kinds[k]] += t;
  }
  P.kinds.clear();
}

template <typename T>
void run_factor(SnExec &ex, const KKTDev &k, const LDLParams &p, const int *run, int *ok,
                cudaStream_t st) {
  set_sn_attrs<T>();
  const SnDev &d = ex.d;
  for (const SnLaunch &L : ex.fact) {
    prof_begin(ex, L, st);
    switch (L.kind) {
      case SN_SMALL_FACTOR:
        k_sn_small<T><<<L.count, kSmallThreads, (L.smem + kSnSmallMax) * sizeof(T), st>>>(
            d, k, p, L.begin, run, ok);
        break;
      case SN_ASSEMBLE:
        k_sn_assemble<T><<<L.count, kAsmThreads, 0, st>>>(d, k, L.begin, run);
        break;
      case SN_DIAG:
        k_sn_diag<T><<<L.count, kDiagThreads, diag_smem<T>(), st>>>(d, k, p, L.begin, run, ok);
        break;
      case SN_TRSM:
        k_sn_trsm<T><<<L.count, kTrsmThreads, trsm_smem<T>(), st>>>(d, L.begin, run);
        break;
      case SN_UPDATE:
        if (sizeof(T) == 8)
          k_sn_update_f64<<<L.count, kUpdThreads, gemm_smem<double>(), st>>>(d, L.begin, run);
        else
          k_sn_update_f32<<<L.count, 128, gemm_smem<float>(), st>>>(d, L.begin, run);
        break;
      default:
        break;
    }
    prof_end(ex, st);
    ex.launches++;
  }
  prof_collect(ex);
}

// one pass y <- K^-1 y for the instances with srun set
template <typename T>
void run_solve_pass(SnExec &ex, cudaStream_t st) {
  set_sn_attrs<T>();
  const SnDev &d = ex.d;
  for (const SnLaunch &L : ex.fwd) {
    prof_begin(ex, L, st);
    switch (L.kind) {
      case SN_FWD_SMALL: k_sn_fwd_small<T><<<(L.count + 7) / 8, 256, 0, st>>>(d, L.begin, L.count); break;
      case SN_FWD_DIAG:
        k_sn_fwd_front<T><<<L.count, kSubThreads, Sub<T>::bytes, st>>>(d, L.begin);
        break;
      default: break;
    }
    prof_end(ex, st);
    ex.launches++;
  }
  k_sn_dscale<<<nb256(d.vcount), 256, 0, st>>>(d);
  for (const SnLaunch &L : ex.bwd) {
    prof_begin(ex, L, st);
    switch (L.kind) {
      case SN_BWD_SMALL: k_sn_bwd_small<T><<<(L.count + 7) / 8, 256, 0, st>>>(d, L.begin, L.count); break;
      case SN_BWD_DIAG:
        k_sn_bwd_front<T><<<L.count, kSubThreads, Sub<T>::bytes, st>>>(d, L.begin);
        break;
      default: break;
    }
    prof_end(ex, st);
    ex.launches++;
  }
  ex.launches++;
  prof_collect(ex);
}

// one pass, replayed from a CUDA graph when possible (direct launches while
// profiling or if capturing failed)
template <typename T>
void solve_pass(SnExec &ex, cudaStream_t st) {
  if (!ex.prof.on && !ex.g_pass && !ex.graph_failed) {
    set_sn_attrs<T>();
    bool ok = ex.cap || cudaStreamCreateWithFlags(&ex.cap, cudaStreamNonBlocking) == cudaSuccess;
    cudaGraph_t g = nullptr;
    const long long before = ex.launches;
    if (ok) ok = cudaStreamBeginCapture(ex.cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (ok) {
      run_solve_pass<T>(ex, ex.cap);
      ok = cudaStreamEndCapture(ex.cap, &g) == cudaSuccess && g;
    }
    if (ok) ok = cudaGraphInstantiate(&ex.g_pass, g, 0) == cudaSuccess;
    if (g) cudaGraphDestroy(g);
    ex.pass_launches = ex.launches - before;
    ex.launches = before;
    if (!ok) {
      ex.g_pass = nullptr;
      ex.graph_failed = true;
      cudaGetLastError();  // clear a capture error; the pass runs directly
    }
  }
  if (!ex.prof.on && ex.g_pass) {
    cudaGraphLaunch(ex.g_pass, st);
    ex.launches += ex.pass_launches;
  } else {
    run_solve_pass<T>(ex, st);
  }
}

}  // namespace

void sn_set_profiling(SnExec &ex, bool on) {
  ex.prof.on = on;
  ex.prof.kinds.clear();
  if (on) {
    ex.ir_solves = ex.ir_sweeps = ex.ir_unconverged = 0;
    ex.ir_worst = 0.0;
  }
  if (on)
    for (int k = 0; k < SN_KINDS; ++k) {
      ex.prof.ms[k] = ex.prof.flops[k] = 0.0;
      ex.prof.calls[k] = 0;
    }
}

void sn_get_profile(const SnExec &ex, double *ms, double *flops, long long *calls) {
  for (int k = 0; k < SN_KINDS; ++k) {
    if (ms) ms[k] = ex.prof.ms[k];
    if (flops) flops[k] = ex.prof.flops[k];
    if (calls) calls[k] = ex.prof.calls[k];
  }
}

SnExec::~SnExec() {
  if (g_pass) cudaGraphExecDestroy(g_pass);
  if (cap) cudaStreamDestroy(cap);
  for (cudaEvent_t e : prof.pool) cudaEventDestroy(e);
  if (h_srun) pinned_give(h_srun);
  if (h_flags) pinned_give(h_flags);
  if (h_nrm) pinned_give(h_nrm);
}

bool sn_exec_create(const SnPlan &P, bool fp32, int B, int vbase, int vcount,
                    const std::vector<int> &vinst, DevArena &A, SnExec &ex) {
  ex.fp32 = fp32;
  ex.B = B;
  ex.fact = P.fact;
  ex.fwd = P.fwd;
  ex.bwd = P.bwd;
  ex.insts = P.insts;
  ex.small_smem = P.small_smem_max;
  ex.flops = P.flops;
  SnDev &d = ex.d;
  d.inst = A.upload(P.inst);
  d.col0g = A.upload(P.col0g);
  d.ncol = A.upload(P.ncol);
  d.nrow = A.upload(P.nrow);
  d.u0 = A.upload(P.u0);
  d.ld = A.upload(P.ld);
  d.cbase = A.upload(P.cbase);
  d.fix_off = A.upload(P.fix_off);
  d.rel_off = A.upload(P.rel_off);
  d.ch_ptr = A.upload(P.ch_ptr);
  d.ch = A.upload(P.ch);
  d.uoff = A.upload(P.uoff);
  d.fidx = A.upload(P.fidx);
  d.rel = A.upload(P.rel);
  d.acol = A.upload(P.acol);
  d.foff = A.upload(P.foff);
  d.woff = A.upload(P.woff);
  d.soff = A.upload(P.soff);
  d.amap = reinterpret_cast<const int2 *>(A.upload(P.amap));
  d.tasks = reinterpret_cast<const int4 *>(A.upload(P.tasks));
  d.gath0 = A.upload(P.gath0);
  d.gptr = A.upload(P.gptr);
  d.gidx = A.upload(P.gidx);
  d.cl_ptr = A.upload(P.cl_ptr);
  d.clist = reinterpret_cast<const int4 *>(A.upload(P.clist));
  const size_t ts = fp32 ? 4 : 8;
  d.F = fp32 ? (void *)A.alloc<float>(P.f_elems) : (void *)A.alloc<double>(P.f_elems);
  d.W = fp32 ? (void *)A.alloc<float>(P.w_elems) : (void *)A.alloc<double>(P.w_elems);
  (void)ts;
  {  // every published vector starts empty
    const unsigned long long bits = kSubEmpty;
    double empty;
    memcpy(&empty, &bits, sizeof(empty));
    d.S = A.upload(std::vector<double>(std::max<long long>(P.s_elems, 1), empty));
  }
  d.tickets = A.upload(std::vector<unsigned>(std::max(P.ntickets, 1), 0u));
  d.ntickets = P.ntickets;
  d.U = A.alloc<double>(P.u_elems);
  d.Dinv = A.alloc<double>((size_t)vbase + vcount);
  d.eps = A.alloc<double>(B);
  d.srun = A.alloc<int>(B);
  d.nrm = A.alloc<unsigned long long>(2 * (size_t)B);
  d.b = A.alloc<double>(vcount);
  d.x = A.alloc<double>(vcount);
  d.xn = A.alloc<double>(vcount);
  d.e = A.alloc<double>(vcount);
  d.y = A.alloc<double>(vcount);
  d.vinst = A.upload(vinst);
  d.vbase = vbase;
  d.vcount = vcount;
  ex.d_insts = A.upload(P.insts);
  ex.d_flags = A.alloc<int>(B);
  if (pinned_take(&ex.h_srun, sizeof(int) * B) != cudaSuccess) return false;
  if (pinned_take(&ex.h_flags, sizeof(int) * B) != cudaSuccess) return false;
  if (pinned_take(&ex.h_nrm, sizeof(unsigned long long) * 2 * B) != cudaSuccess) return false;
  return A.err == cudaSuccess;
}

void sn_factor(SnExec &ex, const KKTDev &k, const LDLParams &p, const int *run, int *ok,
               double *eps_out, cudaStream_t st) {
  if (ex.insts.empty()) return;
  k_sn_eps<<<(int)ex.insts.size(), kAsmThreads, 0, st>>>(ex.d, k, p, ex.d_insts, run, eps_out);
  ex.launches++;
  if (ex.fp32)
    run_factor<float>(ex, k, p, run, ok, st);
  else
    run_factor<double>(ex, k, p, run, ok, st);
}

void sn_solve(SnExec &ex, const KKTDev &k, const LDLParams &p, const int *run, const double *rx,
              const double *rz, double *lx, double *lz, int *ok, cudaStream_t st) {
  const int n = (int)ex.insts.size();
  if (n == 0) return;
  SnDev &d = ex.d;
  const int B = ex.B;
  auto pass = [&]() {
    if (ex.fp32)
      solve_pass<float>(ex, st);
    else
      solve_pass<double>(ex, st);
  };
  auto upload_srun = [&](const std::vector<char> &on) {
    cudaStreamSynchronize(st);  // the previous upload has left the staging
    for (int i = 0; i < B; ++i) ex.h_srun[i] = 0;
    for (int a = 0; a < n; ++a) ex.h_srun[ex.insts[a]] = on[a] ? 1 : 0;
    cudaMemcpyAsync(d.srun, ex.h_srun, sizeof(int) * B, cudaMemcpyHostToDevice, st);
  };
  auto read_nrm = [&]() {
    cudaMemcpyAsync(ex.h_nrm, d.nrm, sizeof(unsigned long long) * 2 * B, cudaMemcpyDeviceToHost,
                    st);
    cudaStreamSynchronize(st);
  };
  auto as_double = [](unsigned long long u) {
    double v;
    memcpy(&v, &u, sizeof(v));
    return v;
  };
  // instances taking part: run and ok
  k_sn_flags<<<nb256(n), 256, 0, st>>>(ex.d_insts, n, run, ok, ex.d_flags);
  cudaMemcpyAsync(ex.h_flags, ex.d_flags, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  std::vector<char> act(n), live(n), bad(n, 0);
  bool any = false;
  for (int a = 0; a < n; ++a) {
    act[a] = ex.h_flags[a] != 0;
    any = any || act[a];
  }
  if (!any) return;
  upload_srun(act);
  k_sn_zero_nrm<<<nb256(B), 256, 0, st>>>(d, 0, B);
  k_sn_zero_nrm<<<nb256(B), 256, 0, st>>>(d, 1, B);
  k_sn_rhs<<<nb256(d.vcount), 256, 0, st>>>(d, k, rx, rz);
  pass();
  k_sn_vec<<<nb256(d.vcount), 256, 0, st>>>(d, 0);  // x = y
  k_sn_resid<<<nb256(d.vcount), 256, 0, st>>>(d, k, d.x);
  read_nrm();
  std::vector<double> normb(n), norme(n);
  for (int a = 0; a < n; ++a) {
    if (!act[a]) continue;
    const int i = ex.insts[a];
    normb[a] = as_double(ex.h_nrm[2 * i]);
    norme[a] = as_double(ex.h_nrm[2 * i + 1]);
    if (!std::isfinite(norme[a])) bad[a] = 1;  // non-finite solution
    live[a] = act[a] && !bad[a] && p.ir_enable;
  }
  // iterative refinement (kktsolver_directldl_gpu.jl:349-410): stop at the
  // tolerance, after ir_maxiter sweeps, or when a sweep improves the error
  // by less than ir_stopratio (keeping the better iterate)
  for (int it = 0; p.ir_enable && it < p.ir_maxiter; ++it) {
    std::vector<char> cont(n, 0);
    bool anyc = false;
    for (int a = 0; a < n; ++a) {
      if (!live[a]) continue;
      if (norme[a] <= p.ir_abstol + p.ir_reltol * normb[a]) {
        live[a] = 0;
        continue;
      }
      cont[a] = 1;
      anyc = true;
    }
    if (!anyc) break;
    ex.ir_sweeps++;
    upload_srun(cont);
    k_sn_vec<<<nb256(d.vcount), 256, 0, st>>>(d, 1);  // y = e
    pass();
    k_sn_vec<<<nb256(d.vcount), 256, 0, st>>>(d, 2);  // xn = x + y
    k_sn_zero_nrm<<<nb256(B), 256, 0, st>>>(d, 1, B);
    k_sn_resid<<<nb256(d.vcount), 256, 0, st>>>(d, k, d.xn);
    read_nrm();
    std::vector<char> accept(n, 0);
    bool anya = false;
    for (int a = 0; a < n; ++a) {
      if (!cont[a]) continue;
      const double ne = as_double(ex.h_nrm[2 * ex.insts[a] + 1]);
      if (!std::isfinite(ne)) {
        bad[a] = 1;
        live[a] = 0;
        continue;
      }
      const double ratio = norme[a] / ne;
      if (ratio < p.ir_stopratio) {
        live[a] = 0;
        if (ratio > 1.0) accept[a] = 1;
      } else {
        accept[a] = 1;
      }
      if (accept[a]) {
        norme[a] = ne;
        anya = true;
      }
    }
    if (anya) {
      upload_srun(accept);
      k_sn_vec<<<nb256(d.vcount), 256, 0, st>>>(d, 3);  // x = xn
    }
  }
  std::vector<char> good(n);
  for (int a = 0; a < n; ++a) good[a] = act[a] && !bad[a];
  for (int a = 0; a < n; ++a) {
    if (!act[a]) continue;
    ex.ir_solves++;
    const double tol = p.ir_abstol + p.ir_reltol * normb[a];
    if (p.ir_enable && !bad[a] && norme[a] > tol) {
      ex.ir_unconverged++;
      ex.ir_worst = std::max(ex.ir_worst, norme[a] / tol);
    }
  }
  upload_srun(good);
  k_sn_out<<<nb256(d.vcount), 256, 0, st>>>(d, k, lx, lz);
  bool anybad = false;
  for (int a = 0; a < n; ++a) {
    ex.h_flags[a] = bad[a];
    anybad = anybad || bad[a];
  }
  if (anybad) {
    cudaMemcpyAsync(ex.d_flags, ex.h_flags, sizeof(int) * n, cudaMemcpyHostToDevice, st);
    k_sn_clear_ok<<<nb256(n), 256, 0, st>>>(ex.d_insts, ex.d_flags, n, ok);
  }
  cudaStreamSynchronize(st);  // pinned staging is reused by the next call
}

}  // namespace clgpu
