// ldl_sliced.cu -- sparse LDL^T of the small instances: one block of
// kSlWarps warps per instance, dense work vectors in shared memory, every
// sparse sum laid out as slices (sliced.hpp).
//
// What bounds it: the elimination tree gives 20-40 dependent levels of a few
// dozen short sums each, so an instance alone is a chain of shared gathers,
// exchanges and barriers, and a full batch is as many of those chains as fit an
// SM (issue slots 38 % busy with four blocks resident, DRAM 25 %).  So the code
// of a page is straight-line (a lane owns one run of at most four terms, no
// segment bookkeeping in the loop), copies are off the path (a warp of its own
// in the solves, a ring per warp in the factorisation), and several warps
// share an instance's levels.  One warp per instance with a two-slot ring and
// per-entry bookkeeping before this took, on 4096 MPC instances (N up to 1222,
// one solve to 1e-8), 15.7 / 8.4 / 7.4 ms for two-side solves / one-side solves
// / factorisations; this takes 10.5 / 7.6 / 5.4 ms.  One instance of N = 1057:
// 4.7 / 2.5 / 1.2 ms before, 1.7 / 1.3 / 1.0 ms now.
//
// Sums run in the order sliced.hpp fixes (products and sums spelled __dmul_rn /
// __dadd_rn / __dsub_rn, which are never contracted), so a result does not
// depend on the batch, on the spread over warps, nor on whether one or two
// right-hand sides are solved.
#include <type_traits>

#include "ldl.cuh"
#include "sliced.hpp"

namespace clgpu {

namespace {

constexpr int kNT = 32 * kSlWarps;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ void cp16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
// The block meets, its warps at different places of the code: the copying warp and
// the adding ones in the solves, warps with different numbers of pages in the
// factorisation.  (__syncthreads is only defined where the whole block takes the
// same path; barrier.sync counts the warps that arrive.)
__device__ __forceinline__ void meet() {
  asm volatile("barrier.sync.aligned 1, %0;\n" ::"n"(kNT) : "memory");
}
__device__ __forceinline__ void meet(int n) {
#pragma unroll 1
  for (; n > 0; --n) meet();
}

// The block's stage ring in shared memory: the forward, backward and residual
// stages in a circle.  The last warp copies them with cp.async, kSlRing stages
// ahead; the others take one page of a stage each.  A level is a few hundred
// cycles, so nothing of the copying may be on its path: with each warp copying
// its own pages (a ring of two per warp) the batch's two-side solves took 11.4
// ms, so 10.5.  A deeper ring costs a resident block per SM (14.6 ms with four
// slots).  A thread reads its next stage's words and values before it meets the
// others.
template <typename T>
struct Ring {
  static constexpr int kVals = kSlStage * kSlRun * 8, kSlot = kVals + kSlStage * 16;
  unsigned char *mem;
  const uint8_t *table;  // shared memory: stored lanes of each stage
  int n, nl;             // stages in the circle, of them factor
  // copying warp: next stage, its slot, and where its data lies (this lane's)
  const unsigned char *words0, *vals0, *kvals0, *words, *vals, *kvals;
  int at, in;
  // the others: the stage after the one in registers and its slot
  int cur, out;
  double v[kSlRun];
  uint4 e;
  bool busy, used;       // the warp has a page; the lane is one of its

  __device__ __forceinline__ void issue(int lane) {
    const int nu = table[at];
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(mem)) + in * kSlot;
    const bool fac = at < nl;
    const unsigned char *v = fac ? vals : kvals;
    const int halves = fac ? kSlRun * (int)sizeof(T) / 16 : kSlRun / 2;
#pragma unroll
    for (int h = 0; h < kSlStagePages; ++h) {
      const int l = lane + 32 * h;
      if (l < nu) {
        cp16(s + 16 * l, v + 512 * h);
        if (halves == 2) cp16(s + 16 * (kSlStage + l), v + 512 * h + 16 * nu);
        cp16(s + kVals + 16 * l, words + 512 * h);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    words += 16 * nu;
    (fac ? vals : kvals) += 16 * halves * nu;
    if (++at == n) {
      at = 0;
      words = words0;
      vals = vals0;
      kvals = kvals0;
    }
    in = in + 1 == kSlRing ? 0 : in + 1;
  }
  // stages up to the one after the next are in shared memory
  __device__ __forceinline__ void landed() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kSlRing - 2) : "memory");
  }
  __device__ __forceinline__ void take(int tid) {
    const int nu = table[cur];
    busy = (tid & ~31) < nu;
    used = tid < nu;
    if (busy) {
      const int l = min(tid, nu - 1);  // (idle lanes add up unused sums)
      const unsigned char *s = mem + out * kSlot + 16 * l;
      if (sizeof(T) == 8 || cur >= nl) {
        const double2 a = *reinterpret_cast<const double2 *>(s);
        const double2 b = *reinterpret_cast<const double2 *>(s + 16 * kSlStage);
        v[0] = a.x;
        v[1] = a.y;
        v[2] = b.x;
        v[3] = b.y;
      } else {
        const float4 a = *reinterpret_cast<const float4 *>(s);
        v[0] = a.x;
        v[1] = a.y;
        v[2] = a.z;
        v[3] = a.w;
      }
      e = *reinterpret_cast<const uint4 *>(s + kVals);
    }
    cur = cur + 1 == n ? 0 : cur + 1;
    out = out + 1 == kSlRing ? 0 : out + 1;
  }
};

// ns stages of a pass: per segment the sum of value * y_r[gathered slot].
// RESID = false: y_r[target] -= sum; RESID = true: emit(target, sums) on its
// last lane.  y holds NR values per slot.
template <typename T, int NR, bool RESID, typename Emit>
__device__ __forceinline__ void sl_stages(Ring<T> &ring, int ns, int N, double *y, int tid,
                                          Emit emit) {
  if (tid >= kSlStage) {
#pragma unroll 1
    for (; ns > 0; --ns) {
      ring.issue(tid - kSlStage);
      ring.landed();
      meet();
    }
    return;
  }
  const unsigned char *yb = reinterpret_cast<const unsigned char *>(y);
#pragma unroll 1
  for (; ns > 0; --ns) {
    if (ring.busy) {
      const uint4 e = ring.e;
      const uint32_t id[kSlRun] = {e.x & 0xffffu, e.y & 0xffffu, e.z & 0xffffu, e.w & 0xffffu};
      const uint32_t t = ring.used ? e.x >> 16 : (uint32_t)N, meta = e.y >> 16, ctl = e.w >> 16;
      double acc[NR], old[NR];
      // a segment's target is written once per level, so its old value can be
      // read before the sum, off the dependent chain
      if (!RESID) {
#pragma unroll
        for (int r = 0; r < NR; ++r) old[r] = y[t * NR + r];
      }
#pragma unroll
      for (int c = 0; c < kSlRun; ++c) {
        double g[NR];
        if (NR == 2) {
          const double2 u = *reinterpret_cast<const double2 *>(yb + id[c] * NR);
          g[0] = u.x;
          g[NR - 1] = u.y;
        } else {
          g[0] = *reinterpret_cast<const double *>(yb + id[c]);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const double x = __dmul_rn(ring.v[c], g[r]);
          acc[r] = c == 0 ? x : __dadd_rn(acc[r], x);
        }
        if (c == 0 && (ctl & 8u)) {  // (slot N is zero: no carry)
#pragma unroll
          for (int r = 0; r < NR; ++r) acc[r] = __dadd_rn(acc[r], y[(e.z >> 16) * NR + r]);
        }
      }
      const int reach = (int)(meta & 31u), steps = (int)(ctl & 7u);
#pragma unroll 1
      for (int h = 0; h < steps; ++h) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const double o = __shfl_up_sync(kFull, acc[r], 1u << h);
          if ((1 << h) <= reach) acc[r] = __dadd_rn(acc[r], o);
        }
      }
      if (ctl & 16u) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const double o = __shfl_up_sync(kFull, acc[r], 1);
          if (meta & 32u) acc[r] = __dadd_rn(acc[r], o);
        }
      }
      if (t < (unsigned)N) {
        if (RESID) {
          emit(t, acc);
        } else {
#pragma unroll
          for (int r = 0; r < NR; ++r) y[t * NR + r] = __dsub_rn(old[r], acc[r]);
        }
      } else if (t > (unsigned)N) {
#pragma unroll
        for (int r = 0; r < NR; ++r) y[t * NR + r] = acc[r];
      }
    }
    ring.take(tid);
    meet();
  }
}

// Vector loops of a block: each thread loads U elements of its stride before
// it uses any of them, so a loop costs one memory round trip per U * kNT.
constexpr int kU = 8;
#define SL_VEC(i, N, LOAD, USE)                                 \
  for (int i##0 = tid; i##0 < (N); i##0 += kNT * kU) {          \
    _Pragma("unroll") for (int u = 0; u < kU; ++u) {            \
      const int i = i##0 + kNT * u;                             \
      if (i < (N)) { LOAD }                                     \
    }                                                           \
    _Pragma("unroll") for (int u = 0; u < kU; ++u) {            \
      const int i = i##0 + kNT * u;                             \
      if (i < (N)) { USE }                                      \
    }                                                           \
  }

// block maxima of NR values (all threads get them); synchronises the block
template <int NR>
__device__ __forceinline__ void block_max_nr(double (&v)[NR], double (*red)[kSlWarps]) {
#pragma unroll
  for (int r = 0; r < NR; ++r) v[r] = warp_max(v[r]);
  __syncthreads();  // earlier reads of red are done
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int r = 0; r < NR; ++r) red[r][threadIdx.x >> 5] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    v[r] = red[r][0];
#pragma unroll
    for (int w = 1; w < kSlWarps; ++w) v[r] = fmax(v[r], red[r][w]);
  }
}

}  // namespace

// Solves NR right-hand sides with one factor, with iterative refinement by
// the rules of kktsolver_directldl_gpu.jl:349-410 per side.  A side that has
// finished keeps its accepted iterate in global scratch; its slots of y run
// along unused.
template <typename T, int NR>
__global__ void __launch_bounds__(kNT, kSlSolveBlocks)
    k_sl_solve(KKTDev k, LDLParams prm, const int *run, SolveIO<NR> io, int *ok, int first) {
  const int inst = k.sl_solve_inst[first + blockIdx.x];
  if (!run[inst] || !ok[inst]) return;
  const SlInst &si = k.sl[inst];
  const int N = si.N, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ double red[NR][kSlWarps];
  // stage ring | y (carries included) | b | stage table
  double *y = reinterpret_cast<double *>(sm_raw + kSlRing * Ring<T>::kSlot);
  double *b = y + (size_t)(N + 1 + si.ncarry) * NR;
  uint8_t *table = reinterpret_cast<uint8_t *>(b + (size_t)N * NR);
  const int vo = si.voff;
  double *x[NR], *e[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    x[r] = (r == 0 ? k.x : k.x2) + vo;
    e[r] = (r == 0 ? k.e : k.e2) + vo;
  }
  const int *__restrict__ gs = k.gsrc + vo;
  const T *Dinv = reinterpret_cast<const T *>(k.Dinv) + vo;
  const int nf = si.nf, nb = si.nb, nr = si.nr;
  for (int i = tid; i < nf + nb + nr; i += kNT) table[i] = k.sl_used[si.stage0 + i];
  __syncthreads();
  Ring<T> ring;
  ring.mem = sm_raw;
  ring.table = table;
  ring.nl = nf + nb;
  ring.n = nf + nb + nr;
  ring.at = ring.in = ring.cur = ring.out = 0;
  if (tid >= kSlStage) {
    const int lane = tid - kSlStage;
    ring.words0 = reinterpret_cast<const unsigned char *>(k.sl_ent + 4 * (size_t)si.lane0) +
                  16 * lane;
    ring.vals0 = reinterpret_cast<const unsigned char *>(
                     reinterpret_cast<const T *>(k.sl_val) + (size_t)si.vlane0 * kSlRun) +
                 16 * lane;
    ring.kvals0 = reinterpret_cast<const unsigned char *>(k.Kx + si.kx0) + 16 * lane;
    ring.words = ring.words0;
    ring.vals = ring.vals0;
    ring.kvals = ring.kvals0;
#pragma unroll 1
    for (int h = 0; h < kSlRing; ++h) ring.issue(lane);
    ring.landed();
  }
  double normb[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) normb[r] = 0.0;
  {
    int g[kU];
    double v[kU][NR];
    for (int i0 = tid; i0 < N; i0 += kNT * kU) {
#pragma unroll
      for (int u = 0; u < kU; ++u) g[u] = i0 + kNT * u < N ? gs[i0 + kNT * u] : -1;
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int r = 0; r < NR; ++r)
          v[u][r] = g[u] >= 0 ? io.rx[r][g[u]] : (g[u] == -1 ? 0.0 : io.rz[r][-g[u] - 2]);
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = i0 + kNT * u;
        if (i < N) {
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            b[i * NR + r] = v[u][r];
            y[i * NR + r] = v[u][r];
            normb[r] = fmax(normb[r], fabs(v[u][r]));
          }
        }
      }
    }
  }
  if (tid < NR) y[N * NR + tid] = 0.0;  // the slot padding gathers
  __syncthreads();  // the first two stages are in
  if (tid < kSlStage) ring.take(tid);
  block_max_nr<NR>(normb, red);
  int ntri = 0, nres = 0, nir = 0;  // passes (profiling)
  double tv[kU];
  auto trisolve = [&]() {
    ++ntri;
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      if (dir == 1) {
        SL_VEC(i, N, tv[u] = double(Dinv[i]);, {
          for (int r = 0; r < NR; ++r) y[i * NR + r] *= tv[u];
        })
        __syncthreads();
      }
      sl_stages<T, NR, false>(ring, dir == 0 ? nf : nb, N, y, tid,
                              [](uint32_t, double (&)[NR]) {});
    }
  };
  // e_r = b_r - K y_r; norme[r] = ||e_r||_inf (+inf when not finite), the sides on[r]
  auto residual = [&](const bool (&on)[NR], double (&norme)[NR]) {
    ++nres;
    double mx[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) mx[r] = 0.0;
    sl_stages<T, NR, true>(ring, nr, N, y, tid, [&](uint32_t t, double (&sum)[NR]) {
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (on[r]) {
          const double ev = __dsub_rn(b[t * NR + r], sum[r]);
          e[r][t] = ev;
          mx[r] = fmax(mx[r], isfinite(ev) ? fabs(ev) : CUDART_INF);
        }
    });
    block_max_nr<NR>(mx, red);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (on[r]) norme[r] = mx[r];
  };
  trisolve();
  bool good = true;
  if (prm.ir_enable) {
    // x keeps the accepted iterate; y holds the candidate the residual reads.
    // One thread decides which sides go on and leaves it in shared memory: a
    // sweep has meetings of the whole block, so the block follows one decision.
    // (As a bit mask in a register of every thread, nvcc 12.9 drops the two-side
    // build's sweeps.  It is its optimiser, before ptxas: the same with ptxas at
    // -O1, right when written with a flag per side.  The one-side results, which
    // the two-side ones equal bit for bit, show it.)
    __shared__ bool todo[NR];
    bool on[NR];
    double norme[NR], tol[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) on[r] = true;
    residual(on, norme);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      tol[r] = prm.ir_abstol + prm.ir_reltol * normb[r];
      for (int i = tid; i < N; i += kNT) x[r][i] = y[i * NR + r];
      good = good && isfinite(norme[r]);
    }
    if (tid == 0) {
#pragma unroll
      for (int r = 0; r < NR; ++r) todo[r] = good && norme[r] > tol[r];
    }
    __syncthreads();
    for (int it = 0; it < prm.ir_maxiter; ++it) {
      bool any = false;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        on[r] = todo[r];
        any = any || on[r];
      }
      if (!any) break;
      double last[NR];
      // (block_max_nr has synchronised since the last reads of y)
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        last[r] = norme[r];
        if (on[r]) {
          ++nir;
          SL_VEC(i, N, tv[u] = e[r][i];, y[i * NR + r] = tv[u];)
        }
      }
      __syncthreads();
      trisolve();
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (on[r])
          SL_VEC(i, N, tv[u] = x[r][i];, y[i * NR + r] += tv[u];)
      __syncthreads();
      residual(on, norme);
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (on[r]) {
          if (isfinite(norme[r])) {
            // kktsolver_directldl_gpu.jl:390-400: keep the candidate if it
            // improved on the last error; stop when the improvement ratio is
            // below stopratio
            const double ratio = last[r] / norme[r];
            if (ratio > 1.0 || ratio >= prm.ir_stopratio)
              for (int i = tid; i < N; i += kNT) x[r][i] = y[i * NR + r];
            on[r] = !(ratio < prm.ir_stopratio) && norme[r] > tol[r];
          } else {
            good = false;
          }
        }
      // (every thread has read todo before the sweep's meetings)
      if (tid == 0) {
#pragma unroll
        for (int r = 0; r < NR; ++r) todo[r] = good && on[r];
      }
      __syncthreads();
    }
  } else {
    double bad[1] = {0.0};
#pragma unroll
    for (int r = 0; r < NR; ++r)
      for (int i = tid; i < N; i += kNT) {
        x[r][i] = y[i * NR + r];
        if (!isfinite(y[i * NR + r])) bad[0] = 1.0;
      }
    block_max_nr<1>(bad, red);
    if (bad[0] > 0.0) good = false;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");  // stages of a round that is not run
  if (k.prof_bytes && tid == 0) {
    // algorithmic bytes: a substitution reads the factor (value + word per
    // entry, both directions) and D^-1, a residual reads K (value + word);
    // vectors are read / written once per use
    const double nl = si.nl, nk = si.nk, ts = sizeof(T);
    k.prof_bytes[(NR == 1 ? 1 : 2) * (size_t)k.B + inst] +=
        NR * 12.0 * N + ntri * (2.0 * nl * (4 + ts) + ts * N) +
        nres * (12.0 * nk + NR * 8.0 * N) + nir * 24.0 * N + NR * 28.0 * N;
  }
  if (!good) {
    if (tid == 0) ok[inst] = 0;
    return;
  }
  // x was written by the thread that reads it here (the same stride)
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    double *lx = io.lx[r], *lz = io.lz[r];
    const double *xr = x[r];
    int g[kU];
    SL_VEC(i, N, g[u] = gs[i]; tv[u] = xr[i];, {
      if (g[u] >= 0) {
        if (lx) lx[g[u]] = tv[u];
      } else if (g[u] <= -2) {
        if (lz) lz[-g[u] - 2] = tv[u];
      }
    })
  }
}

// ------------------------------------------------------------------------
// Factorisation.  Shared memory holds V: the diagonal [0, N), replaced by 1 /
// d_j once pivot j is taken, and U = L D [N, N + nl), initialised from K
// (static regularisation on the diagonal), a zero for padding and the carries.
// Per level: the warps' pages of updates V(t) -= U(i,k) U(j,k) / d_k; the lane
// that completes a diagonal takes its pivot at once (dynamic regularisation,
// QDLDL's Dsigns check), so a level has one meeting.  The leaves' pivots come
// first.  At the end L = U / d is written in substitution order.
//
// T is the storage type of L, D and D^-1, A the elimination's arithmetic:
// A = float (with T = float) is the mixed form, whose products, sums and
// pivot inverses are FP32 operations on the KKT values rounded to FP32.
__device__ __forceinline__ double sl_pivot(double dj, bool neg, const LDLParams &prm) {
  if (prm.dyn_reg) {
    const double sgn = neg ? -1.0 : 1.0;
    if (sgn * dj <= prm.dyn_eps) dj = prm.dyn_delta * sgn;
  }
  return dj;
}
__device__ __forceinline__ double sl_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float sl_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sl_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sl_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sl_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sl_sub(float a, float b) { return __fsub_rn(a, b); }

template <typename T, typename A>
__global__ void __launch_bounds__(kNT, kSlFactorBlocks)
    k_sl_factor(KKTDev k, LDLParams prm, const int *run, int *ok, double *eps_out, int first) {
  constexpr bool F32 = std::is_same<A, float>::value;
  const int inst = k.sl_factor_inst[first + blockIdx.x];
  if (!run[inst]) return;
  const SlInst &si = k.sl[inst];
  const int N = si.N, nl = si.nl, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ double red[1][kSlWarps];
  // op ring | expected pivot signs | V
  unsigned char *oring = sm_raw + warp * kSlOpRing * 512;
  signed char *sign = reinterpret_cast<signed char *>(sm_raw + kSlWarps * kSlOpRing * 512);
  A *V = reinterpret_cast<A *>(sign + (((size_t)N + 15) & ~(size_t)15));
  const int vo = si.voff;
  T *Dinv = reinterpret_cast<T *>(k.Dinv) + vo;
  const SlWarp &sw = si.w[warp];
  const unsigned char *ops =
      reinterpret_cast<const unsigned char *>(k.sl_ops + (size_t)(si.opage0 + sw.opage) *
                                                             kSlOpWords) + 16 * lane;
  const int nop = sw.nop, oskip = sw.oskip;
  const unsigned oaddr = static_cast<unsigned>(__cvta_generic_to_shared(oring)) + 16 * lane;
#pragma unroll
  for (int h = 0; h < kSlOpRing; ++h) {
    if (h < nop) cp16(oaddr + 512 * h, ops + (size_t)h * 512);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // ---- K into the work positions, the diagonal's static regularisation
  for (int i = tid; i < N + nl + 1 + si.nopcarry; i += kNT) V[i] = A(0);
  {
    int c[kU];
    SL_VEC(i, N, c[u] = k.sl_sign[vo + i];, sign[i] = (signed char)c[u];)
  }
  __syncthreads();
  {
    const double *__restrict__ kx = k.Kx + si.kx0;
    const uint16_t *__restrict__ kd = k.sl_kdst + si.kx0;
    const int nks = si.nkx;
    for (int i0 = tid; i0 < nks; i0 += kNT * kU) {
      unsigned p[kU];
      double v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) p[u] = i0 + kNT * u < nks ? kd[i0 + kNT * u] : kSlNone;
#pragma unroll
      for (int u = 0; u < kU; ++u) v[u] = i0 + kNT * u < nks ? kx[i0 + kNT * u] : 0.0;
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (p[u] != kSlNone) V[p[u]] = A(v[u]);
    }
  }
  __syncthreads();
  double eps = 0.0;
  if (prm.static_reg) {
    double mx[1] = {0.0};
    if constexpr (F32) {  // (from K itself: V holds it rounded)
      const double *__restrict__ kx = k.Kx + si.kx0;
      for (int j = tid; j < N; j += kNT) mx[0] = fmax(mx[0], fabs(kx[k.sl_kdiag[vo + j]]));
    } else {
      for (int j = tid; j < N; j += kNT) mx[0] = fmax(mx[0], fabs(V[j]));
    }
    block_max_nr<1>(mx, red);
    eps = prm.static_c + prm.static_prop * mx[0];
    const A ea = A(eps);
    for (int j = tid; j < N; j += kNT) V[j] = sl_add(V[j], sign[j] < 0 ? -ea : ea);
    __syncthreads();
  }
  bool finite = true;
  // pivot j with its completed diagonal dj: D^-1 stored, the value the
  // elimination continues with returned
  auto pivot = [&](int j, double dj) {
    dj = sl_pivot(dj, sign[j] < 0, prm);
    const T djs = T(dj);
    const T dis = T(1.0 / double(djs));
    Dinv[j] = dis;
    // FP32: the stored inverse is the elimination's value
    const double r = F32 || std::is_same<T, double>::value ? double(dis) : 1.0 / dj;
    if (!isfinite(r) || !isfinite(double(djs)) || !isfinite(double(dis))) finite = false;
    return A(r);
  };
  for (int i = tid; i < si.nleaf; i += kNT) {
    const int j = k.sl_leaf[vo + i];
    V[j] = pivot(j, double(V[j]));
  }
  __syncthreads();
  const int zero = N + nl;
  uint4 o = make_uint4(0, 0, 0, 0);
  int slot = 0;
  // op page p into registers, its slot refilled; one page ahead of use
  auto take = [&](int p) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kSlOpRing - 1) : "memory");
    o = *reinterpret_cast<const uint4 *>(oring + 512 * slot + 16 * lane);
    if (p + kSlOpRing < nop) cp16(oaddr + 512 * slot, ops + (size_t)(p + kSlOpRing) * 512);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    slot = slot + 1 == kSlOpRing ? 0 : slot + 1;
  };
  if (nop > 0) take(0);  // (a lane reads back the 16 bytes it copied)
  meet(oskip);
#pragma unroll 1
  for (int p = 0; p < nop; ++p) {
    constexpr unsigned m = 0x7fffu, mk = 0x1fffu;  // positions, diagonal positions
    const unsigned t = __funnelshift_r(o.z, o.w, 22) & m;
    // each target is written once per level end, so its old value is read
    // before the sum, off the dependent chain
    const A old = V[t];
    A x = sl_mul(sl_mul(V[o.x & m], V[(o.x >> 15) & m]), V[__funnelshift_r(o.x, o.y, 30) & mk]);
    x = sl_add(x, V[zero + ((o.w >> 5) & 0x7ffu)]);  // the carry, or zero
    const A x1 = sl_mul(sl_mul(V[(o.y >> 11) & m], V[__funnelshift_r(o.y, o.z, 26) & m]),
                        V[(o.z >> 9) & mk]);
    x = sl_add(x, x1);
    const int reach = (int)((o.w >> 16) & 31u), steps = (int)((o.w >> 22) & 7u);
#pragma unroll 1
    for (int h = 0; h < steps; ++h) {
      const A u = __shfl_up_sync(kFull, x, 1u << h);
      if ((1 << h) <= reach) x = sl_add(x, u);
    }
    {
      const A u = __shfl_up_sync(kFull, x, 1);
      if ((o.w >> 21) & 1u) x = sl_add(x, u);
    }
    if (t < (unsigned)N)
      V[t] = pivot((int)t, double(sl_sub(old, x)));
    else if (t != (unsigned)zero)
      V[t] = t < (unsigned)zero ? sl_sub(old, x) : x;
    const int ends = (int)(o.w >> 25);
    if (p + 1 < nop) take(p + 1);
    meet(ends);
  }
  // ---- L = U / d, into the order the substitutions read it
  {
    const uint16_t *__restrict__ ec = k.sl_ecol + si.ecol0;
    unsigned c[kU];
    SL_VEC(e, nl, c[u] = ec[e];, V[N + e] = sl_mul(V[N + e], V[c[u]]);)
  }
  const int bad = __syncthreads_or(finite ? 0 : 1);
  {
    const A *M = V + N;
    T *val = reinterpret_cast<T *>(k.sl_val) + (size_t)si.vlane0 * kSlRun;
    const uint16_t *__restrict__ lp = k.sl_lpos + (size_t)si.vlane0 * kSlRun;
    const int n = si.nvlane * kSlRun;
    for (int i0 = 2 * tid; i0 < n; i0 += 2 * kNT * kU) {
      unsigned p[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        p[u] = i0 + 2 * kNT * u < n
                   ? *reinterpret_cast<const unsigned *>(lp + i0 + 2 * kNT * u) : 0u;
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = i0 + 2 * kNT * u;
        if (i < n) {
          const unsigned pa = p[u] & 0xffffu, pb = p[u] >> 16;
          const T va = pa == kSlNone ? T(0) : T(M[pa]), vb = pb == kSlNone ? T(0) : T(M[pb]);
          if constexpr (sizeof(T) == 8)
            *reinterpret_cast<double2 *>(val + i) = make_double2(va, vb);
          else
            *reinterpret_cast<float2 *>(val + i) = make_float2(va, vb);
        }
      }
    }
  }
  if (tid == 0) {
    if (k.prof_bytes) {
      // K (value + work position), the ops, D^-1, and the factor in both orders
      // (value written, position read)
      const double ts = sizeof(T);
      k.prof_bytes[inst] += 10.0 * si.nk + 4.0 * si.nops + 2.0 * nl * (2.0 + ts) +
                            N * (ts + 1.0);
    }
    if (bad) ok[inst] = 0;
    if (eps_out) eps_out[inst] = eps;
  }
}

// The instances are grouped by shared memory (sl_groups), one launch per
// group, so that one large instance does not set the others' residency.
template <typename T, typename A>
static void factor_groups(const KKTDev &k, const LDLParams &p, const int *run, int *ok,
                          double *eps_out, cudaStream_t st) {
  for (int g = 0; g < k.sl_factor.n; ++g) {
    const SlGroup &gr = k.sl_factor.g[g];
    const int sm = sizeof(A) == 8 ? gr.smem : gr.smem2;
    k_sl_factor<T, A><<<gr.count, kNT, sm, st>>>(k, p, run, ok, eps_out, gr.first);
  }
}

template <typename T, int NR>
static void solve_groups(const KKTDev &k, const LDLParams &p, const int *run,
                         const SolveIO<NR> &io, int *ok, cudaStream_t st) {
  for (int g = 0; g < k.sl_solve.n; ++g) {
    const SlGroup &gr = k.sl_solve.g[g];
    k_sl_solve<T, NR><<<gr.count, kNT, NR == 1 ? gr.smem : gr.smem2, st>>>(k, p, run, io, ok,
                                                                        gr.first);
  }
}

static void sl_attrs() {
  static const bool done = [] {
    auto big = [](auto kern) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSlSmemMax);
      cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared);
    };
    big(k_sl_factor<double, double>);
    big(k_sl_factor<float, double>);
    big(k_sl_factor<float, float>);
    big(k_sl_solve<double, 1>);
    big(k_sl_solve<double, 2>);
    big(k_sl_solve<float, 1>);
    big(k_sl_solve<float, 2>);
    return true;
  }();
  (void)done;
}

void sl_factor(const KKTDev &k, bool fp32, bool arith32, const LDLParams &p, const int *run,
               int *ok, double *eps_out, cudaStream_t st) {
  sl_attrs();
  if (fp32 && arith32)
    factor_groups<float, float>(k, p, run, ok, eps_out, st);
  else if (fp32)
    factor_groups<float, double>(k, p, run, ok, eps_out, st);
  else
    factor_groups<double, double>(k, p, run, ok, eps_out, st);
}
void sl_solve(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
              const SolveIO<1> &io, int *ok, cudaStream_t st) {
  sl_attrs();
  if (fp32)
    solve_groups<float, 1>(k, p, run, io, ok, st);
  else
    solve_groups<double, 1>(k, p, run, io, ok, st);
}
void sl_solve2(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
               const SolveIO<2> &io, int *ok, cudaStream_t st) {
  sl_attrs();
  if (fp32)
    solve_groups<float, 2>(k, p, run, io, ok, st);
  else
    solve_groups<double, 2>(k, p, run, io, ok, st);
}

}  // namespace clgpu
