// ldl.cu -- batched sparse LDL^T numeric factorisation and solves (sm_100a).
//
// The block kernels: one block of 256 threads per instance, work vectors in
// global scratch, for the instances whose factor is too large for the shared
// memory of ldl_sliced.cu but too sparse for the supernodal path.
//
// Both the factorisation and the triangular solves are scheduled by
// elimination-tree levels (computed once by the symbolic phase): a column
// depends only on columns of lower levels, so every column of a level is
// processed concurrently and one barrier separates levels.  The KKT trees of
// the interior-point systems are bushy (height ~ N/10), which turns the
// O(N) chain of dependent steps into O(height).
//
// Factorisation, left-looking:
//   * wide level (>= NT/2 columns): one thread per column.  The column's
//     entries are accumulated in place: the lower part of K(:,j) and every
//     update column k (k in row j of L) are merged into column j's sorted
//     row list (the etree guarantees struct(L(j+1:,k)) is a subset of
//     struct(L(:,j))).
//   * narrow level: the whole block cooperates on one column through a dense
//     accumulator indexed by row; the update columns are applied one after
//     another with the threads spread over each column's rows.
// No floating-point atomics are used, so the factor of an instance is
// bitwise identical whether it is solved alone or inside any batch.
// Static regularisation (kktsolver_directldl_gpu.jl:216-260: eps = c +
// prop*||diag||_inf, diag +/- eps by the expected sign) is applied when the
// diagonal is read, so the stored KKT keeps its true diagonal for the
// refinement residual; dynamic regularisation follows the CPU path
// (sign*D(j) <= eps_dyn -> D(j) = sign*delta).
//
// Solve: forward substitution gathers each row of L (row pattern), backward
// substitution gathers each column, both level by level; then iterative
// refinement against the unregularised KKT exactly as
// kktsolver_directldl_gpu.jl:349-409.  In the mixed-precision form (the
// reference's :cudssmixed) L and D are STORED in FP32; accumulation,
// substitution arithmetic, the refinement residual and the iterate are FP64.
#include <type_traits>
#include "ldl.cuh"
#include "sn_exec.cuh"

namespace clgpu {

static constexpr int kNT = 256;

template <int NT>
__device__ __forceinline__ void bar_sync() {
  if (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double *red) {
  v = warp_sum(v);
  if (NT == 32) return v;
  int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NT / 32; ++i) t += red[i];
    red[NT / 32] = t;
  }
  __syncthreads();
  return red[NT / 32];
}
template <int NT>
__device__ __forceinline__ double block_max(double v, double *red) {
  v = warp_max(v);
  if (NT == 32) return v;
  int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = red[0];
    for (int i = 1; i < NT / 32; ++i) t = fmax(t, red[i]);
    red[NT / 32] = t;
  }
  __syncthreads();
  return red[NT / 32];
}

// Dynamic regularisation of pivot dj (kktsolver_directldl.jl:224-229 via
// QDLDL's Dsigns check): the FP64 pivot the elimination continues with.
__device__ __forceinline__ double pivot_value(double dj, signed char sg, const LDLParams &prm) {
  if (prm.dyn_reg) {
    const double sgn = double(sg);
    if (sgn * dj <= prm.dyn_eps) dj = prm.dyn_delta * sgn;
  }
  return dj;
}
// Stores pivot j: D and Dinv in the storage type T (Dinv is the inverse of
// the stored pivot so the solves see a consistent pair) and the FP64 pivot
// in Dacc, which aliases D in FP64 mode.  False if a stored value is not
// finite.
template <typename T>
__device__ __forceinline__ bool store_pivot(T *D, T *Dinv, double *Dacc, int j, double dj) {
  const T djs = T(dj);
  const T dis = T(1.0 / double(djs));
  D[j] = djs;
  Dinv[j] = dis;
  Dacc[j] = dj;
  return isfinite(double(djs)) && isfinite(double(dis));
}
// Stores factor entry q: the storage copy, and the FP64 value the rest of the
// elimination reads when the two differ.
template <typename T>
__device__ __forceinline__ void store_l(T *Lx, double *Lacc, int q, double v) {
  Lx[q] = T(v);
  if (!std::is_same<T, double>::value) Lacc[q] = v;
}
// FP32 operations on FP32 values held in FP64 slots (the mixed form's
// elimination)
__device__ __forceinline__ double f32r(double x) { return double(float(x)); }
__device__ __forceinline__ double f32mul(double a, double b) {
  return double(__fmul_rn(float(a), float(b)));
}
__device__ __forceinline__ double f32add(double a, double b) {
  return double(__fadd_rn(float(a), float(b)));
}
__device__ __forceinline__ double f32sub(double a, double b) {
  return double(__fsub_rn(float(a), float(b)));
}
// the pivot the FP32 elimination continues with: its stored inverse
__device__ __forceinline__ double f32inv(double dj) {
  return double(float(1.0 / double(float(dj))));
}

template <typename T, int NT, bool AR32 = false>
__global__ void __launch_bounds__(NT, 4) k_ldl_factor(KKTDev k, LDLParams prm, const int *run,
                                                   int *ok, double *eps_out) {
  int inst = blockIdx.x;
  if (!run[inst]) return;
  int N = k.N[inst];
  if (k.cls[inst] != 2) return;
  // AR32: FP32 arithmetic throughout (the mixed form's elimination)
  static_assert(!AR32 || std::is_same<T, float>::value, "FP32 arithmetic stores FP32");
  constexpr bool F32 = AR32;
  __shared__ double red[NT / 32 + 1];
  const int vo = k.voff[inst], po = k.poff[inst];
  double *w = k.w + vo;
  T *Lx = reinterpret_cast<T *>(k.Lx);
  // FP64 factor values the elimination reads (aliases Lx / D in FP64 mode)
  double *Lacc = k.Lacc ? k.Lacc : reinterpret_cast<double *>(k.Lx);
  T *D = reinterpret_cast<T *>(k.D) + vo;
  T *Dinv = reinterpret_cast<T *>(k.Dinv) + vo;
  double *Dacc = (k.Dacc ? k.Dacc : reinterpret_cast<double *>(k.D)) + vo;
  const int *Kp = k.Kp + po, *Lp = k.Lp + po, *Rp = k.Rp + po;
  const int *Kdiag = k.Kdiag + vo;
  const int *nodes = k.lvl_nodes + vo;
  const int *lptr = k.lvl_ptr + k.lvl_off[inst];
  const int nlev = k.nlev[inst];
  const signed char *sg = k.Dsign + vo;
  const int tid = threadIdx.x;
  for (int i = tid; i < N; i += NT) w[i] = 0.0;
  double eps = 0;
  if (prm.static_reg) {
    double mx = 0;
    for (int i = tid; i < N; i += NT) mx = fmax(mx, fabs(k.Kx[Kdiag[i]]));
    mx = block_max<NT>(mx, red);
    eps = prm.static_c + prm.static_prop * mx;
  }
  bar_sync<NT>();
  bool finite = true;
  for (int l = 0; l < nlev; ++l) {
    const int a = lptr[l], b = lptr[l + 1];
    if (b - a >= NT / 2) {
      // ---- wide level: one thread per column, merge into the column
      for (int idx = a + tid; idx < b; idx += NT) {
        const int j = nodes[idx];
        const int q0 = Lp[j], q1 = Lp[j + 1];
        for (int q = q0; q < q1; ++q) Lacc[q] = 0.0;
        double dj = 0.0;
        int q = q0;
        for (int p = Kp[j]; p < Kp[j + 1]; ++p) {
          int c = k.Kj[p];
          if (c < j) continue;
          if (c == j) {
            if constexpr (F32)
              dj = f32add(f32r(k.Kx[p]), f32r(sg[j] > 0 ? eps : -eps));
            else
              dj = k.Kx[p] + (sg[j] > 0 ? eps : -eps);
            continue;
          }
          while (q < q1 && k.Li[q] != c) ++q;
          if (q < q1) Lacc[q] = F32 ? f32r(k.Kx[p]) : k.Kx[p];
        }
        for (int r = Rp[j]; r < Rp[j + 1]; ++r) {
          const int kk = k.Rk[r], pos = k.Rpos[r];
          const double ljk = Lacc[pos];
          double f;
          if constexpr (F32) {
            f = f32mul(ljk, Dacc[kk]);
            dj = f32sub(dj, f32mul(ljk, f));
          } else {
            f = ljk * Dacc[kk];
            dj -= ljk * f;
          }
          const int pe = Lp[kk + 1];
          q = q0;
          for (int p = pos + 1; p < pe; ++p) {
            const int i = k.Li[p];
            while (q < q1 && k.Li[q] != i) ++q;
            if (q < q1) {
              if constexpr (F32)
                Lacc[q] = f32sub(Lacc[q], f32mul(Lacc[p], f));
              else
                Lacc[q] -= Lacc[p] * f;
            }
          }
        }
        dj = pivot_value(dj, sg[j], prm);
        if (F32) dj = f32r(dj);
        const double dinv = F32 ? f32inv(dj) : 1.0 / dj;
        if (!isfinite(dinv)) finite = false;
        for (int qq = q0; qq < q1; ++qq)
          store_l(Lx, Lacc, qq, F32 ? f32mul(Lacc[qq], dinv) : Lacc[qq] * dinv);
        if (!store_pivot(D, Dinv, Dacc, j, dj)) finite = false;
      }
      bar_sync<NT>();
    } else {
      // ---- narrow level: the block cooperates on each column
      for (int idx = a; idx < b; ++idx) {
        const int j = nodes[idx];
        for (int p = Kp[j] + tid; p < Kp[j + 1]; p += NT) {
          int c = k.Kj[p];
          if (c > j)
            w[c] = F32 ? f32r(k.Kx[p]) : k.Kx[p];
          else if (c == j)
            w[c] = F32 ? f32add(f32r(k.Kx[p]), f32r(sg[j] > 0 ? eps : -eps))
                       : k.Kx[p] + (sg[j] > 0 ? eps : -eps);
        }
        bar_sync<NT>();
        // update columns applied one after another (threads over the rows
        // of each update column, fixed order: the result is bitwise
        // reproducible and independent of the batch composition)
        const int r0 = Rp[j], r1 = Rp[j + 1];
        for (int rb = r0; rb < r1; rb += 32) {
          const int lane = tid & 31;
          int mypos = 0, myend = 0;
          double myf = 0.0, myl = 0.0;
          if (rb + lane < r1) {
            const int kk = k.Rk[rb + lane];
            mypos = k.Rpos[rb + lane];
            myend = Lp[kk + 1];
            myl = Lacc[mypos];
            myf = F32 ? f32mul(myl, Dacc[kk]) : myl * Dacc[kk];
          }
          const int cnt = min(32, r1 - rb);
          for (int t = 0; t < cnt; ++t) {
            const int pos = __shfl_sync(0xffffffffu, mypos, t);
            const int pe = __shfl_sync(0xffffffffu, myend, t);
            const double f = __shfl_sync(0xffffffffu, myf, t);
            const double ljk = __shfl_sync(0xffffffffu, myl, t);
            if constexpr (F32) {
              if (tid == 0) w[j] = f32sub(w[j], f32mul(ljk, f));
              for (int p = pos + 1 + tid; p < pe; p += NT)
                w[k.Li[p]] = f32sub(w[k.Li[p]], f32mul(Lacc[p], f));
            } else {
              if (tid == 0) w[j] -= ljk * f;
              for (int p = pos + 1 + tid; p < pe; p += NT) w[k.Li[p]] -= Lacc[p] * f;
            }
            bar_sync<NT>();
          }
        }
        double dj = pivot_value(w[j], sg[j], prm);
        if (F32) dj = f32r(dj);
        const double dinv = F32 ? f32inv(dj) : 1.0 / dj;
        if (!isfinite(dinv)) finite = false;
        for (int q = Lp[j] + tid; q < Lp[j + 1]; q += NT) {
          const int i = k.Li[q];
          store_l(Lx, Lacc, q, F32 ? f32mul(w[i], dinv) : w[i] * dinv);
          w[i] = 0.0;
        }
        bar_sync<NT>();
        if (tid == 0) {
          if (!store_pivot(D, Dinv, Dacc, j, dj)) finite = false;
          w[j] = 0.0;
        }
        bar_sync<NT>();
      }
    }
  }
  // copy of L in row order, which the forward substitution reads (every level
  // ended with a barrier, so all of Lx is written)
  {
    T *LxR = reinterpret_cast<T *>(k.LxR);
    const int rbeg = Rp[0], rend = Rp[N];
    for (int r = rbeg + tid; r < rend; r += NT) LxR[r] = Lx[k.Rpos[r]];
  }
  double bad = block_max<NT>(finite ? 0.0 : 1.0, red);
  if (k.prof_bytes && tid == 0) {
    // algorithmic bytes: K (indices + values) and the symbolic structure read
    // once, L, D, D^-1 and the row-order copy of L written once
    const double nl = Lp[N] - Lp[0], nk = Kp[N] - Kp[0], ts = sizeof(T);
    k.prof_bytes[inst] += 12.0 * nk + 16.0 * N + 12.0 * nl + ts * (nl + 2.0 * N) +
                          nl * (4.0 + ts);
  }
  if (tid == 0) {
    if (bad > 0) ok[inst] = 0;
    if (eps_out) eps_out[inst] = eps;
  }
}

// One node at a time over a run of consecutive narrow levels [a, e) of a
// schedule: y[node] -= sum_r V[r] * y[I[r]] over the node's entries
// [s.y, s.z), the block sharing each sum.  Nothing but y depends on the
// previous node, so each thread loads its first entry of the NEXT node (and
// that node's schedule record) before it reduces the current one; thread t
// accumulates entries s.y + t, s.y + t + NT, ... in order, as a plain loop
// would, so the result does not depend on the prefetch.
template <typename T, int NT>
__device__ __forceinline__ void narrow_run(const int4 *__restrict__ sched, int a, int e,
                                           const T *__restrict__ V,
                                           const int *__restrict__ I, double *y,
                                           double *red, int tid) {
  int4 s = sched[a];
  double pv = 0.0;
  int pk = -1;
  if (s.y + tid < s.z) {
    pv = double(V[s.y + tid]);
    pk = I[s.y + tid];
  }
  for (int idx = a; idx < e; ++idx) {
    int4 sn = make_int4(0, 0, 0, 0);
    if (idx + 1 < e) sn = sched[idx + 1];
    double nv = 0.0;
    int nk = -1;
    if (sn.y + tid < sn.z) {
      nv = double(V[sn.y + tid]);
      nk = I[sn.y + tid];
    }
    double t = 0.0;
    if (pk >= 0) t += pv * y[pk];
    for (int r = s.y + tid + NT; r < s.z; r += NT) t += double(V[r]) * y[I[r]];
    t = block_sum<NT>(t, red);
    if (tid == 0) y[s.x] -= t;
    bar_sync<NT>();
    s = sn;
    pv = nv;
    pk = nk;
  }
}

// y <- L^{-T} D^{-1} L^{-1} y, level-scheduled gathers.  Wide levels: one
// thread per node walks the node's row (forward) or column (backward).
// Runs of narrow levels: narrow_run.
template <typename T, int NT>
__device__ void ldl_trisolve(const KKTDev &k, int inst, int N, int vo, double *y,
                             double *red, int tid) {
  const T *Lx = reinterpret_cast<const T *>(k.Lx);
  const T *LxR = reinterpret_cast<const T *>(k.LxR);
  const T *Dinv = reinterpret_cast<const T *>(k.Dinv) + vo;
  const int4 *fs = k.fsched + vo, *bs = k.bsched + vo;
  const int *lptr = k.lvl_ptr + k.lvl_off[inst];
  const int nlev = k.nlev[inst];
  // forward: y_i -= sum_k L(i,k) y_k over the row pattern of i
  for (int l = 0; l < nlev;) {
    const int a = lptr[l], b = lptr[l + 1];
    if (b - a >= NT / 2) {
      for (int idx = a + tid; idx < b; idx += NT) {
        const int4 sc = fs[idx];
        double t = y[sc.x];
        for (int r = sc.y; r < sc.z; ++r) t -= double(LxR[r]) * y[k.Rk[r]];
        y[sc.x] = t;
      }
      bar_sync<NT>();
      ++l;
      continue;
    }
    int l2 = l + 1;
    while (l2 < nlev && lptr[l2 + 1] - lptr[l2] < NT / 2) ++l2;
    narrow_run<T, NT>(fs, a, lptr[l2], LxR, k.Rk, y, red, tid);
    l = l2;
  }
  for (int i = tid; i < N; i += NT) y[i] *= double(Dinv[i]);
  bar_sync<NT>();
  // backward: y_j -= sum_i L(i,j) y_i over column j (ancestors), root first
  for (int l = nlev - 1; l >= 0;) {
    const int a = N - lptr[l + 1], b = N - lptr[l];
    if (b - a >= NT / 2) {
      for (int idx = a + tid; idx < b; idx += NT) {
        const int4 sc = bs[idx];
        double t = y[sc.x];
        for (int p = sc.y; p < sc.z; ++p) t -= double(Lx[p]) * y[k.Li[p]];
        y[sc.x] = t;
      }
      bar_sync<NT>();
      --l;
      continue;
    }
    int l2 = l - 1;
    while (l2 >= 0 && lptr[l2 + 1] - lptr[l2] < NT / 2) --l2;
    narrow_run<T, NT>(bs, a, N - lptr[l2 + 1], Lx, k.Li, y, red, tid);
    l = l2;
  }
}

// e = b - K xi ; returns ||e||_inf (non-finite -> +inf)
template <int NT>
__device__ double refine_error(const KKTDev &k, int N, int po, const double *b,
                               const double *xi, double *e, double *red) {
  const int *Kp = k.Kp + po;
  double mx = 0;
  bool bad = false;
  for (int r = threadIdx.x; r < N; r += NT) {
    double t = 0;
    for (int p = Kp[r]; p < Kp[r + 1]; ++p) t += k.Kx[p] * xi[k.Kj[p]];
    double er = b[r] - t;
    e[r] = er;
    if (!isfinite(er)) bad = true;
    mx = fmax(mx, fabs(er));
  }
  mx = block_max<NT>(mx, red);
  double anybad = block_max<NT>(bad ? 1.0 : 0.0, red);
  return anybad > 0 ? CUDART_INF : mx;
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, 4) k_ldl_solve(KKTDev k, LDLParams prm, const int *run,
                                                  const double *rx, const double *rz,
                                                  double *lx, double *lz, int *ok) {
  int inst = blockIdx.x;
  if (!run[inst] || !ok[inst]) return;
  int N = k.N[inst];
  if (k.cls[inst] != 2) return;
  __shared__ double red[NT / 32 + 1];
  int vo = k.voff[inst], po = k.poff[inst];
  int tid = threadIdx.x;
  double *y = k.yf + vo;
  double *b = k.b + vo, *x = k.x + vo, *e = k.e + vo, *dx = k.dx + vo;
  const int *gs = k.gsrc + vo;
  double nb = 0;
  for (int i = tid; i < N; i += NT) {
    int g = gs[i];
    double v = g >= 0 ? rx[g] : (g == -1 ? 0.0 : rz[-g - 2]);
    b[i] = v;
    y[i] = v;
    nb = fmax(nb, fabs(v));
  }
  double normb = block_max<NT>(nb, red);
  bar_sync<NT>();
  ldl_trisolve<T, NT>(k, inst, N, vo, y, red, tid);
  for (int i = tid; i < N; i += NT) x[i] = y[i];
  bar_sync<NT>();
  bool good = true;
  if (prm.ir_enable) {
    double norme = refine_error<NT>(k, N, po, b, x, e, red);
    if (!isfinite(norme)) good = false;
    for (int it = 0; good && it < prm.ir_maxiter; ++it) {
      if (norme <= prm.ir_abstol + prm.ir_reltol * normb) break;
      double last = norme;
      for (int i = tid; i < N; i += NT) y[i] = e[i];
      bar_sync<NT>();
      ldl_trisolve<T, NT>(k, inst, N, vo, y, red, tid);
      for (int i = tid; i < N; i += NT) dx[i] = y[i] + x[i];
      bar_sync<NT>();
      norme = refine_error<NT>(k, N, po, b, dx, e, red);
      if (!isfinite(norme)) {
        good = false;
        break;
      }
      double ratio = last / norme;
      if (ratio < prm.ir_stopratio) {
        if (ratio > 1.0) {
          double *t = x;
          x = dx;
          dx = t;
        }
        break;
      }
      double *t = x;
      x = dx;
      dx = t;
    }
  } else {
    double bad = 0;
    for (int i = tid; i < N; i += NT)
      if (!isfinite(x[i])) bad = 1;
    if (block_max<NT>(bad, red) > 0) good = false;
  }
  if (!good) {
    if (tid == 0) ok[inst] = 0;
    return;
  }
  for (int i = tid; i < N; i += NT) {
    int g = gs[i];
    if (g >= 0) {
      if (lx) lx[g] = x[i];
    } else if (g <= -2) {
      if (lz) lz[-g - 2] = x[i];
    }
  }
}

template <typename T, bool AR32>
static void launch_factor(const KKTDev &k, const LDLParams &p, const int *run, int *ok,
                          double *eps_out, cudaStream_t st) {
  if (k.has_large)
    k_ldl_factor<T, kNT, AR32><<<k.B, kNT, 0, st>>>(k, p, run, ok, eps_out);
}
template <typename T>
static void launch_solve(const KKTDev &k, const LDLParams &p, const int *run,
                         const double *rx, const double *rz, double *lx, double *lz, int *ok,
                         cudaStream_t st) {
  if (k.has_large)
    k_ldl_solve<T, kNT><<<k.B, kNT, 0, st>>>(k, p, run, rx, rz, lx, lz, ok);
}

void ldl_factor(const KKTDev &k, bool fp32, const LDLParams &p, const int *run, int *ok,
                double *eps_out, cudaStream_t st, bool arith32) {
  sl_factor(k, fp32, arith32, p, run, ok, eps_out, st);
  if (fp32 && arith32)
    launch_factor<float, true>(k, p, run, ok, eps_out, st);
  else if (fp32)
    launch_factor<float, false>(k, p, run, ok, eps_out, st);
  else
    launch_factor<double, false>(k, p, run, ok, eps_out, st);
  if (k.sn) sn_factor(*k.sn, k, p, run, ok, eps_out, st);
}

void ldl_solve(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
               const double *rx, const double *rz, double *lx, double *lz, int *ok,
               cudaStream_t st) {
  sl_solve(k, fp32, p, run, SolveIO<1>{{rx}, {rz}, {lx}, {lz}}, ok, st);
  if (fp32)
    launch_solve<float>(k, p, run, rx, rz, lx, lz, ok, st);
  else
    launch_solve<double>(k, p, run, rx, rz, lx, lz, ok, st);
  if (k.sn) sn_solve(*k.sn, k, p, run, rx, rz, lx, lz, ok, st);
}

void ldl_solve2(const KKTDev &k, bool fp32, const LDLParams &p, const int *run,
                const double *rx0, const double *rz0, double *lx0, double *lz0,
                const double *rx1, const double *rz1, double *lx1, double *lz1, int *ok,
                cudaStream_t st) {
  sl_solve2(k, fp32, p, run,
            SolveIO<2>{{rx0, rx1}, {rz0, rz1}, {lx0, lx1}, {lz0, lz1}}, ok, st);
  auto block = [&](auto tag) {
    using T = decltype(tag);
    launch_solve<T>(k, p, run, rx0, rz0, lx0, lz0, ok, st);
    launch_solve<T>(k, p, run, rx1, rz1, lx1, lz1, ok, st);
  };
  if (fp32)
    block(float());
  else
    block(double());
  if (k.sn) {
    sn_solve(*k.sn, k, p, run, rx0, rz0, lx0, lz0, ok, st);
    sn_solve(*k.sn, k, p, run, rx1, rz1, lx1, lz1, ok, st);
  }
}

}  // namespace clgpu
