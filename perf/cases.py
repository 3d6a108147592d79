"""The workloads this library's speed is measured on.

listed() names them, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (solver or handle set up, new values in
hand), run() is one pass through the public entry points, exact() is the
64-bit value of the outputs that have a closed form.

Solves stop at tolerances, or after a number of iterations, at which the
iterate is still determined by the data to FP64 accuracy: below them the last
steps of the MPC family depend on the order of every sum, so two correct
solvers return different digits there.
"""
import ctypes
import functools

import numpy as np
import scipy.sparse as sp
import torch

from cuclarabel_b200 import BatchSolver, Solver, _lib, problems
from cuclarabel_b200.api import Settings

MPC_FAMILY = 4096  # structures the MPC cases take their instances from
PSD_SIDE = 10


def listed():
    return [
        # an adviser's tool: one small portfolio re-solved for new expected
        # returns; launches and latency set the time
        {"name": "portfolio_50", "kind": "portfolio", "assets": 50, "factors": 5},
        # the same for an ordinary fund: budget row over all assets
        {"name": "portfolio_200", "kind": "portfolio", "assets": 200, "factors": 10},
        # one controller, a new state each period, solved alone
        {"name": "mpc_single", "kind": "mpc", "first": 12, "count": 1, "method": "cudss",
         "tol": 1e-5, "max_iter": 200},
        # resident controllers served by the slot protocol
        {"name": "mpc_serve_256", "kind": "serve", "first": 256, "count": 256, "tol": 1e-5},
        # a fleet with a fixed budget of five iterations per period, FP32
        # factorisation with FP64 refinement
        {"name": "mpc_mixed_512", "kind": "mpc", "first": 1024, "count": 512,
         "method": "cudssmixed", "tol": 1e-8, "max_iter": 5},
        # the benchmark batch: every problem value new, every solution read
        {"name": "mpc_4096", "kind": "mpc", "first": 0, "count": 4096, "method": "cudss",
         "tol": 1e-5, "max_iter": 200},
        # relaxations: semidefinite programs of a few small blocks, as a batch
        {"name": "psd_lp_32", "kind": "psd_lp", "side": 8, "blocks": 3, "count": 32},
        # one larger mixed-cone problem on the dense-front factorisation
        {"name": "socp_2000", "kind": "socp", "scale": 0.1},
        # a caller's own interior-point loop: refactor and solve one large KKT
        # system (20000 variables, 60000 rows, 3000 second-order cones)
        {"name": "kkt_86000", "kind": "kkt", "scale": 1.0},
        # the same loop's cone operations, one iteration of them, per cone
        # family and at sizes where every vector is read from HBM
        {"name": "cones_socp", "kind": "cones", "nonneg": 2_800_000, "soc": 300_000, "dim": 10,
         "exp": 0, "pow": 0, "psd": 0},
        {"name": "cones_exp_pow", "kind": "cones", "nonneg": 500_000, "soc": 0, "dim": 10,
         "exp": 1_000_000, "pow": 250_000, "psd": 0},
        {"name": "cones_psd", "kind": "cones", "nonneg": 0, "soc": 0, "dim": 10, "exp": 0,
         "pow": 0, "psd": 40_000},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["portfolio", "mpc", "mpc", "serve", "psd_lp", "socp", "kkt", "cones",
                       "cones"])
    if kind == "portfolio":
        return {"kind": kind, "assets": _log(rng, 20, 200), "factors": rng.randint(3, 10)}
    if kind == "mpc":
        c = {"kind": kind, "first": rng.randrange(MPC_FAMILY), "count": _log(rng, 1, 4000)}
        if rng.random() < 0.3:
            return {**c, "method": rng.choice(["cudssmixed", "mixed_f64elim"]), "tol": 1e-8,
                    "max_iter": rng.randint(3, 5)}
        return {**c, "method": "cudss", "tol": rng.choice([1e-3, 1e-4, 1e-5]), "max_iter": 200}
    if kind == "serve":
        return {"kind": kind, "first": rng.randrange(MPC_FAMILY), "count": _log(rng, 8, 1000),
                "tol": rng.choice([1e-3, 1e-4, 1e-5])}
    if kind == "psd_lp":
        return {"kind": kind, "side": rng.randint(3, 12), "blocks": rng.randint(1, 4),
                "count": _log(rng, 1, 32)}
    if kind == "socp":
        return {"kind": kind, "scale": round(0.01 * 10 ** rng.random(), 4)}
    if kind == "kkt":
        return {"kind": kind, "scale": round(0.02 * 40 ** rng.random(), 4)}
    c = {"kind": kind, "nonneg": 0, "soc": 0, "dim": rng.randint(2, 24), "exp": 0, "pow": 0,
         "psd": 0}
    which = rng.randrange(3)
    if which == 0:
        c["nonneg"], c["soc"] = _log(rng, 1000, 2_000_000), _log(rng, 100, 100_000)
    elif which == 1:
        c["nonneg"], c["exp"], c["pow"] = (_log(rng, 100, 200_000), _log(rng, 100, 800_000),
                                           _log(rng, 100, 200_000))
    else:
        c["psd"] = _log(rng, 50, 30_000)
    return c


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _mpc(i):
    """One MPC structure, with what new values of it are drawn from."""
    P, q, A, b, cones = problems.mpc_qp(i % MPC_FAMILY)
    return P, q, A, b, cones, sp.csc_matrix(P + sp.triu(P, 1).T)


def _stack(mats):
    """Block-diagonal CSC of many CSC matrices."""
    rows = np.concatenate([[0], np.cumsum([m.shape[0] for m in mats])])
    nnz = np.concatenate([[0], np.cumsum([m.nnz for m in mats])])
    idx = np.concatenate([m.indices + r for m, r in zip(mats, rows)])
    ptr = np.concatenate([m.indptr[:-1] + z for m, z in zip(mats, nnz)] + [nnz[-1:]])
    data = np.concatenate([m.data for m in mats])
    return sp.csc_matrix((data, idx, ptr), shape=(rows[-1], len(ptr) - 1))


@functools.lru_cache(maxsize=4)
def _mpc_batch(first, count):
    base = [_mpc(first + k) for k in range(count)]
    kinds = []  # per row: 0 equality, 1 nonnegative, 2 cone head, 3 cone tail
    for p in base:
        for c in p[4]:
            t = c.spec()[0]
            kinds.append(np.full(c.nvars(), t) if t < 2 else np.r_[2, np.full(c.nvars() - 1, 3)])
    return (base, _stack([p[0] for p in base]), _stack([p[5] for p in base]),
            _stack([p[2] for p in base]), np.concatenate(kinds))


def _interior(r, kinds, equality):
    """A point inside the cones of the rows; 0 (slack) or N(0,1) (dual) on
    the equality rows."""
    v = r.standard_normal(len(kinds))
    v[kinds == 1] = r.uniform(0.5, 2, int(np.sum(kinds == 1)))
    heads = np.flatnonzero(kinds == 2)
    if len(heads):
        cone = np.cumsum(kinds == 2)
        norm2 = np.zeros(len(heads))
        np.add.at(norm2, (cone - 1)[kinds == 3], v[kinds == 3] ** 2)
        v[heads] = 1.0 + np.sqrt(norm2)
    if not equality:
        v[kinds == 0] = 0.0
    return v


def _mpc_values(first, count, seed, matrices):
    """New values for a batch: states, slacks and duals drawn afresh (and the
    matrices' entries moved by a per cent), so every instance stays feasible
    and bounded."""
    base, P, Pf, A, kinds = _mpc_batch(first, count)
    r = np.random.default_rng(seed)
    Av, An = A.data, A
    if matrices:
        Av = A.data * (1 + 0.01 * r.standard_normal(A.nnz))
        An = sp.csc_matrix((Av, A.indices, A.indptr), shape=A.shape)
    x0 = r.standard_normal(A.shape[1])
    s0, z0 = _interior(r, kinds, False), _interior(r, kinds, True)
    q, b = -(Pf @ x0) - An.T @ z0, An @ x0 + s0
    return base, P.data.copy(), q, Av.copy(), b


def _tol(t):
    return dict(tol_gap_abs=t, tol_gap_rel=t, tol_feas=t)


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _split(v, sizes):
    return np.split(v, np.cumsum(sizes)[:-1])


def _kkt_matrix(scale, seed):
    """KKT matrix of the large mixed-cone family at an interior iterate:
    [P A'; A -H] with H diagonal on the nonnegative rows and the diagonal plus
    rank-two expansion (two extra rows) on each second-order cone."""
    P, _, A, _, cones = problems.mixed_socp(scale, seed)
    r = np.random.default_rng(seed + 1)
    n, m = A.shape[1], A.shape[0]
    nz, nn = cones[0].dim, cones[1].dim
    k = len(cones) - 2
    d = cones[2].dim
    # an entry of its own column makes every equality row independent, so the
    # system has one solution
    A = A + sp.csc_matrix((2 + np.abs(r.standard_normal(nz)),
                           (np.arange(nz), r.permutation(n)[:nz])), shape=(m, n))
    eta2 = np.exp(r.normal(0, 1, k))
    w1 = 0.5 * r.standard_normal((k, d - 1))
    w0 = np.sqrt(1 + np.sum(w1 * w1, 1))
    wsq = w0 * w0 + np.sum(w1 * w1, 1)
    dd = 0.5 / wsq
    u0 = np.sqrt(wsq - dd)
    u = np.concatenate([u0[:, None], (2 * w0 / u0)[:, None] * w1], 1)
    v = np.concatenate([np.zeros((k, 1)),
                        np.sqrt(2 * (2 + 1 / wsq) / (2 * wsq - 1 / wsq))[:, None] * w1], 1)
    Dm = np.ones((k, d))
    Dm[:, 0] = dd
    hdiag = np.concatenate([np.zeros(nz), np.exp(r.normal(0, 1.5, nn)),
                            (eta2[:, None] * Dm).ravel()])
    rows = (nz + nn + np.arange(k * d)).repeat(2)
    cols = np.stack([np.repeat(2 * np.arange(k), d), np.repeat(2 * np.arange(k) + 1, d)],
                    1).ravel()
    vals = np.stack([-(eta2[:, None] * v).ravel(), -(eta2[:, None] * u).ravel()], 1).ravel()
    E = sp.csr_matrix((vals, (rows, cols)), shape=(m, 2 * k))
    ext = np.stack([-eta2, eta2], 1).ravel()
    Pf = P + sp.triu(P, 1).T
    # the zero rows keep their (zero) diagonal as an entry of the pattern
    H = sp.csr_matrix((-hdiag, np.arange(m), np.arange(m + 1)), shape=(m, m))
    K = sp.bmat([[Pf, A.T, None], [A, H, E], [None, E.T, sp.diags(ext)]], format="csr")
    K.sort_indices()
    signs = np.concatenate([np.ones(n), -np.ones(m), np.tile([-1, 1], k)]).astype(np.int8)
    x = r.standard_normal(K.shape[0])
    return K, signs, x


def _cone_rows(case):
    return (case["nonneg"], case["soc"] * case["dim"], 3 * case["exp"], 3 * case["pow"],
            case["psd"] * PSD_SIDE * (PSD_SIDE + 1) // 2)


def _triangle():
    ii = [i for j in range(PSD_SIDE) for i in range(j + 1)]
    jj = [j for j in range(PSD_SIDE) for i in range(j + 1)]
    return ii, jj


def _cone_inputs(case, seed, device):
    """Strictly interior s and z, steps dz and ds, and a vector x."""
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    f8 = dict(dtype=torch.float64, device=device, generator=g)

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, **f8)

    k, d = case["soc"], case["dim"]
    alpha = uni(0.2, 0.8, case["pow"])

    def point():
        tail = torch.randn(k, d - 1, **f8)
        head = 1 + tail.norm(dim=1, keepdim=True) * uni(1.05, 2, k, 1)
        e = torch.tensor([-1.051383945322714, 0.556409619469370, 1.258967884768947],
                         dtype=torch.float64, device=device) * uni(0.5, 2, case["exp"], 1)
        e = e + 0.02 * torch.randn(case["exp"], 3, **f8)
        p = torch.stack([(1 + alpha).sqrt(), (2 - alpha).sqrt(), torch.zeros_like(alpha)], 1)
        p = p * uni(0.5, 2, case["pow"], 1)
        p[:, 2] = 0.1 * torch.randn(case["pow"], **f8)
        E = 0.1 * torch.randn(case["psd"], PSD_SIDE, PSD_SIDE, **f8)
        M = torch.eye(PSD_SIDE, dtype=torch.float64, device=device) + (E + E.mT) / 2
        return torch.cat([uni(0.5, 2, case["nonneg"]), torch.cat([head, tail], 1).reshape(-1),
                          e.reshape(-1), p.reshape(-1), _svec(M).reshape(-1)])

    s, z = point(), point()
    m = s.numel()
    dz, ds = 0.2 * torch.randn(m, **f8), 0.2 * torch.randn(m, **f8)
    return s, z, dz, ds, torch.randn(m, **f8), alpha.cpu().numpy()


class _Handle:
    """A C handle that is destroyed with the state that holds it."""

    def __init__(self, h, destroy):
        self.h, self._destroy = h, destroy

    def __del__(self):
        if self._destroy is not None and self.h:
            self._destroy(self.h)
            self.h = None


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "portfolio":
        P, q, A, b, cones = problems.portfolio(seed, case["assets"], case["factors"])
        st["solver"] = Solver(P, q, A, b, cones)
        r = np.random.default_rng(seed + 1)
        st["q"] = q.copy()
        st["q"][:case["assets"]] = -(3 + 9 * r.uniform(0, 1, case["assets"])) / 100.0
    elif kind == "mpc":
        base, Pv, q, Av, b = _mpc_values(case["first"], case["count"], seed, case["count"] > 1)
        opts = dict(direct_solve_method=case["method"], max_iter=case["max_iter"],
                    **_tol(case["tol"]))
        if case["count"] == 1:
            st.update(solver=Solver(*base[0][:5], **opts), q=q, b=b)
        else:
            st.update(kind="batch", solver=BatchSolver([p[:5] for p in base], **opts),
                      stream=torch.cuda.Stream(), out=None)
            st.update(P=_pinned(Pv), q=_pinned(q), A=_pinned(Av), b=_pinned(b))
    elif kind == "serve":
        base, _, q, _, b = _mpc_values(case["first"], case["count"], seed, False)
        st.update(solver=BatchSolver([p[:5] for p in base], **_tol(case["tol"])),
                  stream=torch.cuda.Stream(), slots=list(range(case["count"])),
                  q=_split(q, [len(p[1]) for p in base]),
                  b=_split(b, [len(p[3]) for p in base]))
    elif kind == "psd_lp":
        pbs = [problems.psd_lp(case["side"], case["blocks"], seed=seed * 64 + k)
               for k in range(case["count"])]
        st.update(kind="batch", solver=BatchSolver(pbs, **_tol(1e-6)),
                  stream=torch.cuda.Stream(), out=None, P=None, A=None,
                  q=_pinned(np.concatenate([p[1] for p in pbs])),
                  b=_pinned(np.concatenate([p[3] for p in pbs])))
    elif kind == "socp":
        pb = problems.mixed_socp(case["scale"], seed)
        st.update(kind="mpc", solver=Solver(*pb, **_tol(1e-4)), q=pb[1], b=pb[3])
    elif kind == "kkt":
        K, signs, x = _kkt_matrix(case["scale"], seed)
        L, h = _lib.load(), ctypes.c_void_p()
        Kp, Kj = K.indptr.astype(np.int32), K.indices.astype(np.int32)
        cs = Settings().to_c()
        rc = L.clgpu_ldl_create(K.shape[0], Kp.ctypes.data_as(_lib.ip),
                                Kj.ctypes.data_as(_lib.ip),
                                signs.ctypes.data_as(ctypes.POINTER(ctypes.c_byte)),
                                ctypes.byref(cs), ctypes.byref(h))
        if rc != 0:
            raise RuntimeError("clgpu_ldl_create: %d" % rc)
        st.update(L=L, handle=_Handle(h, L.clgpu_ldl_destroy), K=torch.from_numpy(K.data).cuda(),
                  b=torch.from_numpy(K @ x).cuda(),
                  x=torch.empty(K.shape[0], dtype=torch.float64, device="cuda"))
    else:
        s, z, dz, ds, x, alpha = _cone_inputs(case, seed, "cuda")
        counts = [(1, case["nonneg"], 1 if case["nonneg"] else 0), (2, case["dim"], case["soc"]),
                  (3, 3, case["exp"]), (4, 3, case["pow"]), (5, PSD_SIDE, case["psd"])]
        types = np.concatenate([np.full(c, t, np.int32) for t, _, c in counts])
        dims = np.concatenate([np.full(c, d, np.int32) for _, d, c in counts])
        par = np.zeros(len(types))
        par[types == 4] = alpha
        L, h = _lib.load(), ctypes.c_void_p()
        rc = L.clgpu_cones_create(len(types), types.ctypes.data_as(_lib.ip),
                                  dims.ctypes.data_as(_lib.ip), par.ctypes.data_as(_lib.dp), 5,
                                  ctypes.byref(h))
        if rc != 0:
            raise RuntimeError("clgpu_cones_create: %d" % rc)
        st.update(L=L, handle=_Handle(h, L.clgpu_cones_destroy), s=s, z=z, dz=dz, ds=ds, x=x,
                  y=torch.empty_like(s), aff=torch.empty_like(s), shift=torch.empty_like(s),
                  off=torch.empty_like(s))
    return st


# --------------------------------------------------------------------- run
def _ok(rc):
    if rc != 0:
        raise RuntimeError("clgpu call returned %d" % rc)


def run(st):
    kind = st["kind"]
    if kind == "portfolio":
        st["solver"].update_q(st["q"])
        return _solution(st["solver"].solve())
    if kind == "mpc":
        st["solver"].update_q(st["q"])
        st["solver"].update_b(st["b"])
        return _solution(st["solver"].solve())
    if kind == "batch":
        sv, sh = st["solver"], st["stream"].cuda_stream
        sv.update_data(P=st["P"], q=st["q"], A=st["A"], b=st["b"], stream=sh)
        sv.solve_only(sh)
        st["out"] = r = sv.results(out=st["out"], view=True)
        return {"x": r["x"], "s": r["s"], "z": r["z"], "status": r["status"],
                "iterations": r["info"]["iterations"].copy(),
                "objective": r["info"]["obj_val"].copy()}
    if kind == "serve":
        sv, sh = st["solver"], st["stream"].cuda_stream
        sv.serve_admit(st["slots"], st["q"], st["b"], sh)
        sols, running = {}, 1
        while running:
            done, running = sv.serve_step(sh)
            for k, s in zip(done, sv.serve_collect(done, sh)):
                sols[k] = s
        sols = [sols[k] for k in st["slots"]]
        return {"x": np.concatenate([s.x for s in sols]),
                "s": np.concatenate([s.s for s in sols]),
                "z": np.concatenate([s.z for s in sols]),
                "objective": np.array([s.obj_val for s in sols]),
                "status": np.array([int(s.status) for s in sols]),
                "iterations": np.array([s.iterations for s in sols])}
    L, h, sh = st["L"], st["handle"].h, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "kkt":
        eps = ctypes.c_double()
        _ok(L.clgpu_ldl_refactor(h, _ptr(st["K"]), ctypes.byref(eps), sh))
        _ok(L.clgpu_ldl_solve(h, _ptr(st["b"]), _ptr(st["x"]), sh))
        return {"x": st["x"], "eps": eps.value}
    s, z, dz, ds = (_ptr(st[k]) for k in ("s", "z", "dz", "ds"))
    alpha = ctypes.c_double()
    _ok(L.clgpu_update_scaling(h, s, z, 1.0, 0, sh))
    _ok(L.clgpu_mul_Hs(h, _ptr(st["y"]), _ptr(st["x"]), sh))
    _ok(L.clgpu_affine_ds(h, _ptr(st["aff"]), s, sh))
    _ok(L.clgpu_combined_ds_shift(h, _ptr(st["shift"]), dz, ds, z, 0.1, sh))
    _ok(L.clgpu_ds_from_dz_offset(h, _ptr(st["off"]), _ptr(st["shift"]), z, sh))
    _ok(L.clgpu_step_length(h, dz, ds, z, s, 1.0, 0.99, 0.8, 1e-4, ctypes.byref(alpha), sh))
    # the shift itself lives in the scaled frame, which the semidefinite cones
    # know up to the signs of their singular vectors: its offset is the result
    return {"Hs_x": st["y"], "affine_ds": st["aff"], "offset": st["off"], "alpha": alpha.value}


def _solution(s):
    return {"x": s.x, "s": s.s, "z": s.z, "objective": s.obj_val, "status": int(s.status),
            "iterations": s.iterations}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass that no implementation saves: a solve
    reads its data and writes its solution, and per iteration (counts typical
    of the family) reads the KKT values for the factor and both residuals,
    writes the factor and reads it for two solves, and reads and writes its
    iterate, residuals and two steps once."""
    kind = case["kind"]
    if kind == "kkt" or kind == "socp":
        # the trailing block of these random patterns is dense
        n, entries, flops = 86000 * case["scale"], 1.9e8 * case["scale"] ** 2, \
            2.4e12 * case["scale"] ** 3
        per = 14 if kind == "socp" else 1
        return {"bytes": per * 8 * (3 * entries + 60 * n), "flops": per * (flops + 8 * entries)}
    if kind == "cones":
        nn, soc, exp, pow_, psd = _cone_rows(case)
        t = PSD_SIDE * (PSD_SIDE + 1) // 2
        # rows in: s, z (scaling and step), x, dz, ds; rows out: three vectors
        rows = 8 * (nn + soc + exp + pow_ + psd) * 8
        state = 8 * (2 * nn + 3 * soc) + 24 * 8 * (exp + pow_) // 3 + 8 * 300 * (psd // t)
        flops = 40 * nn + 60 * soc + 1500 * (exp + pow_) // 3 + 20 * PSD_SIDE ** 3 * (psd // t)
        return {"bytes": rows + state, "flops": flops}
    if kind == "portfolio":
        a, k = case["assets"], case["factors"]
        n, m, iters, count = 3 * a + k, 4 * a + k + 1, 8, 1
        kkt, fac = 2 * (a * k // 2 + 7 * a) + n + m, a * k + 10 * a
    elif kind == "psd_lp":
        t = case["side"] * (case["side"] + 1) // 2
        n, iters, count = case["blocks"] * t, 7, case["count"]
        m = n + max(1, n // 4)
        kkt, fac = case["blocks"] * t * t + 20 * n, case["blocks"] * t * t + 20 * n
    else:
        n, m, count = 210, 420, case["count"]
        iters = min(9, case.get("max_iter", 200))
        kkt, fac = 12 * n, 11 * n
    per = 8 * (3 * kkt + 3 * fac + 8 * n + 16 * m)
    return {"bytes": count * (iters * per + 8 * (2 * n + 3 * m + kkt)),
            "flops": count * iters * (20 * fac + 12 * kkt + 60 * (n + m))}


# ------------------------------------------------------------------- exact
def _svec(M):
    ii, jj = _triangle()
    w = torch.tensor([1.0 if i == j else 2.0 ** 0.5 for i, j in zip(ii, jj)],
                     dtype=torch.float64, device=M.device)
    return M[:, ii, jj] * w


def _smat(v):
    ii, jj = _triangle()
    w = torch.tensor([1.0 if i == j else 0.5 ** 0.5 for i, j in zip(ii, jj)],
                     dtype=torch.float64, device=v.device)
    M = torch.zeros(len(v), PSD_SIDE, PSD_SIDE, dtype=torch.float64, device=v.device)
    M[:, ii, jj] = v * w
    M[:, jj, ii] = v * w
    return M


def _soc_exact(s, z, dz, ds, x):
    """Nesterov-Todd scaling of second-order cones held one per row."""
    def jdot(a, b):
        return a[:, 0] * b[:, 0] - (a[:, 1:] * b[:, 1:]).sum(1)

    def jnorm(a):
        t = a[:, 1:].norm(dim=1)
        return ((a[:, 0] - t) * (a[:, 0] + t)).sqrt()

    def times(w, eta, v, sign):
        w1v1 = (w[:, 1:] * v[:, 1:]).sum(1)
        head = w[:, 0] * v[:, 0] + sign * w1v1
        tail = v[:, 1:] + (sign * v[:, 0] + w1v1 / (1 + w[:, 0]))[:, None] * w[:, 1:]
        return eta[:, None] * torch.cat([head[:, None], tail], 1)

    def circ(a, b):
        return torch.cat([(a * b).sum(1, keepdim=True),
                          a[:, :1] * b[:, 1:] + b[:, :1] * a[:, 1:]], 1)

    def reach(v, dv):
        # smallest positive root of (v + a dv)' J (v + a dv), J-product scaled
        a, b, c = jdot(dv, dv), 2 * jdot(v, dv), jnorm(v) ** 2
        disc = b * b - 4 * a * c
        q = -0.5 * (b + torch.where(b >= 0, 1.0, -1.0) * disc.clamp(min=0).sqrt())
        roots = torch.stack([q / a, c / q])
        roots = torch.where((roots > 0) & (disc >= 0), roots, float("inf"))
        return float(roots.min())

    ns, nz = jnorm(s), jnorm(z)
    sb, zb = s / ns[:, None], z / nz[:, None]
    gamma = ((1 + (sb * zb).sum(1)) / 2).sqrt()
    w = sb.clone()
    w[:, 0] += zb[:, 0]
    w[:, 1:] -= zb[:, 1:]
    w = w / (2 * gamma[:, None])
    eta = (ns / nz).sqrt()
    lam = times(w, eta, z, 1.0)
    hx = times(w, eta, times(w, eta, x, 1.0), 1.0)
    shift = circ(times(w, 1 / eta, ds, -1.0), times(w, eta, dz, 1.0))
    shift[:, 0] -= 0.1
    # lam \ shift
    c0 = jdot(lam, shift) / jnorm(lam) ** 2
    inv = torch.cat([c0[:, None], (shift[:, 1:] - c0[:, None] * lam[:, 1:]) / lam[:, :1]], 1)
    return hx, circ(lam, lam), times(w, eta, inv, 1.0), min(reach(z, dz), reach(s, ds))


def _psd_exact(s, z, dz, ds, x):
    S, Z, DZ, DS, X = (_smat(v) for v in (s, z, dz, ds, x))
    L1, L2 = torch.linalg.cholesky(S), torch.linalg.cholesky(Z)
    U, lam, Vt = torch.linalg.svd(L2.mT @ L1)
    R = L1 @ Vt.mT / lam.sqrt()[:, None, :]
    Ri = (U.mT @ L2.mT) / lam.sqrt()[:, :, None]
    dzs, dss = R.mT @ DZ @ R, Ri @ DS @ Ri.mT
    shift = (dss @ dzs + dzs @ dss) / 2 - 0.1 * torch.eye(PSD_SIDE, dtype=S.dtype,
                                                         device=S.device)
    inv = 2 * shift / (lam[:, :, None] + lam[:, None, :])
    WW = R @ R.mT

    def reach(L, D):
        T = torch.linalg.solve_triangular(L, D, upper=False)
        T = torch.linalg.solve_triangular(L, T.mT, upper=False)
        low = torch.cat([torch.linalg.eigvalsh(t)[:, 0]
                         for t in ((T + T.mT) / 2).split(4096)]).min()
        return float("inf") if low >= 0 else -1.0 / float(low)
    return (_svec(WW @ X @ WW), _svec(torch.diag_embed(lam * lam)), _svec(R @ inv @ R.mT),
            min(reach(L2, DZ), reach(L1, DS)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "kkt":
        # the right-hand side is K times this vector
        return {"x": _kkt_matrix(case["scale"], seed)[2], "eps": None}
    if kind != "cones" or case["exp"] or case["pow"]:
        # a solve ends at its tolerance, not at the optimum, and the
        # exponential and power cones' scaling is the end of an inner
        # iteration: neither has a closed form
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s, z, dz, ds, x, _ = _cone_inputs(case, seed, dev)
    nn, soc = case["nonneg"], case["soc"] * case["dim"]
    v = [t[:nn] for t in (s, z, dz, ds, x)]
    parts = [(v[0] / v[1] * v[4], v[0] * v[1], (v[2] * v[3] - 0.1) / v[1])]
    alpha = 1.0
    if nn:
        for a, b in ((v[1], v[2]), (v[0], v[3])):
            alpha = min(alpha, float(torch.where(b < 0, -a / b, float("inf")).min()))
    for f, lo, hi, width in ((_soc_exact, nn, nn + soc, case["dim"]),
                             (_psd_exact, nn + soc, s.numel(),
                              PSD_SIDE * (PSD_SIDE + 1) // 2)):
        if hi > lo:
            *p, a = f(*(t[lo:hi].view(-1, width) for t in (s, z, dz, ds, x)))
            parts.append([t.reshape(-1) for t in p])
            alpha = min(alpha, a)
    h, a, o = (torch.cat([p[k].reshape(-1) for p in parts]) for k in range(3))
    return {"Hs_x": h, "affine_ds": a, "offset": o, "alpha": alpha}
