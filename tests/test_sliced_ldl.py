"""The block-per-instance LDL^T (csrc/ldl_sliced.cu) where its layouts have
edges: sums that span several chunks of their stream (rows and columns of more
than 128 and 256 terms), levels of one short page and of many pages, an
instance without off-diagonal factor entries, and pivots without dynamic
regularisation."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from cuclarabel_b200 import (BatchSolver, NonnegativeConeT, Solver, ZeroConeT, _lib, problems)
from cuclarabel_b200.api import Settings, _prep_problem
from helpers import ITER_TOL, OBJ_RTOL, rel_err


def budget(n, seed=0):
    """min x'Px/2 + q'x, sum x = 1, x >= 0: one row of n entries."""
    r = np.random.default_rng(seed)
    A = sp.vstack([sp.csc_matrix(np.ones((1, n))), -sp.identity(n)], format="csc")
    return (sp.diags(r.uniform(0.5, 2, n), format="csc"), r.standard_normal(n), A,
            np.concatenate([[1.0], np.zeros(n)]), [ZeroConeT(1), NonnegativeConeT(n)])


CASES = {
    "one_variable": lambda: (sp.csc_matrix([[2.0]]), np.array([-1.0]), sp.csc_matrix([[1.0]]),
                             np.array([0.3]), [NonnegativeConeT(1)]),
    "budget_127": lambda: budget(127),
    "budget_128": lambda: budget(128),
    "budget_300": lambda: budget(300),
    "psd_3": lambda: problems.psd_lp(3, 1, seed=2),
    "psd_8": lambda: problems.psd_lp(8, 3, seed=2),
    "mpc_small": lambda: problems.mpc_qp(5, n=20),
    "mpc_large": lambda: problems.mpc_qp(6, n=400),
}


@pytest.mark.parametrize("name", CASES)
def test_layouts_replay_on_the_host(name):
    cp, keep, n, m = _prep_problem(*CASES[name]())
    st = Settings().to_c()
    r = ctypes.c_double()
    rc = _lib.load().clgpu_debug_factor_stream(ctypes.byref(cp), ctypes.byref(st),
                                               ctypes.byref(r))
    assert rc == 0 and r.value < 1e-12, (rc, r.value)


@pytest.mark.gpu
@pytest.mark.parametrize("dyn", [True, False])
@pytest.mark.parametrize("name", CASES)
def test_solves_match_the_oracle(cuda_device, name, dyn):
    import oracle
    pb = CASES[name]()
    sol = Solver(*pb, dynamic_regularization_enable=dyn).solve()
    ref = oracle.solve(*pb)
    assert sol.status.name == ref["status_name"] == "SOLVED"
    assert rel_err(sol.obj_val, ref["obj_val"]) < OBJ_RTOL
    assert abs(sol.iterations - ref["iterations"]) <= ITER_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["cudss", "cudssmixed", "mixed_f64elim"])
def test_mixed_sizes_give_the_bits_of_each_alone(cuda_device, method):
    """Instances of very different shared-memory needs in one batch (so in
    several launches) return exactly what each returns alone."""
    pbs = [c() for c in CASES.values()]
    opts = dict(direct_solve_method=method, max_iter=4)
    for pb, s in zip(pbs, BatchSolver(pbs, **opts).solve()):
        a = BatchSolver([pb], **opts).solve()[0]
        assert np.array_equal(a.x, s.x) and np.array_equal(a.s, s.s) and np.array_equal(a.z, s.z)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["cudss", "cudssmixed", "mixed_f64elim"])
def test_two_sides_in_one_launch_are_each_its_own_solve(cuda_device, method):
    """Bit for bit, refinement included (the FP32 factors need several sweeps,
    and the two sides stop after different numbers of them)."""
    pbs = [c() for c in CASES.values()] + [problems.portfolio(2, 50, 5), problems.mpc_qp(7, n=900)]
    opts = dict(direct_solve_method=method, max_iter=8)
    for a, b in zip(BatchSolver(pbs, fused_solves=True, **opts).solve(),
                    BatchSolver(pbs, fused_solves=False, **opts).solve()):
        assert a.status == b.status and a.iterations == b.iterations
        assert np.array_equal(a.x, b.x) and np.array_equal(a.s, b.s) and np.array_equal(a.z, b.z)


# factors of more than 2^14 positions, up to what a block's shared memory takes
# (28 k), and one above it
LARGE = {"psd_10x4": lambda: problems.psd_lp(10, 4, seed=2),
         "psd_12x3": lambda: problems.psd_lp(12, 3, seed=2),
         "mpc_1200": lambda: problems.mpc_qp(5, n=1200),
         "mpc_2000": lambda: problems.mpc_qp(5, n=2000),
         "psd_12x4": lambda: problems.psd_lp(12, 4, seed=2)}


@pytest.mark.parametrize("name,want", [("psd_10x4", 0), ("psd_12x3", 0), ("mpc_1200", -4),
                                       ("mpc_2000", -4), ("psd_12x4", -3)])
def test_large_layouts_replay_on_the_host(name, want):
    """-4: takes these kernels, too large for the dense comparison; -3: does not
    take them."""
    cp, keep, n, m = _prep_problem(*LARGE[name]())
    st = Settings().to_c()
    r = ctypes.c_double()
    rc = _lib.load().clgpu_debug_factor_stream(ctypes.byref(cp), ctypes.byref(st),
                                               ctypes.byref(r))
    assert rc == want and (rc or r.value < 1e-12), (rc, r.value)


@pytest.mark.gpu
@pytest.mark.parametrize("name", LARGE)
def test_large_solves_match_the_oracle(cuda_device, name):
    import oracle
    pb = LARGE[name]()
    sol = Solver(*pb).solve()
    ref = oracle.solve(*pb)
    assert sol.status.name in ("SOLVED", "ALMOST_SOLVED") and ref["status_name"] == "SOLVED"
    assert rel_err(sol.obj_val, ref["obj_val"]) < OBJ_RTOL
    two = BatchSolver([pb] * 2, max_iter=6, fused_solves=False).solve()
    one = BatchSolver([pb], max_iter=6).solve()[0]
    assert all(np.array_equal(one.x, t.x) and np.array_equal(one.z, t.z) for t in two)


def _entries(pb, method="cudss"):
    cp, keep, n, m = _prep_problem(*pb)
    st = Settings(direct_solve_method=method).to_c()
    sn, ent = ctypes.c_int(), ctypes.c_longlong()
    assert _lib.load().clgpu_debug_instance_path(ctypes.byref(cp), ctypes.byref(st),
                                                 ctypes.byref(sn), ctypes.byref(ent)) == 0
    return sn.value, ent.value


@pytest.mark.parametrize("assets", [20, 50, 200])
def test_coupled_problems_are_ordered_by_minimum_degree(assets):
    """A budget row over all assets: dissection would leave 2 to 13 times K's
    entries, minimum degree stays below them (7 N bounds K here)."""
    P, q, A, b, cones = problems.portfolio(3, assets, 5)
    sn, ent = _entries((P, q, A, b, cones))
    assert sn == 0 and ent < 2 * A.nnz + len(q) + len(b)


@pytest.mark.parametrize("seed", [0, 1881, 2335, 3584])
def test_banded_problems_keep_dissection(seed):
    """The control family (its densest factor and deepest tree among them):
    minimum degree has less fill there but trees three to eight times as
    deep, so a shallow tree with more entries shows dissection."""
    pb = problems.mpc_qp(seed)
    cp, keep, n, m = _prep_problem(*pb)
    sn, ent = _entries(pb)
    nnz = 2 * pb[2].nnz + n + m  # K without the cones' blocks
    assert sn == 0 and ent > 0.5 * nnz


@pytest.mark.parametrize("method", ["cudss", "cudssmixed"])
def test_launch_groups_of_needs_around_a_threshold(method):
    """The first two need the same shared memory with one side and, with two,
    exactly 56 KB and 16 bytes more (the stage table is in both needs once), so
    by the one-side need alone they alternate between two launch groups.  Any
    batch takes at most three launches of each kind, every instance in one."""
    from cuclarabel_b200._lib import ClgpuProblem
    pair = [problems.mpc_qp(557, n=440), problems.mpc_qp(64, n=443)]
    pbs = pair * 5 + [problems.mpc_qp(5, n=n) for n in (20, 430, 1000)]
    base = [_prep_problem(*p) for p in pbs]
    arr = (ClgpuProblem * len(base))(*[b[0] for b in base])
    st = Settings(direct_solve_method=method).to_c()
    counts = (ctypes.c_int * 3)()
    rc = _lib.load().clgpu_debug_launch_groups(arr, len(base), ctypes.byref(st), counts)
    assert rc == 0 and counts[2] == len(base)
    assert 1 <= counts[0] <= 3 and 1 <= counts[1] <= 3, list(counts)


@pytest.mark.parametrize("method", ["cudssmixed", "mixed_f64elim"])
def test_fp32_factors_keep_dissection_unless_it_is_five_times_denser(method):
    """Minimum degree takes pivots that cost an FP32 factor digits: it stays for
    budgets over all assets, not for a few coupled semidefinite blocks."""
    dense, mild = problems.portfolio(3, 50, 5), problems.psd_lp(8, 3, seed=2)
    assert _entries(dense, method) == _entries(dense)
    assert _entries(mild, method)[1] > 1.5 * _entries(mild)[1]
