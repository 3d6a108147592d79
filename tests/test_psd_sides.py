"""PSD scaling and step length on both sides of the side limit (16) of the
kernels that give a lane a rotation and a thread a matrix: sides at the edges,
cone counts that do not fill a warp (8) or a block, and matrices with repeated
or zero eigenvalues, against the oracle.  Tolerances are those of
test_gpu_cones.py: FP64 arithmetic with condition numbers below about 1e2."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_cones import GPUCones, close

pytestmark = pytest.mark.gpu

SIDES = {"one": [1], "two": [2] * 3, "three": [3] * 9, "ten": [10] * 17, "fifteen": [15] * 5,
         "sixteen": [16] * 35, "seventeen": [17] * 3, "mixed": [1, 16, 7, 2, 15, 10, 8, 3, 5] * 4,
         "mixed_large": [1, 16, 17, 2, 9]}


def interior(rng, n):
    A = rng.standard_normal((n, n))
    M = 0.5 * np.eye(n) + A @ A.T / n
    return np.array([M[i, j] if i == j else M[i, j] * np.sqrt(2)
                     for j in range(n) for i in range(j + 1)])


def svec_eye(sides, value):
    return np.concatenate([[value if i == j else 0.0 for j in range(n) for i in range(j + 1)]
                           for n in sides])


@pytest.mark.parametrize("name", list(SIDES))
def test_psd_sides(cuda_device, name):
    sides = SIDES[name]
    specs = [(5, n, 0.0) for n in sides]
    rng = np.random.default_rng(len(sides))
    s = np.concatenate([interior(rng, n) for n in sides])
    z = np.concatenate([interior(rng, n) for n in sides])
    C, G = oracle.Cones(specs), GPUCones(specs)
    d_s, d_z = G.dev(s), G.dev(z)
    assert C.update_scaling(s, z, 1.0, 0) == 0
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_z.data_ptr(), 1.0, 0, None) == 0
    hs = G.empty(G.hs_len)
    assert G.L.clgpu_get_Hs(G.h, hs.data_ptr(), None) == 0
    assert close(hs.cpu().numpy()[:C.hs_len], C.get_Hs(), 1e-11)
    out = G.empty(C.numel)
    stz, sts = rng.standard_normal(C.numel) * 0.1, rng.standard_normal(C.numel) * 0.1
    d_stz, d_sts = G.dev(stz), G.dev(sts)
    assert G.L.clgpu_combined_ds_shift(G.h, out.data_ptr(), d_stz.data_ptr(),
                                       d_sts.data_ptr(), d_z.data_ptr(), 0.37, None) == 0
    assert close(out.cpu().numpy(), C.combined_ds_shift(stz, sts, z, 0.37), 1e-10)
    steps = [(rng.standard_normal(C.numel) * k, rng.standard_normal(C.numel) * k)
             for k in (0.5, 2.0, 1e-3)]
    steps.append((-2.0 * s, svec_eye(sides, 0.5)))  # direction along s: clustered eigenvalues
    steps.append((np.zeros(C.numel), -3.0 * z))
    steps.append((np.zeros(C.numel), np.zeros(C.numel)))
    for dz, ds in steps:
        ref = C.step_length(dz, ds, z, s, 1.0)
        a = ctypes.c_double()
        d_dz, d_ds = G.dev(dz), G.dev(ds)
        assert G.L.clgpu_step_length(G.h, d_dz.data_ptr(), d_ds.data_ptr(), d_z.data_ptr(),
                                     d_s.data_ptr(), 1.0, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                     None) == 0
        assert abs(a.value - ref) <= 1e-10 * max(1.0, ref), (a.value, ref)


# both sides of the lines between the products' and the step lengths' kernels
LINES = {"two_many": [2, 1] * 40, "six": [6, 4] * 9, "seven": [7] * 33, "eight_2000": [8] * 2000,
         "eight_2001": [8, 3, 5] * 667, "nine": [9, 2] * 17}


@pytest.mark.parametrize("name", list(LINES))
def test_psd_sides_at_the_lines(cuda_device, name):
    SIDES[name] = LINES[name]
    test_psd_sides(cuda_device, name)


@pytest.mark.parametrize("n", [1, 8, 16])
def test_psd_repeated_eigenvalues(cuda_device, n):
    """s = z = I: the scaling is the identity and every eigenvalue of the step's
    matrix is the same, or all but one are."""
    specs = [(5, n, 0.0)] * 3
    s = svec_eye([n] * 3, 1.0)
    C, G = oracle.Cones(specs), GPUCones(specs)
    d_s = G.dev(s)
    assert C.update_scaling(s, s, 1.0, 0) == 0
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_s.data_ptr(), 1.0, 0, None) == 0
    v = np.ones(n) / np.sqrt(n)
    rank1 = -4.0 * np.outer(v, v)
    m = n * (n + 1) // 2
    low = np.array([rank1[i, j] * (1.0 if i == j else np.sqrt(2))
                    for j in range(n) for i in range(j + 1)])
    for ds in (-4.0 * s, np.concatenate([low, 0 * low, -low]), np.concatenate([-s[:2 * m], low])):
        a = ctypes.c_double()
        d_ds = G.dev(ds)
        assert G.L.clgpu_step_length(G.h, d_ds.data_ptr(), d_ds.data_ptr(), d_s.data_ptr(),
                                     d_s.data_ptr(), 1.0, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                     None) == 0
        ref = C.step_length(ds, ds, s, s, 1.0)
        assert abs(a.value - ref) <= 1e-12 * n, (a.value, ref)


def test_psd_scaling_failure_small_side(cuda_device):
    specs = [(5, 4, 0.0)] * 9
    s = svec_eye([4] * 9, 1.0)
    bad = s.copy()
    bad[7 * 10] = -1.0
    G = GPUCones(specs)
    d_s, d_b = G.dev(s), G.dev(bad)
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_s.data_ptr(), 1.0, 0, None) == 0
    assert G.L.clgpu_update_scaling(G.h, d_b.data_ptr(), d_s.data_ptr(), 1.0, 0, None) != 0
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_b.data_ptr(), 1.0, 0, None) != 0


@pytest.mark.parametrize("sides", [[0, 0], [0, 3, 0, 5], [0, 17]])
def test_psd_empty_cones_set_no_limit(cuda_device, sides):
    """A cone of side 0 has no eigenvalue and limits no step, alone, beside
    small cones and beside large ones."""
    specs = [(5, n, 0.0) for n in sides]
    G = GPUCones(specs)
    s = svec_eye(sides, 1.0)
    d_s, d_d = G.dev(np.append(s, 0.0)), G.dev(np.append(-0.5 * s, 0.0))
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_s.data_ptr(), 1.0, 0, None) == 0
    for _ in range(3):
        a = ctypes.c_double()
        assert G.L.clgpu_step_length(G.h, d_d.data_ptr(), d_d.data_ptr(), d_s.data_ptr(),
                                     d_s.data_ptr(), 5.0, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                     None) == 0
        # the other cones' step to the boundary is 2
        assert a.value == pytest.approx(2.0 if max(sides) else 5.0, rel=1e-12)


@pytest.mark.parametrize("n", [4, 16])
@pytest.mark.parametrize("coupling", [3e-155, 1e-158, 1e-161, 1e-170, 1e-320, 0.25])
@pytest.mark.parametrize("scale", [1.0, 1e-300, 1e-150, 1e155, 1e250])
def test_psd_step_at_the_ends_of_the_range(cuda_device, n, coupling, scale):
    """s = z = I, so the step's matrix is the direction itself: rows whose squares
    leave FP64's range, beside entries of order one and alone.  The eigenvalue's
    error is at most about n^1.5 eps |A|, and |A| is of its own order: far below
    the 1e-12 asked for."""
    G = GPUCones([(5, n, 0.0)] * 3)
    s = svec_eye([n] * 3, 1.0)
    d_s = G.dev(s)
    assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_s.data_ptr(), 1.0, 0, None) == 0
    M = np.full((n, n), coupling) * np.sign(np.sin(np.add.outer(np.arange(n), np.arange(n)) + 1.0))
    M[np.diag_indices(n)] = np.resize([-4.0, -1.0, 2.0, 3.0], n)
    low = np.linalg.eigvalsh(M)[0]
    v = np.array([M[i, j] * (1.0 if i == j else np.sqrt(2))
                  for j in range(n) for i in range(j + 1)]) * scale
    for ds in (np.concatenate([0 * v, v, 0 * v]), np.concatenate([-v[:1] * np.abs(s[:len(v)]), v, v])):
        a = ctypes.c_double()
        d_d, zero = G.dev(ds), G.dev(0 * ds)
        assert G.L.clgpu_step_length(G.h, d_d.data_ptr(), zero.data_ptr(), d_s.data_ptr(),
                                     d_s.data_ptr(), 1e305, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                     None) == 0
        assert a.value == pytest.approx(1.0 / (-low * scale), rel=1e-12, abs=0)


def test_psd_step_of_directions_that_are_not_finite(cuda_device):
    """As the iteration of the larger sides answers: a NaN sets no limit, an
    infinite direction of a 1 x 1 cone a step of zero."""
    for n, value, want in ((5, np.nan, 1.0), (1, -np.inf, 0.0), (1, np.inf, 1.0)):
        G = GPUCones([(5, n, 0.0)])
        d_s = G.dev(svec_eye([n], 1.0))
        d_d, zero = G.dev(np.full(n * (n + 1) // 2, value)), G.dev(np.zeros(n * (n + 1) // 2))
        assert G.L.clgpu_update_scaling(G.h, d_s.data_ptr(), d_s.data_ptr(), 1.0, 0, None) == 0
        a = ctypes.c_double()
        assert G.L.clgpu_step_length(G.h, d_d.data_ptr(), zero.data_ptr(), d_s.data_ptr(),
                                     d_s.data_ptr(), 1.0, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                     None) == 0
        assert a.value == want, (n, value, a.value)


@pytest.mark.parametrize("others", [[20], [17, 1], [8] * 2100, [2, 9, 16]])
def test_psd_results_do_not_depend_on_the_other_cones(cuda_device, others):
    """Bit for bit, with cones beside them that take other kernels: larger sides,
    and so many that the products go the other way."""
    sides = [3, 8, 2, 7, 16, 1, 9, 6]
    rng = np.random.default_rng(5)
    s, z = (np.concatenate([interior(rng, n) for n in sides]) for _ in range(2))
    so, zo = (np.concatenate([interior(rng, n) for n in others]) for _ in range(2))
    d1, d2 = (rng.standard_normal(len(s)) for _ in range(2))
    do = np.zeros(len(so))
    res = []
    for extra in (False, True):
        specs = [(5, n, 0.0) for n in sides + (others if extra else [])]
        cat = lambda a, b: np.concatenate([a, b]) if extra else a  # noqa: E731
        G = GPUCones(specs)
        ds, dz, a1, a2 = (G.dev(v) for v in (cat(s, so), cat(z, zo), cat(d1, do), cat(d2, do)))
        L, st = G.L, None
        assert L.clgpu_update_scaling(G.h, ds.data_ptr(), dz.data_ptr(), 1.0, 0, st) == 0
        out = []
        o = G.empty(len(cat(s, so)))
        assert L.clgpu_mul_Hs(G.h, o.data_ptr(), a1.data_ptr(), st) == 0
        out.append(o.cpu().numpy()[:len(s)].copy())
        assert L.clgpu_combined_ds_shift(G.h, o.data_ptr(), a1.data_ptr(), a2.data_ptr(),
                                         dz.data_ptr(), 0.37, st) == 0
        out.append(o.cpu().numpy()[:len(s)].copy())
        assert L.clgpu_ds_from_dz_offset(G.h, o.data_ptr(), a2.data_ptr(), dz.data_ptr(), st) == 0
        out.append(o.cpu().numpy()[:len(s)].copy())
        for k in (0.1, 3.0):
            b1, b2 = G.dev(k * cat(d1, do)), G.dev(k * cat(d2, do))
            a = ctypes.c_double()
            assert L.clgpu_step_length(G.h, b1.data_ptr(), b2.data_ptr(), dz.data_ptr(),
                                       ds.data_ptr(), 1.0, 0.99, 0.8, 1e-4, ctypes.byref(a),
                                       st) == 0
            out.append(np.array([a.value]))
        res.append(out)
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_psd_programs_give_the_bits_of_each_alone(cuda_device):
    from cuclarabel_b200 import BatchSolver, problems
    pbs = [problems.psd_lp(n, 2, seed=n) for n in (2, 3, 8, 9, 16, 18)]
    for pb, s in zip(pbs, BatchSolver(pbs, max_iter=5).solve()):
        a = BatchSolver([pb], max_iter=5).solve()[0]
        assert np.array_equal(a.x, s.x) and np.array_equal(a.s, s.s) and np.array_equal(a.z, s.z)
