"""Blocked fronts of the supernodal LDL^T at the widths where their kernels can
go wrong: pivot blocks and update regions below, at and above one 128-column
panel, first panels of one to seven 16-column units, several panels in a chain,
and fronts whose solve waits for children.  The systems are diagonally dominant
(condition below 1e3), so factor and refined solution are good to 1e-12; the
bound here is 1e-9 of the solution."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from cuclarabel_b200 import Settings, _lib

pytestmark = pytest.mark.gpu

# widths of two coupled dense blocks and of the root block both touch
FRONTS = [(130, 130, 16), (145, 17, 129), (200, 300, 257), (129, 640, 100), (260, 131, 400),
          (20, 150, 1030)]


def system(rng, widths, n=6400):
    """Dense blocks A, B (not coupled) and C (coupled to both), and single
    columns that each touch up to three entries of one block."""
    a, b, c = widths
    k = a + b + c
    lo = [0, a, a + b, k]
    rows, cols = [], []
    for i, j in ((0, 0), (1, 1), (2, 2), (0, 2), (1, 2)):
        r, q = np.meshgrid(np.arange(lo[i], lo[i + 1]), np.arange(lo[j], lo[j + 1]))
        rows.append(r.ravel())
        cols.append(q.ravel())
    for t in range(k, n):
        blk = rng.integers(3)
        q = rng.integers(lo[blk], lo[blk + 1], 3)
        rows.append(np.full(3, t))
        cols.append(q)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    K = sp.coo_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(n, n)).tocsr()
    K = K + K.T
    K.setdiag(0)
    signs = np.where(rng.random(n) < 0.5, 1, -1).astype(np.int8)
    K = (K + sp.diags(signs * (np.abs(K).sum(1).A1 if hasattr(np.abs(K).sum(1), "A1")
                               else np.asarray(np.abs(K).sum(1)).ravel()) * 1.1 + signs)).tocsr()
    K.sort_indices()
    p = rng.permutation(n)
    K = K[p][:, p].tocsr()
    K.sort_indices()
    return K, signs[p]


@pytest.mark.parametrize("widths", FRONTS)
@pytest.mark.parametrize("mixed", [0, 1])
def test_blocked_fronts(cuda_device, widths, mixed):
    import torch
    rng = np.random.default_rng(sum(widths))
    K, signs = system(rng, widths)
    L, h = _lib.load(), ctypes.c_void_p()
    Kp, Kj = K.indptr.astype(np.int32), K.indices.astype(np.int32)
    st = Settings()
    if mixed:
        st.direct_solve_method = "cudssmixed"
    cs = st.to_c()
    assert L.clgpu_ldl_create(K.shape[0], Kp.ctypes.data_as(_lib.ip), Kj.ctypes.data_as(_lib.ip),
                              signs.ctypes.data_as(ctypes.POINTER(ctypes.c_byte)),
                              ctypes.byref(cs), ctypes.byref(h)) == 0
    try:
        Kx = torch.from_numpy(K.data).cuda()
        for trial in range(3):
            x = rng.standard_normal(K.shape[0])
            b = torch.from_numpy(K @ x).cuda()
            out = torch.zeros_like(b)
            eps = ctypes.c_double()
            if trial < 2:  # the third solve reuses the factor
                assert L.clgpu_ldl_refactor(h, ctypes.c_void_p(Kx.data_ptr()), ctypes.byref(eps),
                                            None) == 0
            assert L.clgpu_ldl_solve(h, ctypes.c_void_p(b.data_ptr()),
                                     ctypes.c_void_p(out.data_ptr()), None) == 0
            assert np.abs(out.cpu().numpy() - x).max() <= 1e-9 * np.abs(x).max()
    finally:
        L.clgpu_ldl_destroy(h)
