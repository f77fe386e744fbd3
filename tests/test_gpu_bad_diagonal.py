"""A row without a diagonal entry ends a resident solve with a breakdown
whatever else the first residual holds, and the statistics of that solve are
those of the right-hand side."""

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _up(torch, rt, a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(rt.device)


@pytest.mark.parametrize("n", [5, 4000, 60000])
def test_complex_system_reports_its_norm(torch, n):
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    A = sp.diags([np.full(n, 2.0 + 1j), np.full(n - 1, -0.5), np.full(n - 1, -0.5)], [0, 1, -1]).tolil()
    A[n // 2, n // 2] = 0.0
    A = A.tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    b = np.random.default_rng(n).uniform(-1.0, 1.0, n) + 0.5j
    x = torch.zeros(2 * n, dtype=torch.float64, device=rt.device)
    st = N.SolveStats()
    d = [_up(torch, rt, a) for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32),
                                     A.data.astype(complex).view(np.float64), b.view(np.float64))]
    N.check(rt.lib.cfem_cocg_solve(rt.ctx, n, *[N.ptr(a) for a in d], N.ptr(x), 1e-12, 100,
                                   ctypes.byref(st), rt.stream()))
    assert st.status == N.CFEM_ERR_BREAKDOWN and st.iterations == 0
    assert abs(st.bnorm - np.linalg.norm(b)) <= 1e-12 * np.linalg.norm(b)
    assert abs(st.relres - 1.0) <= 1e-12


@pytest.mark.parametrize("n", [64, 60000])
def test_breakdown_beside_an_overflowing_magnitude(torch, n):
    """Row 0's entry at a Dirichlet DOF is so large that the sum of magnitudes
    squared overflows, while its residual is that of the others."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import BlockSystem, pcg
    rt = N.runtime()
    A = sp.diags([np.full(n, 2.0), np.full(n - 1, -0.5), np.full(n - 1, -0.5)], [0, 1, -1]).tolil()
    A[0, 1] = A[1, 0] = 1e160
    A[n - 7, n - 7] = 0.0
    A = A.tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    b = np.ones(n)
    b[0] = 1e160
    x = np.zeros(n)
    x[1] = 1.0
    fixed = np.zeros(n, dtype=np.uint8)
    fixed[1] = 1
    s = BlockSystem(rt, n, 1, *[_up(torch, rt, a) for a in (A.indptr.astype(np.int32),
                                                            A.indices.astype(np.int32), A.data, b, x, fixed)])
    assert pcg([s], N.SOLVE_FP64, 1e-12, 500)[0].status == N.CFEM_ERR_BREAKDOWN
