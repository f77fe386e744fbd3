"""Every bounded wait of the cooperative launches, run out on purpose by
CFEM_PARAM_BARRIER_HOLD with a short limit: the launch returns, the host reads
CFEM_ERR_TIMEOUT, and the same context then solves as before. The resident CG's
wait is in test_gpu_failures.py; here the two-level barrier of the launch over
CSR arrays (block Jacobi keeps it), the complex solver's sums and the flags of
the coarse inverse."""

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_resident import _block_system, _system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


@pytest.fixture
def rt(torch):
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    yield rt
    rt.set_param(N.PARAM_BARRIER_HOLD, 0)
    rt.set_param(N.PARAM_BARRIER_TIMEOUT_US, 4000000)
    N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_AUTO))


def _timeout_then_same(rt, solve):
    from cloudfem_b200 import _native as N
    want = solve()
    rt.set_param(N.PARAM_BARRIER_TIMEOUT_US, 20000)
    rt.set_param(N.PARAM_BARRIER_HOLD, 1)
    with pytest.raises(N.CfemError) as info:
        solve()
    assert info.value.status == N.CFEM_ERR_TIMEOUT
    rt.set_param(N.PARAM_BARRIER_HOLD, 0)
    rt.set_param(N.PARAM_BARRIER_TIMEOUT_US, 4000000)
    assert np.array_equal(solve(), want)


@pytest.mark.parametrize("noalloc", [False, True])
def test_grid_barrier_of_the_csr_launch(torch, rt, noalloc):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg, pcg_noalloc
    data = _system(800, 3, "wide", 1)
    N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_PERSISTENT))

    def solve():
        s = _block_system(torch, rt, data, 3)
        s.precond = N.PRECOND_BLOCK
        r = pcg_noalloc(s, N.SOLVE_FP64, 1e-13, 2000) if noalloc else pcg([s], N.SOLVE_FP64, 1e-13, 2000)[0]
        assert r.status == N.CFEM_OK
        return s.x.cpu().numpy()

    _timeout_then_same(rt, solve)


def test_sums_of_the_complex_solver(torch, rt):
    from cloudfem_b200 import _native as N
    n = 4000
    A = (_system(n, 1, "wide", 5)[0] + 1j * sp.identity(n)).tocsr()
    A.sort_indices()
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rt.device)  # noqa: E731
    ip, ix = up(A.indptr.astype(np.int32)), up(A.indices.astype(np.int32))
    va, vb = up(A.data.view(np.float64)), up(np.ones(n, dtype=complex).view(np.float64))

    def solve():
        x = torch.zeros(2 * n, dtype=torch.float64, device=rt.device)
        st = N.SolveStats()
        N.check(rt.lib.cfem_cocg_solve(rt.ctx, n, N.ptr(ip), N.ptr(ix), N.ptr(va), N.ptr(vb), N.ptr(x),
                                       1e-12, 2000, ctypes.byref(st), rt.stream()))
        assert st.status == N.CFEM_OK
        return x.cpu().numpy()

    _timeout_then_same(rt, solve)


def test_flags_of_the_coarse_inverse(torch, rt):
    """About 28 pieces, 14 pivot blocks: all but the first wait for a flag."""
    from cloudfem_b200.mesh import box_mesh_tet10
    from cloudfem_b200.physics.elastic_tet10 import solve_elasticity_tet10
    m = box_mesh_tet10(6, 4, 4)

    def solve():
        return np.stack(solve_elasticity_tet10(m, 1.0, 0.3, bc={"xmin": (0.0, 0.0, 0.0)},
                                               traction={"xmax": (0.0, 0.0, -1.0)}))

    _timeout_then_same(rt, solve)
