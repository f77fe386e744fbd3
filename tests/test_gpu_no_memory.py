"""A resident plan that finds no device memory for one of its parts
(CFEM_PARAM_ALLOC_FAIL makes its n-th allocation fail): the system is solved by
the scheduler that had it before, and nothing stays allocated. Systems and
tolerances are those of test_gpu_resident.py."""

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
    rt.set_param(N.PARAM_ALLOC_FAIL, 0)


def _solves(rt, solve, parts):
    """solve() with every part failing in turn, then with none: the launches and
    the answer of each."""
    from cloudfem_b200 import _native as N
    out = []
    idle = rt.trim(0)
    for n in list(range(1, parts + 2)) + [0]:
        rt.set_param(N.PARAM_ALLOC_FAIL, n)
        before = rt.launches()
        x = solve()
        out.append((rt.launches() - before, x))
        rt.set_param(N.PARAM_ALLOC_FAIL, 0)
        assert rt.trim(0) <= idle, n
    return out


def _check(out, tol):
    """Every failing part was one of the plan's (another number of launches than
    without: the five launches of a resident solve, the graphs' hundreds), the one
    past the last is not."""
    x = out[-1][1]
    for launches, y in out[:-2]:
        assert launches != out[-1][0]
        assert np.linalg.norm(y - x) <= 2 * tol * np.linalg.norm(x)
    assert out[-2][0] == out[-1][0] and np.array_equal(out[-2][1], x)


@pytest.mark.parametrize("mode,rtol,tol", [("FP64", 1e-13, 1e-12), ("MIXED", 1e-10, 1e-9)])
def test_one_system_and_a_dealt_batch(torch, rt, mode, rtol, tol):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    for kind, sizes, parts in ("band", [120000], 4), ("wide", [40, 500, 3000, 9000] * 12, 6):
        datas = {n: _system(n, 1, kind, n) for n in set(sizes)}

        def solve():
            systems = [_block_system(torch, rt, datas[n], 1) for n in sizes]
            for r in pcg(systems, getattr(N, "SOLVE_" + mode), rtol, 2000):
                assert r.status == N.CFEM_OK
            return torch.cat([s.x for s in systems]).cpu().numpy()

        solve()
        _check(_solves(rt, solve, parts), tol)


def test_elasticity_with_nodes(torch, rt):
    """The coarse correction's three allocations, then the resident plan's four;
    the plain solve after a failure meets the same failure (only its plan's four)."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.mesh import box_mesh_tet10
    from cloudfem_b200.physics.elastic_tet10 import solve_elasticity_tet10
    m = box_mesh_tet10(6, 4, 4)

    def solve():
        return np.stack(solve_elasticity_tet10(m, 1.0, 0.3, bc={"xmin": (0.0, 0.0, 0.0)},
                                               traction={"xmax": (0.0, 0.0, -1.0)}))

    solve()
    _check(_solves(rt, solve, 7), 1e-9)


@pytest.mark.parametrize("mode,rtol,tol", [("FP64", 1e-13, 1e-12), ("MIXED", 1e-10, 1e-9)])
def test_slots(torch, rt, mode, rtol, tol):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import SlotEngine
    data = _system(4000, 1, "wide", 3)

    def solve():
        eng = SlotEngine(rt, 2, 1, getattr(N, "SOLVE_" + mode), 4000, 4000 * 30)
        system = _block_system(torch, rt, data, 1)
        eng.assign(system, rtol, 2000)
        for _ in range(200):
            eng.run(1)
            done = eng.poll()
            if done:
                break
        assert done[0][2].status == N.CFEM_OK
        eng.close()
        return system.x.cpu().numpy()

    solve()
    _check(_solves(rt, solve, 4), tol)


def test_complex_system(torch, rt):
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

    solve()
    _check(_solves(rt, solve, 4), 1e-10)
