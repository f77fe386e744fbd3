"""Which path a solve takes, by the launches it makes: a comparison with another
scheduler says nothing where both took the same one. A resident solve is five
launches (rows to blocks, row orders, columns, values, the solve), the graphs
hundreds, one launch over the CSR arrays a few others. Systems are those of
test_gpu_resident.py."""

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_coarse_limits import _timed
from test_gpu_resident import SHAPES, _block_system, _system

pytestmark = pytest.mark.gpu

RESIDENT = 5
DEALT = 11       # + order (2), copies of pattern, values and vectors (3), solution back
COARSE = 14      # + order (3), copies (2), geometry, coarse matrix, its inverse, solution back


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _launches(rt, systems, md, rtol, max_iter=2000):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    if md == N.SOLVE_MIXED:
        for s in systems:
            s.ensure_fp32()
    before = rt.launches()
    for r in pcg(systems, md, rtol, max_iter):
        assert r.status == N.CFEM_OK
    return rt.launches() - before


@pytest.mark.parametrize("bs", [1, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("n,kind", SHAPES)
def test_one_system(torch, n, kind, mode, bs):
    """Resident but for 3x3 rows of fewer than 20 blocks in mixed precision and for
    a scattered pattern whose 3x3 halo is past shared memory."""
    from cloudfem_b200 import _native as N
    if bs == 3 and kind == "band" and n > 50000:
        n = 50001
    rt = N.runtime()
    md, rtol = (N.SOLVE_FP64, 1e-13) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10)
    data = _system(n, bs, kind, 1000 * bs + n)
    got = _launches(rt, [_block_system(torch, rt, data, bs)], md, rtol)
    short = bs == 3 and mode == "mixed" and data[3][-1] < 20 * n
    wide_halo = bs == 3 and kind == "scatter" and n == 100000
    assert (got == RESIDENT) == (not short and not wide_halo), got


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_batches(torch, mode):
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    md, rtol = (N.SOLVE_FP64, 1e-13) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10)
    for kind, sizes, dealt in (("wide", [40, 500, 3000, 9000] * 12, True), ("wide", [2000] * 148, True),
                               ("wide", [2000] * 149, False), ("scatter", [60000] * 6 + [9000] * 24, False)):
        datas = {n: _system(n, 1, kind, n) for n in set(sizes)}
        got = _launches(rt, [_block_system(torch, rt, datas[n], 1) for n in sizes], md, rtol)
        assert got == DEALT if dealt else got > 5 * DEALT, (kind, len(sizes), got)
    datas = [_system(n, 1, "wide", n) for n in (70, 9000, 700, 30000)]
    got = _launches(rt, [_block_system(torch, rt, d, 1) for d in datas], md, rtol)
    assert RESIDENT < got <= RESIDENT + 3        # whole systems, up to four launches


@pytest.mark.parametrize("cells,tet10", [((3, 3, 3), True), ((12, 9, 8), True), ((40, 6, 1), True),
                                         ((14, 9, 8), False), ((200, 1, 1), False)])
def test_elasticity_with_nodes(torch, cells, tet10):
    """With the part's coordinates the corrected solve, in fewer iterations than
    the plain one; with NaN coordinates the plain one after it."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import DeviceMesh
    from cloudfem_b200.mesh import box_mesh, box_mesh_tet10
    m = (box_mesh_tet10 if tet10 else box_mesh)(*cells, xlim=(0.0, cells[0]), ylim=(0.0, cells[1]),
                                                zlim=(0.0, cells[2]))
    dm = DeviceMesh(m)
    vals, _ = dm.assemble_elastic(N.OP_T10_ELAST if tet10 else N.OP_P1_ELAST, 200.0, 0.3)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dm.rt.device)  # noqa: E731
    mask = up(np.repeat(np.asarray(m.nodes)[:, 0] < 1e-9, 3).astype(np.uint8))
    b = up(np.random.default_rng(3).uniform(-1.0, 1.0, 3 * dm.n_nodes))
    res = {}
    for name, nodes in (("plain", None), ("true", dm.nodes), ("nan", torch.full_like(dm.nodes, float("nan")))):
        r, _, launches = _timed(torch, dm, vals, b, mask, 1e-10, 20000, nodes, repeats=1)
        assert r.status == N.CFEM_OK
        res[name] = (r.iterations, launches)
    assert res["plain"][1] == RESIDENT
    assert res["true"][1] == COARSE and res["true"][0] < res["plain"][0]
    assert res["nan"] == (res["plain"][0], COARSE - 1 + RESIDENT)


@pytest.mark.parametrize("n,kind", [(1, "band"), (700, "arrow"), (9000, "band"), (4000, "scatter"),
                                    (120000, "band")])
def test_complex_system(torch, n, kind):
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    A = (_system(n, 1, kind, 7 * n + 1)[0] + 1j * sp.identity(n)).tocsr()
    A.sort_indices()
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rt.device)  # noqa: E731
    d = [up(A.indptr.astype(np.int32)), up(A.indices.astype(np.int32)), up(A.data.view(np.float64)),
         up(np.ones(n, dtype=complex).view(np.float64))]
    x = torch.zeros(2 * n, dtype=torch.float64, device=rt.device)
    st = N.SolveStats()
    before = rt.launches()
    N.check(rt.lib.cfem_cocg_solve(rt.ctx, n, *[N.ptr(a) for a in d], N.ptr(x), 1e-12, 2000,
                                   ctypes.byref(st), rt.stream()))
    assert st.status == N.CFEM_OK
    assert rt.launches() - before == RESIDENT
