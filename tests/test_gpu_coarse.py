"""Elasticity solves with the coarse correction on rigid-body modes
(cfem_pcg_solve_nodes) against SciPy's residual and the plain solve: few
pieces and all of them, thin parts whose pieces are flat or nearly on a line,
pieces without a free DOF, numberings that scatter the pieces, coordinates
that say nothing or are not numbers (the answer may not depend on them).

Tolerances: a solve to rtol ends on the FP64 true residual of A x = b on the
free DOFs, so SciPy's residual is at most rtol times the norm of the lifted
load (or at the solver's round-off floor, 16 eps of |A| |x|), plus what
evaluating it rounds: (entries of a row + 2) eps of |A| |x| + |b|. 1 % is added for the norms' own rounding.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
FLOOR = 16     # a residual this many eps of its terms counts as the round-off floor


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _solve(torch, dm, vals, rhs, x0, mask, mode, rtol, nodes):
    from cloudfem_b200.device import BlockSystem, pcg
    x = torch.from_numpy(x0).to(dm.rt.device)
    pat = dm.pattern
    s = BlockSystem(dm.rt, dm.n_nodes, 3, pat.row_ptr, pat.col, vals, rhs, x, mask, nodes=nodes)
    r = pcg([s], mode, rtol, 20000)[0]
    return x.cpu().numpy(), r


CASES = [
    (True, (3, 3, 3), "face", "true"),        # 343 nodes, a few pieces
    (True, (20, 4, 4), "face", "true"),       # every SM a piece, halos between many
    (True, (40, 6, 1), "face", "true"),       # flat pieces
    (True, (12, 9, 8), "half", "true"),       # pieces without a free DOF
    (True, (9, 9, 9), "face", "shuffled"),    # pieces scattered over the part
    (True, (9, 9, 9), "face", "zero"),        # one point: rotations vanish
    (True, (9, 9, 9), "face", "nan"),         # no correction possible
    (False, (14, 9, 8), "face", "true"),      # P1 rows of 15
    (False, (200, 1, 1), "face", "true"),     # a rod of one cell's section
    (False, (10, 10, 10), "some", "true"),    # single DOFs fixed, values given
]


# (P1 elasticity in mixed precision has no correction)
@pytest.mark.parametrize("mode,tet10,cells,fix,nodes_as",
                         [(m,) + c for m in ("fp64", "mixed") for c in CASES if m == "fp64" or c[0]])
def test_coarse_correction(torch, mode, tet10, cells, fix, nodes_as):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import DeviceMesh
    from cloudfem_b200.mesh import tet10_mesh, tet_mesh
    make = tet10_mesh.box_mesh_tet10 if tet10 else tet_mesh.box_mesh
    mesh = make(*cells, xlim=(0.0, 0.1 * cells[0]), ylim=(0.0, 0.1 * cells[1]), zlim=(0.0, 0.1 * cells[2]))
    rng = np.random.default_rng(5)
    dm = DeviceMesh(mesh)
    n = dm.n_nodes
    vals, _ = dm.assemble_elastic(N.OP_T10_ELAST if tet10 else N.OP_P1_ELAST, 200.0, 0.3)
    A = dm.pattern.to_scipy(3, vals).tocsr()
    b = rng.uniform(-1.0, 1.0, 3 * n)
    x0 = np.zeros(3 * n)
    nodes = np.asarray(mesh.nodes, float)
    mask = np.zeros(3 * n, bool)
    if fix == "face":
        mask[:] = np.repeat(nodes[:, 0] < 1e-9, 3)
    elif fix == "half":
        mask[:] = np.repeat(nodes[:, 0] < 0.05 * cells[0] + 1e-9, 3)
    else:
        mask[:] = rng.random(3 * n) < 0.1
    x0[mask] = rng.uniform(-1e-3, 1e-3, mask.sum())
    if nodes_as == "shuffled":
        nodes = nodes[rng.permutation(n)]
    elif nodes_as == "zero":
        nodes = np.zeros_like(nodes)
    elif nodes_as == "nan":
        nodes = np.full_like(nodes, np.nan)
    dev = dm.rt.device
    d_rhs, d_mask = torch.from_numpy(b).to(dev), torch.from_numpy(mask.astype(np.uint8)).to(dev)
    rtol = 1e-10 if mode == "fp64" else 1e-7
    solve_mode = N.SOLVE_FP64 if mode == "fp64" else N.SOLVE_MIXED
    d_nodes = torch.from_numpy(np.ascontiguousarray(nodes)).to(dev)
    x, r = _solve(torch, dm, vals, d_rhs, x0, d_mask, solve_mode, rtol, d_nodes)
    _, rp = _solve(torch, dm, vals, d_rhs, x0, d_mask, solve_mode, rtol, None)
    assert r.status == 0
    assert np.array_equal(x[mask], x0[mask])
    f = ~mask
    lifted = np.linalg.norm((b - A @ x0)[f])
    width = np.diff(A.indptr).max() + 2
    terms = np.linalg.norm((abs(A) @ abs(x) + abs(b))[f])
    assert np.linalg.norm((b - A @ x)[f]) <= 1.01 * rtol * lifted + (width + FLOOR) * EPS * terms
    again, _ = _solve(torch, dm, vals, d_rhs, x0, d_mask, solve_mode, rtol, d_nodes)
    assert np.array_equal(x, again)
    if nodes_as == "true" and fix == "face" and tet10 and cells[0] >= 20:
        assert 3 * r.iterations < rp.iterations  # the correction was applied
