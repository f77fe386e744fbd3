"""The eliminated phasor system against a node-by-node elimination of the
joined matrix, as the reference does it (em3d_tet10.py:332-356): which sets
hold, which wins where they overlap, complex values, no boundary at all. Same
entries; the right-hand sides differ by the order of a few hundred sums:
1e-13 of the largest term."""

import types

import numpy as np
import pytest
import scipy.sparse as sp

from cloudfem_b200.physics import em3d_tet10 as em

SETS = {"left": np.array([0, 1, 2, 5]), "top": np.array([2, 9, 5]), "none": np.zeros(0, dtype=int)}


@pytest.mark.parametrize("B", [None, (0.1, -0.2, 0.3)])
@pytest.mark.parametrize("boundary,a_bc", [
    (None, None),
    ("left", {"top": (1.0, 2.0j, 3.0 - 1.0j)}),
    (["top", "left"], {"left": lambda x, y, z: (x, y * 1j, z), "top": (0.0, 0.0, 1.0)}),
    (np.array([7, 7, 3]), None),
    ("none", None),
])
def test_eliminated_system(B, boundary, a_bc):
    rng = np.random.default_rng(3)
    n, n_v, w = 11, 6, 50.0
    mesh = types.SimpleNamespace(n_nodes=n, nodes=rng.random((n, 3)), boundaries=SETS)
    K = sp.random(3 * n, 3 * n, 0.3, "csr", random_state=1)
    M = sp.random(3 * n, 3 * n, 0.1, "csr", random_state=2)
    G = sp.random(3 * n, n_v, 0.4, "csr", random_state=4)
    S = sp.random(n_v, n_v, 0.5, "csr", random_state=5)
    rhs = rng.random(3 * n + n_v) + 1j * rng.random(3 * n + n_v)
    A = sp.bmat([[K + 1j * w * M, G], [G.T, S / (1j * w)]], format="csr")
    fixed = {}
    names = ["left", "top", "none"] if boundary is None else boundary
    names = [names] if isinstance(names, str) else names
    nodes = [p for k in names for p in (SETS[k] if isinstance(k, str) else [k])]
    for p in nodes:
        val = 0.5 * np.cross(B, mesh.nodes[p]) if B is not None else np.zeros(3)
        fixed.update({3 * p + m: val[m] for m in range(3)})
    for name, v in (a_bc or {}).items():
        for p in SETS[name]:
            vv = v(*mesh.nodes[p]) if callable(v) else v
            fixed.update({3 * p + m: vv[m] for m in range(3)})
    idx = np.array(sorted(fixed), dtype=int)
    val = np.array([fixed[i] for i in idx], dtype=complex)
    keep = np.ones(3 * n + n_v, dtype=bool)
    keep[idx] = False
    ref = rhs - (A[:, idx] @ val if len(idx) else 0.0)
    A2, b2, keep2, idx2, val2 = em._eliminated(mesh, K, M, G, S, w, rhs.copy(), B, boundary, a_bc)
    assert np.array_equal(keep, keep2) and np.array_equal(idx, idx2) and np.array_equal(val, val2)
    E = (A[keep][:, keep] - A2).tocoo()
    assert E.nnz == 0 or np.abs(E.data).max() <= 1e-15 * np.abs(A.data).max()
    assert np.abs(b2 - ref[keep]).max() <= 1e-13 * (np.abs(A.data).max() + np.abs(rhs).max())


def test_faces_are_not_nodes():
    mesh = types.SimpleNamespace(n_nodes=4, nodes=np.zeros((4, 3)), boundaries={})
    Z = sp.csr_matrix((12, 12))
    with pytest.raises(TypeError):
        em._eliminated(mesh, Z, Z, sp.csr_matrix((12, 1)), sp.csr_matrix((1, 1)), 1.0,
                       np.zeros(13, dtype=complex), None, np.zeros((4, 3), dtype=int), None)
