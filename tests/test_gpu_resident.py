"""The resident scheduler (one cooperative launch, halo and matrix slices in
shared memory) against SciPy's direct solve and the graph scheduler, at the
sizes and shapes where its layout can go wrong: fewer rows than a slice, one
block and several, rows past a window, one very long row, matrices that do
and do not fit shared memory, patterns without a diagonal order, batches of
several launches.

Tolerances (2-norms): the off-diagonal part of every system is 0.8 times a
normalised adjacency, so its eigenvalues lie in [0.2, 2.8]. An FP64 answer at
the round-off floor is then within 1e-12 of the exact one, and a mixed answer
at a relative residual of 1e-10 within about ten times that, 1e-9.
"""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _pattern(n, kind, rng):
    """Symmetric node pattern (bool CSR, diagonal included)."""
    if kind == "band":
        d = [o for o in (1, 2, 7, 40) if o < n]
        P = sp.diags([np.ones(n - o) for o in d] + [np.ones(n)], d + [0], format="coo")
    elif kind == "wide":           # 21 and more entries per row (Tet10-like)
        P = sp.diags([np.ones(n - o) for o in range(min(12, n))], range(min(12, n)), format="coo")
    elif kind == "arrow":          # one row and column with every entry
        P = sp.coo_matrix((np.ones(n), (np.zeros(n, int), np.arange(n))), shape=(n, n))
        P = P + sp.identity(n) + sp.diags([np.ones(n - 1)], [1])
    else:                          # scattered: every block's halo is most of the rows
        m = 6 * n
        P = sp.coo_matrix((np.ones(m), (rng.integers(0, n, m), rng.integers(0, n, m))), shape=(n, n))
        P = P + sp.identity(n)
    P = (P + P.T).tocsr()
    P.data[:] = 1.0
    P.sort_indices()
    return P


def _system(n, bs, kind, seed):
    """SPD block system with off-diagonal sums at most 0.8 of the diagonal."""
    rng = np.random.default_rng(seed)
    P = _pattern(n, kind, rng)
    U = sp.triu(P, 1).tocoo()
    B = rng.uniform(-1.0, 1.0, (U.nnz, bs, bs))
    deg = np.diff(P.indptr)
    w = 1.0 / (bs * np.sqrt(deg[U.row] * deg[U.col]))
    B = 0.8 * B * w[:, None, None]
    rows = np.concatenate([U.row, U.col, np.arange(n)])
    cols = np.concatenate([U.col, U.row, np.arange(n)])
    D = np.broadcast_to(np.eye(bs), (n, bs, bs)) * rng.uniform(1.0, 2.0, (n, 1, 1))
    blocks = np.concatenate([B, B.transpose(0, 2, 1), D])
    order = np.lexsort((cols, rows))
    rows, cols, blocks = rows[order], cols[order], blocks[order]
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    A = sp.bsr_matrix((blocks, cols, indptr), shape=(n * bs, n * bs)).tocsr()
    b = rng.uniform(-1.0, 1.0, n * bs)
    fixed = rng.random(n * bs) < 0.1
    xd = np.where(fixed, rng.uniform(-1.0, 1.0, n * bs), 0.0)
    return A, blocks, cols.astype(np.int32), indptr.astype(np.int32), b, fixed, xd


def _exact(A, b, fixed, xd):
    x = xd.copy()
    f = ~fixed
    x[f] = spla.spsolve(A[f][:, f].tocsc(), b[f] - (A[f][:, fixed] @ xd[fixed]))
    return x


def _block_system(torch, rt, data, bs):
    from cloudfem_b200.device import BlockSystem
    A, blocks, cols, indptr, b, fixed, xd = data
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rt.device)  # noqa: E731
    return BlockSystem(rt, len(indptr) - 1, bs, up(indptr), up(cols), up(blocks.ravel()), up(b),
                       up(xd), up(fixed.astype(np.uint8)))


SHAPES = [(1, "band"), (31, "band"), (33, "band"), (300, "band"), (257, "arrow"), (2561, "band"),
          (6000, "arrow"), (5000, "scatter"), (40000, "band"), (150001, "band"), (100000, "scatter"),
          (9000, "wide"), (30000, "wide")]


@pytest.mark.parametrize("bs", [1, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("n,kind", SHAPES)
def test_matches_direct_and_graph(torch, n, kind, mode, bs):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    if bs == 3 and kind == "band" and n > 50000:
        n = 50001                  # 3x3 blocks: past shared memory at this size already
    rt = N.runtime()
    md, rtol, tol = ((N.SOLVE_FP64, 1e-15, 1e-12) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10, 1e-9))
    data = _system(n, bs, kind, 1000 * bs + n)
    out = []
    for sched in (N.SCHED_AUTO, N.SCHED_GRAPH):
        N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, sched))
        try:
            s = _block_system(torch, rt, data, bs)
            r = pcg([s], md, rtol, 2000)[0]
        finally:
            N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_AUTO))
        assert r.status == N.CFEM_OK, r
        out.append(s.x.cpu().numpy())
    fixed, xd = data[5], data[6]
    assert np.array_equal(out[0][fixed], xd[fixed])
    assert np.linalg.norm(out[0] - out[1]) <= 2 * tol * np.linalg.norm(out[1])
    if n <= 6000 and kind != "scatter":       # (a scattered pattern fills SuperLU's factors)
        x = _exact(data[0], data[4], fixed, xd)
        assert np.linalg.norm(out[0] - x) <= tol * np.linalg.norm(x)


@pytest.mark.parametrize("bs", [1, 3])
def test_batch_of_several_launches_equals_alone(torch, bs):
    """Systems of very different sizes, more blocks than one launch holds:
    each answer bitwise the one alone."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    rt = N.runtime()
    sizes = (70, 9000, 700, 30000)
    datas = [_system(n, bs, "wide", n + bs) for n in sizes]
    for mode, rtol in ((N.SOLVE_FP64, 1e-13), (N.SOLVE_MIXED, 1e-10)):
        systems = [_block_system(torch, rt, d, bs) for d in datas]
        rb = pcg(systems, mode, rtol, 2000)
        for s, d, r in zip(systems, datas, rb):
            alone = _block_system(torch, rt, d, bs)
            ra = pcg([alone], mode, rtol, 2000)[0]
            assert ra.status == N.CFEM_OK and ra.iterations == r.iterations
            assert torch.equal(alone.x, s.x)


@pytest.mark.parametrize("bs", [1, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,sizes", [
    ("wide", [40, 500, 3000, 9000] * 12),       # more blocks than four launches hold
    ("wide", [2000] * 148),                     # one block each on 148 SMs
    ("wide", [2000] * 149),                     # ... one system too many
    ("scatter", [60000] * 6 + [9000] * 24),     # columns that do not fit a block: not dealt
])
def test_batch_with_dealt_blocks(torch, kind, sizes, mode, bs):
    """A batch in one launch with the blocks dealt out, over copies of the
    systems in another row order: against the graph scheduler, then again
    after the values, loads and Dirichlet data changed (a plan's second
    solve must take all of them anew)."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import PcgPlan
    if bs == 3:
        sizes = [max(1, n // 3) for n in sizes]
    rt = N.runtime()
    md, rtol, tol = ((N.SOLVE_FP64, 1e-13, 1e-12) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10, 1e-9))
    made = {}
    for n in set(sizes):
        rng = np.random.default_rng(n)
        A, blocks, cols, indptr, b, fixed, xd = _system(n, bs, kind, n)
        # the rows in a random order, as a mesh generator may number its nodes
        p = rng.permutation(n)
        P = sp.csr_matrix((np.arange(len(cols)) + 1, cols, indptr), shape=(n, n))[p][:, p].tocsr()
        dofs = (bs * p[:, None] + np.arange(bs)).ravel()
        made[n] = (None, blocks[P.data - 1], P.indices.astype(np.int32), P.indptr.astype(np.int32),
                   b[dofs], fixed[dofs], xd[dofs])
    out = []
    for sched in (N.SCHED_AUTO, N.SCHED_GRAPH):
        N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, sched))
        try:
            systems = [_block_system(torch, rt, made[n], bs) for n in sizes]
            if md == N.SOLVE_MIXED:
                for s in systems:
                    s.ensure_fp32()
            plan = PcgPlan(systems, md, rtol, 2000)
            x0 = [s.x.clone() for s in systems]
            got = []
            for turn in range(2):
                for s, x in zip(systems, x0):
                    if turn:
                        s.vals64.mul_(2.0)
                        if s.vals32 is not None:
                            s.vals32.mul_(2.0)
                        s.b.mul_(-4.0)
                    s.x.copy_(x * (-2.0 if turn else 1.0))
                if turn:
                    plan.refresh()
                for r in plan.solve():
                    assert r.status == N.CFEM_OK, r
                got.append([s.x.cpu().numpy() for s in systems])
            plan.close()
        finally:
            N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_AUTO))
        out.append(got)
    for turn in range(2):
        for n, x, ref in zip(sizes, out[0][turn], out[1][turn]):
            fixed, xd = made[n][5], made[n][6]
            assert np.array_equal(x[fixed], xd[fixed] * (-2.0 if turn else 1.0))
            assert np.linalg.norm(x - ref) <= 2 * tol * np.linalg.norm(ref)
    for n, x, x2 in zip(sizes, out[0][0], out[0][1]):   # twice the matrix, -4 times the rest
        assert np.linalg.norm(x2 + 2 * x) <= 4 * tol * np.linalg.norm(x)


def test_refresh_takes_new_values(torch):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import PcgPlan
    rt = N.runtime()
    for bs in (1, 3):
        data = _system(3000, bs, "band", 5)
        s = _block_system(torch, rt, data, bs)
        plan = PcgPlan([s], N.SOLVE_FP64, 1e-15, 2000)
        x0 = s.x.clone()
        assert plan.solve()[0].status == N.CFEM_OK
        first = s.x.clone()
        s.vals64.mul_(2.0)
        s.b.mul_(2.0)
        plan.refresh()
        s.x.copy_(x0)
        assert plan.solve()[0].status == N.CFEM_OK
        assert (s.x - first).abs().max() <= 1e-12 * first.abs().max()
        plan.close()


def test_zero_load_and_missing_mask(torch):
    """b = 0 without Dirichlet data: x = 0 exactly; a row without a diagonal
    entry is reported, not solved."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    rt = N.runtime()
    data = _system(500, 1, "band", 3)
    s = _block_system(torch, rt, data, 1)
    s.fixed = None
    s.b.zero_()
    assert pcg([s], N.SOLVE_FP64, 1e-12, 2000)[0].status == N.CFEM_OK
    assert torch.count_nonzero(s.x) == 0
    A = data[0].tolil()
    A[7, 7] = 0.0
    A = A.tocsr()
    A.eliminate_zeros()
    up = lambda a, t: torch.from_numpy(a.astype(t)).to(rt.device)  # noqa: E731
    s.row_ptr, s.col, s.vals64 = up(A.indptr, np.int32), up(A.indices, np.int32), up(A.data, np.float64)
    s.b.fill_(1.0)
    assert pcg([s], N.SOLVE_FP64, 1e-12, 2000)[0].status == N.CFEM_ERR_BREAKDOWN


@pytest.mark.parametrize("n,kind", [(1, "band"), (33, "band"), (700, "arrow"), (9000, "band"),
                                    (4000, "scatter"), (120000, "band")])
def test_cocg_matches_direct(torch, n, kind):
    """Complex symmetric systems (the phasor solver): one block, several, rows
    longer than a window, entries past shared memory, and a long arrow row.
    The real part has eigenvalues in [0.2, 2.8] and the imaginary part is a
    positive diagonal, so a relative residual of 1e-12 bounds the error by
    about 14e-12 of the solution: 1e-10."""
    import ctypes
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    A, *_ = _system(n, 1, kind, 7 * n + 1)
    rng = np.random.default_rng(n)
    A = (A + 1j * sp.diags(rng.uniform(0.1, 1.0, n))).tocsr()
    A.sort_indices()
    b = rng.uniform(-1.0, 1.0, n) + 1j * rng.uniform(-1.0, 1.0, n)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rt.device)  # noqa: E731
    ip, ix = up(A.indptr.astype(np.int32)), up(A.indices.astype(np.int32))
    va, vb = up(A.data.view(np.float64)), up(b.view(np.float64))
    x = torch.zeros(2 * n, dtype=torch.float64, device=rt.device)
    st = N.SolveStats()
    N.check(rt.lib.cfem_cocg_solve(rt.ctx, n, N.ptr(ip), N.ptr(ix), N.ptr(va), N.ptr(vb), N.ptr(x),
                                   1e-12, 2000, ctypes.byref(st), rt.stream()))
    assert st.status == N.CFEM_OK and st.relres <= 1e-12
    xs = x.cpu().numpy().view(np.complex128)
    assert np.linalg.norm(A @ xs - b) <= 2e-12 * np.linalg.norm(b)
    if kind != "scatter":
        ref = spla.spsolve(A.tocsc(), b)
        assert np.linalg.norm(xs - ref) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("bs", [1, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_slots_go_on_over_rounds(torch, mode, bs):
    """Systems of one block and of many in solve slots, advanced 16 iterations
    a round (state, residual and inverse kept between launches), one released
    on the way and its slot taken again: each answer bitwise that of a slot
    engine of its own, and within the solve tolerance of the direct one
    (tolerances as above)."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import SlotEngine
    rt = N.runtime()
    md, rtol, tol = ((N.SOLVE_FP64, 1e-13, 1e-12) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10, 1e-9))
    sizes = (3, 40, 4000, 12000)
    datas = [_system(n, bs, "wide", n) for n in sizes]
    cap = max(sizes)
    make = lambda d: _block_system(torch, rt, d, bs)  # noqa: E731
    eng = SlotEngine(rt, 3, bs, md, cap, cap * 30)
    done = {}

    def round_(engine):
        engine.run(1)
        for system, tag, res in engine.poll():
            assert res.status == N.CFEM_OK, (tag, res)
            done[tag] = system.x.clone()

    def drain(engine, want):
        for _ in range(400):
            if all(t in done for t in want):
                return
            round_(engine)
        raise AssertionError("slots did not finish")

    first = eng.assign(make(datas[3]), rtol, 2000, tag="gone")
    eng.assign(make(datas[0]), rtol, 2000, tag=0)
    round_(eng)
    eng.release(first)
    for i in (1, 2):
        eng.assign(make(datas[i]), rtol, 2000, tag=i)
    drain(eng, (0, 1, 2))
    eng.assign(make(datas[3]), rtol, 2000, tag=3)
    drain(eng, (3,))
    got = dict(done)
    for i, d in enumerate(datas):
        one = SlotEngine(rt, 1, bs, md, cap, cap * 30)
        one.assign(make(d), rtol, 2000, tag=("alone", i))
        drain(one, (("alone", i),))
        assert torch.equal(done[("alone", i)], got[i]), i
        x = _exact(d[0], d[4], d[5], d[6])
        assert np.linalg.norm(got[i].cpu().numpy() - x) <= tol * np.linalg.norm(x)
        one.close()
    eng.close()
