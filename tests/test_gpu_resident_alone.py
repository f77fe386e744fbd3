"""Mixed-precision scalar systems on the resident kernel: an answer is bitwise
the one alone whatever else is in the batch or in the other solve slots, also
where what the launch holds in shared memory depends on them.

One long row makes a block's padded slices larger than the average block, so
alone (shared memory sized by the average) one slice streams that is held in a
launch of several systems: by the layout's arithmetic at 5,000 rows with one of
400 entries, and in slots at 3,000 rows with one of 600.
"""

from unittest import mock

import numpy as np
import pytest
import scipy.sparse as sp

import test_gpu_resident as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _long_row(n, m, seed):
    P = R._pattern(n, "band", None)
    first = n // 2
    cols = np.arange(first, min(n, first + m))
    Q = sp.coo_matrix((np.ones(len(cols)), (np.full(len(cols), first), cols)), shape=(n, n))
    P = (P + Q + Q.T).tocsr()
    P.data[:] = 1.0
    P.sort_indices()
    with mock.patch.object(R, "_pattern", lambda *a: P):
        return R._system(n, 1, "band", seed)


@pytest.mark.parametrize("n,m", [(5000, 400), (3000, 600), (20000, 900), (700, 300)])
def test_batch_equals_alone_with_a_long_row(torch, n, m):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg
    rt = N.runtime()
    datas = [_long_row(n, m, 1), R._system(4000, 1, "wide", 2), R._system(90, 1, "band", 3)]
    systems = [R._block_system(torch, rt, d, 1) for d in datas]
    batch = pcg(systems, N.SOLVE_MIXED, 1e-10, 2000)
    for s, d, r in zip(systems, datas, batch):
        alone = R._block_system(torch, rt, d, 1)
        ra = pcg([alone], N.SOLVE_MIXED, 1e-10, 2000)[0]
        assert ra.status == r.status == N.CFEM_OK and ra.iterations == r.iterations
        assert torch.equal(alone.x, s.x)


@pytest.mark.parametrize("n,m", [(5000, 400), (3000, 600), (20000, 900)])
def test_slot_equals_alone_with_a_long_row(torch, n, m):
    """Against the solve alone in the slot's own shape: an engine of one slot."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import SlotEngine
    rt = N.runtime()
    datas = [_long_row(n, m, 1), R._system(30000, 1, "wide", 2), R._system(12000, 1, "wide", 3)]

    def solve(which):
        eng = SlotEngine(rt, len(which), 1, N.SOLVE_MIXED, 30000, 30000 * 30)
        for i in which:
            eng.assign(R._block_system(torch, rt, datas[i], 1), 1e-10, 2000, tag=i)
        done = {}
        for _ in range(400):
            if len(done) == len(which):
                break
            eng.run(1)
            for system, tag, res in eng.poll():
                assert res.status == N.CFEM_OK, (tag, res)
                done[tag] = (system.x.clone(), res.iterations)
        eng.close()
        return done

    mix = solve((0, 1, 2))
    for i in range(3):
        x, its = solve((i,))[i]
        assert its == mix[i][1]
        assert torch.equal(x, mix[i][0])
