"""Solve slots whose systems run on the resident kernel and on the captured
graphs in turn. An arrow system (one row and column with every entry) has a
block whose halo does not fit shared memory, so the graphs take it; a banded
one is resident. Systems and tolerances are those of test_gpu_resident.py.
"""

import numpy as np
import pytest

from test_gpu_resident import _block_system, _exact, _system

pytestmark = pytest.mark.gpu

ARROW = {1: 40000, 3: 16000}       # rows past a halo of 224 KB in either precision


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _engine(rt, n_slots, bs, md):
    from cloudfem_b200.device import SlotEngine
    return SlotEngine(rt, n_slots, bs, md, ARROW[bs], 20 * ARROW[bs])


def _rounds(eng, want, most=200):
    """Rounds until the tags have finished: {tag: (x, iterations)}."""
    from cloudfem_b200 import _native as N
    done = {}
    for _ in range(most):
        if all(t in done for t in want):
            return done
        eng.run(1)
        for system, tag, res in eng.poll():
            assert res.status == N.CFEM_OK, (tag, res)
            done[tag] = (system.x.clone(), res.iterations)
    raise AssertionError("slots did not finish")


@pytest.mark.parametrize("bs", [1, 3])
def test_graph_rounds_stop_with_their_last_system(torch, bs):
    """No launch over the slots' capacity once the only system on the graphs has
    finished or was released, also while a resident one runs."""
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    arrow, band = _system(ARROW[bs], bs, "arrow", 1), _system(2000, bs, "band", 2)
    eng = _engine(rt, 2, bs, N.SOLVE_FP64)

    def launches(rounds):
        before = rt.launches()
        eng.run(rounds)
        eng.poll()
        return rt.launches() - before

    assert launches(3) == 0
    eng.assign(_block_system(torch, rt, arrow, bs), 1e-10, 2000, tag="arrow")
    before = rt.launches()
    _rounds(eng, ["arrow"])
    assert rt.launches() - before >= 16              # it ran on the graphs
    assert launches(3) == 0
    slot = eng.assign(_block_system(torch, rt, arrow, bs), 1e-10, 2000, tag="gone")
    eng.run(1)
    eng.release(slot)
    torch.cuda.synchronize()
    assert launches(3) == 0
    eng.assign(_block_system(torch, rt, band, bs), 1e-10, 2000, tag="band")
    assert launches(1) == 1                          # the resident kernel alone
    eng.close()
