"""Solve slots of 3x3 systems on the captured graphs in the sliced-ELL layout:
systems that the resident kernel does not take (in mixed precision rows of fewer
than 20 blocks, in FP64 an arrow whose halo is past shared memory), one after the
other in one slot (its two row-order sets alternate) and in turn with a resident
system, each answer bitwise the same every time. Systems and tolerances are those
of test_gpu_resident.py; the direct solution is the reference."""

import numpy as np
import pytest

from test_gpu_resident import _block_system, _exact, _system
from test_gpu_slots_routes import _rounds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_graph_and_resident_systems_in_turn(torch, mode):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import SlotEngine
    rt = N.runtime()
    md, rtol, tol = ((N.SOLVE_FP64, 1e-13, 1e-12) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10, 1e-9))
    kind, n, m = ("arrow", 16000, 12000) if mode == "fp64" else ("band", 6000, 2500)
    datas = {"a": _system(n, 3, kind, 1), "b": _system(m, 3, kind, 2), "wide": _system(2000, 3, "wide", 3)}
    eng = SlotEngine(rt, 1, 3, md, n, 20 * n)
    seen = {}
    for name in ("a", "b", "a", "wide", "a", "wide", "b", "b"):
        eng.assign(_block_system(torch, rt, datas[name], 3), rtol, 2000, tag=name)
        before = rt.launches()
        x, its = _rounds(eng, [name])[name]
        rounds = rt.launches() - before
        assert (rounds <= its) == (name == "wide")     # a launch a round, or several an iteration
        if name in seen:
            assert its == seen[name][1] and torch.equal(x, seen[name][0])
        else:
            seen[name] = (x, its)
            d = datas[name]
            ref = _exact(d[0], d[4], d[5], d[6])
            assert np.linalg.norm(x.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
    eng.close()
