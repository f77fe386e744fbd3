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


@pytest.mark.parametrize("ending", ["finished", "released"])
def test_slots_give_their_memory_back(torch, ending):
    """What a slot holds on the resident kernel (38 bytes a block of an FP32 3x3
    system, 26 MB for each of these) is the pool's again once its system has
    finished or was released, not when the slot is taken next."""
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    n, held = 30000, 4 * 20 * 2 ** 20
    data = _system(n, 3, "wide", 1)
    from cloudfem_b200.device import SlotEngine
    eng = SlotEngine(rt, 4, 3, N.SOLVE_MIXED, n, 30 * n)
    idle = rt.trim(0)
    slots = [eng.assign(_block_system(torch, rt, data, 3), 1e-10, 2000, tag=i) for i in range(4)]
    eng.run(1)
    assert rt.trim(0) >= idle + held             # the measure sees them
    if ending == "finished":
        _rounds(eng, range(4))
    else:
        for s in slots:
            eng.release(s)
    assert rt.trim(0) <= idle + held // 4
    eng.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_admission_estimates_cover_a_request(torch, precision):
    """What the server takes off its budget for a request covers what the
    request holds on the device while it is in a slot, the resident copy too."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200 import serve
    from cloudfem_b200.mesh import box_mesh, box_mesh_tet10
    rt = N.runtime()
    for kind, mesh in (("p1_heat", box_mesh(60, 60, 60)), ("t10_heat", box_mesh_tet10(24, 24, 24)),
                       ("t10_elast", box_mesh_tet10(16, 16, 16))):
        r = serve.Request(0, kind, mesh)
        srv = serve.Server(precision=precision)
        eng = srv._engine(kind, srv._slot_class(r))
        torch.cuda.empty_cache()
        before = rt.trim(0) + torch.cuda.memory_allocated()
        slot = eng.assign(srv._system(r), srv.rtol, tag=r)
        eng.run(1)
        taken = rt.trim(0) + torch.cuda.memory_allocated() - before
        assert 0 < taken <= r.bytes_estimate() + 64 * 2 ** 20, (kind, taken, r.bytes_estimate())
        eng.release(slot)
        eng.close()


def test_resident_system_over_a_running_graph_system(torch):
    """A slot whose system still runs on the graphs is given to a resident one:
    later rounds leave the first system's x alone, whatever else the graphs run."""
    import ctypes
    from cloudfem_b200 import _native as N
    rt = N.runtime()
    arrow, band = _system(ARROW[1], 1, "arrow", 1), _system(2000, 1, "band", 2)
    eng = _engine(rt, 2, 1, N.SOLVE_FP64)
    first, other = (_block_system(torch, rt, arrow, 1) for _ in range(2))
    slot = eng.assign(first, 1e-30, 2000, tag="first")
    eng.assign(other, 1e-13, 2000, tag="other")
    second = _block_system(torch, rt, band, 1)
    ls = second.linsys(N.SOLVE_FP64, 1e-13, 2000)
    N.check(rt.lib.cfem_pcg_slots_assign(eng.handle, slot, ctypes.byref(ls), rt.stream()))
    torch.cuda.synchronize()
    eng.busy[slot] = (second, "second")
    before = first.x.clone()
    done = _rounds(eng, ["second", "other"])
    assert torch.equal(first.x, before)
    x = _exact(band[0], band[4], band[5], band[6])
    assert np.linalg.norm(done["second"][0].cpu().numpy() - x) <= 1e-12 * np.linalg.norm(x)
    eng.close()
