"""A solve plan used from another stream than the one it was made on: its
set-up and its refreshes come before its solves and before the release of its
memory, without a wait on the host.

The systems are positive definite with eigenvalues in [0.2, 2.8] (see
test_gpu_resident.py); the same plan on one stream is the reference, bitwise.
"""

import pytest

from test_gpu_resident import _block_system, _system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _systems(torch, rt, many):
    """One system, or more than four launches' worth (blocks dealt out)."""
    sizes = [9000] if not many else [300 + 37 * i for i in range(60)] + [12000] * 6
    return [_block_system(torch, rt, _system(n, 1, "wide", n + i), 1) for i, n in enumerate(sizes)]


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_solve_on_another_stream_than_create(torch, mode, many):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import PcgPlan
    rt = N.runtime()
    md, rtol = (N.SOLVE_FP64, 1e-13) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10)
    systems = _systems(torch, rt, many)
    x0 = [s.x.clone() for s in systems]

    def reset():
        for s, x in zip(systems, x0):
            s.x.copy_(x)
        torch.cuda.synchronize()

    plan = PcgPlan(systems, md, rtol, 2000)
    assert all(r.status == N.CFEM_OK for r in plan.solve())
    want = [s.x.clone() for s in systems]
    plan.close()
    made, used = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        reset()
        with torch.cuda.stream(made):
            plan = PcgPlan(systems, md, rtol, 2000)
        with torch.cuda.stream(used):
            assert all(r.status == N.CFEM_OK for r in plan.solve())
        assert all(torch.equal(s.x, w) for s, w in zip(systems, want))
        plan.close()
        with torch.cuda.stream(made):        # released with its set-up still queued
            PcgPlan(systems, md, rtol, 2000).close()


@pytest.mark.parametrize("scheduler", ["AUTO", "GRAPH"])
def test_solve_on_another_stream_than_refresh(torch, scheduler):
    """New values and a refresh queued behind a wait of some milliseconds."""
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import PcgPlan
    rt = N.runtime()
    (s,) = _systems(torch, rt, False)
    x0 = s.x.clone()
    N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, getattr(N, "SCHED_" + scheduler)))
    try:
        plan = PcgPlan([s], N.SOLVE_FP64, 1e-13, 2000)
    finally:
        N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_AUTO))
    refreshed, used = torch.cuda.Stream(), torch.cuda.Stream()
    out = []
    for away in (False, True):
        s.x.copy_(x0)
        torch.cuda.synchronize()
        with torch.cuda.stream(refreshed):
            torch.cuda._sleep(20_000_000)
            s.vals64.mul_(2.0)
            plan.refresh()
        with torch.cuda.stream(used if away else refreshed):
            assert plan.solve()[0].status == N.CFEM_OK
        out.append(s.x.clone())
        torch.cuda.synchronize()
        with torch.cuda.stream(refreshed):
            s.vals64.div_(2.0)
            plan.refresh()
        torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
