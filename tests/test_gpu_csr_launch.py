"""The one launch over the CSR arrays (PERSISTENT without the resident kernel,
whose memory CFEM_PARAM_ALLOC_FAIL withholds): against the direct solution, a
system alone bitwise as in a batch, and the allocation-free call the same.
Systems and tolerances are those of test_gpu_resident.py."""

import numpy as np
import pytest

from test_gpu_resident import _block_system, _exact, _system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


@pytest.mark.parametrize("bs", [1, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_launch_over_csr_arrays(torch, mode, bs):
    from cloudfem_b200 import _native as N
    from cloudfem_b200.device import pcg, pcg_noalloc
    rt = N.runtime()
    md, rtol, tol = ((N.SOLVE_FP64, 1e-13, 1e-12) if mode == "fp64" else (N.SOLVE_MIXED, 1e-10, 1e-9))
    datas = [_system(n, bs, kind, n + bs) for n, kind in ((1, "band"), (33, "band"), (700, "arrow"),
                                                          (2000, "wide"), (9000, "band"))]
    N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_PERSISTENT))
    rt.set_param(N.PARAM_ALLOC_FAIL, 1)
    try:
        systems = [_block_system(torch, rt, d, bs) for d in datas]
        batch = pcg(systems, md, rtol, 2000)
        for s, d, r in zip(systems, datas, batch):
            assert r.status == N.CFEM_OK
            for solve in (lambda t: pcg([t], md, rtol, 2000)[0], lambda t: pcg_noalloc(t, md, rtol, 2000)):
                alone = _block_system(torch, rt, d, bs)
                alone.ensure_fp32()
                before = rt.launches()
                ra = solve(alone)
                assert rt.launches() - before <= 3           # not the graphs, nor the resident kernel
                assert ra.status == N.CFEM_OK and ra.iterations == r.iterations
                assert torch.equal(alone.x, s.x)
            x = _exact(d[0], d[4], d[5], d[6])
            assert np.linalg.norm(s.x.cpu().numpy() - x) <= tol * np.linalg.norm(x)
    finally:
        rt.set_param(N.PARAM_ALLOC_FAIL, 0)
        N.check(rt.lib.cfem_ctx_set_scheduler(rt.ctx, N.SCHED_AUTO))
