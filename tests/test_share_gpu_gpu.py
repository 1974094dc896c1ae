"""Solvers and engines that share the GPU with other streams: no solve claims every SM, the results
are the kernel-by-kernel form's."""
import numpy as np
import pytest
import torch

from gip_b200 import cavity
from test_one_launch_gpu import _band, _t

pytestmark = pytest.mark.gpu

MIXED = dict(mode="mixed", maxit=2000, tol=1e-10, inner_tol=0.1, max_outer=100)


@pytest.mark.parametrize("n,kw,alone,shared", [
    (300, dict(mode="fixed", maxit=9), "block", "block"),
    (5000, dict(mode="fixed", maxit=9), "cluster", "cluster"),
    (20000, dict(mode="fixed", maxit=9), "grid", "loop"),
    (160001, dict(mode="tol", maxit=500, tol=1e-9), "stream", "loop"),
    (5000, MIXED, "precond_cluster", "precond_cluster"), (30000, MIXED, "precond_grid", "loop"),
    (5000, dict(mode="tol", maxit=500, tol=1e-9, precond="amg"), "precond_cluster", "precond_cluster"),
    (30000, dict(mode="tol", maxit=500, tol=1e-9, precond="amg"), "precond_grid", "loop")])
def test_forms_of_a_shared_gpu(gpu, monkeypatch, n, kw, alone, shared):
    from gip_b200 import device as dv
    A = dv.DeviceMatrix(_band(n, n, seed=3))
    b = _t(np.random.default_rng(5).standard_normal(n))
    S = dv.PcgSolver(A, **kw)
    assert S.solve_form() == alone
    S.share_gpu()
    assert S.solve_form() == shared
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    got = S.solve(b, x, torch.zeros_like(b))
    if shared == "loop":  # the same kernels as a solver that never plans another form
        monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        want = dv.PcgSolver(A, **kw).solve(b, y, torch.zeros_like(b))
        assert got == want and torch.equal(x, y)
    S.share_gpu(False)
    assert S.solve_form() == alone


@pytest.mark.parametrize("kw", [dict(pcg_mode="fixed", maxit=20),
                                dict(pcg_mode="mixed", maxit=500, tol=1e-8, inner_tol=0.01,
                                     max_outer=50, precond="amg")], ids=["fixed", "mixed_amg"])
def test_engines_side_by_side(gpu, monkeypatch, kw):
    # three engines on three streams, one of them switched between its steps (its graph is captured
    # again each time): the fields of an engine that runs kernel by kernel
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(33, re=100.0)
    E = [DnsEngine(case, gamma=0.01, **kw) for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in E]
    for e in E:
        e.share_gpu()
    for e, s in zip(E, streams):
        e.advance(2, s)
    last, s = E[2], streams[2]
    last.snapshot(stream=s)
    last.share_gpu(False)
    last.advance(2, s)
    last.snapshot(restore=True, stream=s)
    last.share_gpu()
    for e, s in zip(E, streams):
        e.advance(3, s)
    torch.cuda.synchronize()
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    K = DnsEngine(case, gamma=0.01, **kw)
    K.advance(5)
    for e in E:
        assert e.history()["iters"].tolist() == K.history()["iters"].tolist()
        for k in ("u", "v", "w", "p", "mf"):
            assert np.array_equal(e.field(k), K.field(k)), k
