"""Which form a solver's solves take, on both sides of every line: values are compared elsewhere
(test_one_launch_gpu.py), where a form that is no longer chosen would pass unseen."""
import numpy as np
import pytest
import torch

from gip_b200.formats import Csr
from test_one_launch_gpu import SOLVES, _band

pytestmark = pytest.mark.gpu

FIXED = dict(mode="fixed", maxit=5)


def _form(L, n_all=None, **kw):
    from gip_b200 import device as dv
    A = dv.DeviceMatrix(L)
    return dv.PcgSolver(A, n_all=n_all, **kw).solve_form()


@pytest.mark.parametrize("mode", ["fixed", "tol"])
def test_fp64_jacobi_lines(gpu, mode):
    grid = 4 * 256 * min(torch.cuda.get_device_properties(0).multi_processor_count, 256)
    for n, form in ((1, "block"), (1920, "block"), (1921, "cluster"), (16384, "cluster"),
                    (16385, "grid"), (grid, "grid"), (grid + 1, "stream"), (2300001, "loop")):
        assert _form(_band(n, n, seed=1), mode=mode, maxit=5, tol=1e-9) == form, n


def test_fp64_jacobi_falls_back(gpu, monkeypatch):
    n = 300
    assert _form(_band(n, n + 20, ghost=0.0), n + 20, **FIXED) == "block"
    assert _form(_band(n, n + 20, ghost=-0.25), n + 20, **FIXED) == "loop"   # ghosts not zero
    assert _form(_band(160001, 160001, values=300), **FIXED) == "loop"       # too many values
    i = np.arange(n)
    wide = Csr(n, n, np.arange(0, 9 * n + 1, 9, dtype=np.int32),
               np.sort((i[:, None] + np.arange(9)) % n, 1).astype(np.int32).ravel(),
               np.ones(9 * n))
    assert _form(wide, **FIXED) == "loop"                                    # rows of nine entries
    rp = np.arange(n + 1, dtype=np.int32)
    rp[-1] = n - 1
    empty = Csr(n, n, rp, np.arange(n - 1, dtype=np.int32), np.ones(n - 1))
    assert _form(empty, **FIXED) == "loop"                                   # an empty row
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    assert _form(_band(n, n), **FIXED) == "loop"


@pytest.mark.parametrize("solve", sorted(SOLVES))
def test_preconditioned_lines(gpu, solve):
    kw = SOLVES[solve]
    for n, form in ((300, "precond_cluster"), (20000, "precond_cluster"), (20001, "precond_grid")):
        assert _form(_band(n, n, seed=1), **kw) == form, n
    for values, far in ((0, 32), (100, 700), (300, 0)):  # plain slices, 8-bit table, not packed
        assert _form(_band(70000, 70000, far=far, values=values, seed=8), **kw) == "precond_grid"
    if solve == "tol_amg":  # ghost columns that hold values
        assert _form(_band(300, 320, ghost=-0.25), 320, **kw) == "loop"
    if solve == "mixed":
        for n, form in ((2500000, "precond_grid"), (2500001, "loop")):
            assert _form(_band(n, n, seed=1), **kw) == form, n
    if solve == "mixed_amg":
        for n, form in ((700000, "precond_grid"), (700001, "loop")):
            assert _form(_band(n, n, seed=1), **kw) == form, n


@pytest.mark.parametrize("kw,kernels", [
    (dict(pcg_mode="fixed", maxit=20), 11), (dict(pcg_mode="tol", maxit=500, tol=1e-6), 11),
    (dict(pcg_mode="mixed", maxit=500, tol=1e-6, inner_tol=0.01, max_outer=50, precond="amg"), 11),
    (dict(pcg_mode="mixed", maxit=500, tol=1e-6, inner_tol=0.1, max_outer=50), None),
    (dict(pcg_mode="tol", maxit=500, tol=1e-6, precond="amg"), None)])
@pytest.mark.parametrize("n", [11, 24, 33])
def test_engine_steps(gpu, n, kw, kernels):
    # one launch beside the step's own ten, except where the history's count keeps the loop
    from gip_b200 import cavity
    from gip_b200.device import DnsEngine
    E = DnsEngine(cavity.generate(n, re=100.0)[0], gamma=0.01, **kw)
    E.advance(2)
    h = E.history()
    assert np.all(h["kernels"] == kernels) if kernels else np.all(h["kernels"] > 10 + h["iters"])
