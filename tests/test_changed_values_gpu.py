"""Operators whose values change (spmv_values) after a solver or a graph was made from them:
what runs later reads the values as they are then."""
import numpy as np
import pytest
import torch

from gip_b200.formats import Csr
from test_one_launch_gpu import _band, _t

pytestmark = pytest.mark.gpu

FIXED = dict(mode="fixed", maxit=9)
AMG = dict(mode="tol", maxit=4, tol=1e-14, precond="amg")


def _write(A, csr_values):
    """(eye, v, write): write(eye, v) is the spmv_values call that makes csr_values A's values."""
    from gip_b200 import device as dv
    n = csr_values.size
    eye = dv.DeviceMatrix(Csr(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                              np.ones(n)))
    return eye, _t(csr_values), lambda I, v: I.spmv_values(v, A)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,values,kw,form", [
    (300, 0, FIXED, "block"), (5000, 0, FIXED, "cluster"), (20000, 0, FIXED, "grid"),
    (152000, 0, FIXED, "stream"), (5000, 300, AMG, "precond_cluster"),
    (5000, 0, AMG, "precond_cluster"), (30000, 300, AMG, "precond_grid")])
def test_solvers_follow_ghost_values_written_later(gpu, monkeypatch, n, values, kw, form, captured):
    # planned on ghost columns of zeros; then spmv_values (called after the creation, or captured
    # before it and replayed after it) writes coefficients into them: the same solution as a
    # solver made for the new values that runs kernel by kernel, in the same iterations (dots
    # and products of FP64 in the same order: 1e-10 of the scale is the solvers' parity bar)
    from gip_b200 import device as dv
    n_all = n + 20
    zero = _band(n, n_all, values=values, seed=4, ghost=0.0)
    new = Csr(n, n_all, zero.rowptr, zero.col, np.where(zero.col >= n, -0.25, zero.val))
    A = dv.DeviceMatrix(zero)
    eye, v, write = _write(A, new.val)
    g = torch.cuda.CUDAGraph()
    if captured:
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            write(eye, v)
    S = dv.PcgSolver(A, n_all=n_all, **kw)
    assert captured or S.solve_form() == form
    rng = np.random.default_rng(6)
    b, x0 = _t(rng.standard_normal(n)), _t(rng.standard_normal(n_all))
    x, y = torch.zeros_like(x0), torch.zeros_like(x0)
    S.solve(b, x, x0)
    g.replay() if captured else write(eye, v)
    torch.cuda.synchronize()
    assert S.solve_form() == "loop"
    got = S.solve(b, x, x0)
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    K = dv.PcgSolver(dv.DeviceMatrix(new), n_all=n_all, **kw)
    assert K.solve_form() == "loop"
    want = K.solve(b, y, x0)
    assert (got["status"], got["iterations"]) == (want["status"], want["iterations"])
    assert float((x - y).abs().max()) <= 1e-10 * float(y.abs().max())


@pytest.mark.parametrize("n,form", [(300, "block"), (5000, "cluster"), (20000, "grid")])
def test_forms_without_ghosts_read_new_values(gpu, n, form):
    # no ghost columns and nothing packed: the one-launch forms stay and read the new values (the
    # Jacobi scaling is the old ones', a constant factor of the preconditioner that CG's iterates
    # do not see)
    from gip_b200 import device as dv
    old = _band(n, n, seed=4)
    new = Csr(n, n, old.rowptr, old.col, 2.0 * old.val)
    A = dv.DeviceMatrix(old)
    S = dv.PcgSolver(A, **FIXED)
    eye, v, write = _write(A, new.val)
    write(eye, v)
    torch.cuda.synchronize()
    assert S.solve_form() == form
    b = _t(np.random.default_rng(6).standard_normal(n))
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    S.solve(b, x, torch.zeros_like(b))
    dv.PcgSolver(dv.DeviceMatrix(new), **FIXED).solve(b, y, torch.zeros_like(b))
    assert float((x - y).abs().max()) <= 1e-10 * float(y.abs().max())


@pytest.mark.parametrize("together", [True, False])
def test_captured_products_read_the_values_of_their_replay(gpu, together):
    # a handle large enough for the packed layout: products captured with a later spmv_values
    # (the second replay's products are the new values'), and products captured alone, replayed
    # after an spmv_values that was not captured; the products' sums keep their order, bit for bit
    from gip_b200 import device as dv
    n = 220000
    old = _band(n, n, seed=4)
    new = Csr(n, n, old.rowptr, old.col, np.random.default_rng(1).standard_normal(old.nnz))
    T = dv.DeviceMatrix(old)
    eye = dv.DeviceMatrix(Csr(old.nnz, old.nnz, np.arange(old.nnz + 1, dtype=np.int32),
                              np.arange(old.nnz, dtype=np.int32), np.ones(old.nnz)))
    v = _t(new.val)
    x = torch.randn(n, dtype=torch.float64, device="cuda")
    first = T.spmv(x, torch.zeros_like(x))
    second = dv.DeviceMatrix(new).spmv(x, torch.zeros_like(x))
    y, z, d = torch.zeros_like(x), torch.zeros_like(x), x.new_zeros(1)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        T.spmv(x, y)
        T.spmv_dot(x, z, d)
        if together:
            eye.spmv_values(v, T)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, first) and torch.equal(z, first)
    if not together:
        eye.spmv_values(v, T)
        torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, second) and torch.equal(z, second)
