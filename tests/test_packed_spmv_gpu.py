"""Matrix handles' products from the packed FP64 layout: the sliced layout's results, bit for
bit."""
import numpy as np
import pytest
import torch

from gip_b200.formats import Csr

pytestmark = pytest.mark.gpu


def _operator(n, ncols, values, empty, far, seed):
    """n rows of up to 8 entries near the diagonal (stored order shuffled in a quarter of the
    slices), some rows empty, stored zeros among the values; every far-th row has an entry
    across the matrix (its slice cannot pack)."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(1, 9, n)
    if empty:
        lens[rng.random(n) < 0.1] = 0
        lens[64:128] = 0
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    rows = np.repeat(np.arange(n), lens)
    slot = np.arange(rp[-1]) - rp[rows]
    col = np.clip(rows + 37 * slot - 100, 0, ncols - 1)
    if far:
        pick = (rows % far == 0) & (slot == 0)
        col[pick] = (rows[pick] + ncols // 2) % ncols
    tab = rng.standard_normal(values)
    tab[0] = 0.0
    if values > 3:
        tab[1] = -0.0
    val = tab[rng.integers(0, values, rp[-1])]
    return Csr(n, ncols, rp.astype(np.int32), col.astype(np.int32), val)


@pytest.mark.parametrize("n,extra,values,empty,far", [
    (200000, 0, 15, False, 0), (200001, 500, 16, True, 0), (200031, 0, 7, True, 700),
    (262144, 33, 255, False, 3000), (210000, 0, 400, False, 0), (199999, 0, 5, True, 0)])
def test_packed_products_equal_sliced(gpu, monkeypatch, n, extra, values, empty, far):
    # 15 / 255 distinct values are the most a 4- / 8-bit table holds; 400 do not pack, nor does
    # an operator below the size from which handles pack
    from gip_b200 import device as dv
    m = _operator(n, n + extra, values, empty, far, seed=n + values)
    P = dv.DeviceMatrix(m)
    monkeypatch.setenv("GIPB200_NO_PACK", "1")
    S = dv.DeviceMatrix(m)
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n + extra, dtype=torch.float64, device="cuda", generator=g)
    special = x.clone()
    special[n // 2] = float("inf")     # times stored zeros and in rows that do not have it
    special[n // 3] = float("nan")
    y0 = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    for xv in (x, special):
        for args in ((), (0.5, -0.25, 1)):
            yp, ys = P.spmv(xv, y0.clone(), *args), S.spmv(xv, y0.clone(), *args)
            assert torch.equal(yp.isnan(), ys.isnan())
            assert torch.equal(yp.nan_to_num(7.0), ys.nan_to_num(7.0))
    yp, ys = y0.clone(), y0.clone()
    dp, ds = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    P.spmv_dot(x, yp, dp, n_dot=n - 5)
    S.spmv_dot(x, ys, ds, n_dot=n - 5)
    assert torch.equal(yp, ys)
    scale = float((x[:n - 5] * ys[:n - 5]).abs().sum())
    assert abs(float(dp) - float(ds)) <= 1e-13 * scale  # the dots' bar: another summation order


def test_new_values_replace_the_packed_ones(gpu):
    # values written through spmv_values are what later products of the handle use
    from gip_b200 import device as dv
    n = 220000
    m = _operator(n, n, 9, False, 0, seed=4)
    T = dv.DeviceMatrix(m)
    nnz = m.nnz
    D = dv.DeviceMatrix(Csr(nnz, nnz, np.arange(nnz + 1, dtype=np.int32),
                            np.arange(nnz, dtype=np.int32), np.full(nnz, 2.0)))
    v = torch.from_numpy(np.random.default_rng(1).standard_normal(nnz)).cuda()
    x = torch.randn(n, dtype=torch.float64, device="cuda")
    D.spmv_values(v, T)
    want = dv.DeviceMatrix(Csr(n, n, m.rowptr, m.col, 2.0 * v.cpu().numpy()))
    y = T.spmv(x, torch.zeros(n, dtype=torch.float64, device="cuda"))
    assert torch.equal(y, want.spmv(x, torch.zeros_like(y)))


def test_new_values_reach_an_existing_solver(gpu):
    # a solver that packed its operator when it was created solves with the operator's values
    # of the call: doubled, b = 2 A x has the solution of b = A x at 2 x (the Jacobi scaling,
    # taken at creation, only scales the search by a constant)
    from gip_b200 import device as dv
    n = 180000
    i = np.arange(n)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(1 + (i > 0) + (i < n - 1))
    col = np.concatenate([[c for c in (r - 1, r, r + 1) if 0 <= c < n] for r in range(n)])
    rows = np.repeat(i, np.diff(rp))
    val = np.where(col == rows, 4.0, -1.0)
    A = dv.DeviceMatrix(Csr(n, n, rp.astype(np.int32), col.astype(np.int32), val))
    S = dv.PcgSolver(A, mode="tol", maxit=200, tol=1e-12)
    b = torch.randn(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    assert S.solve(b, x, torch.zeros_like(b))["status"] == 0
    nnz = val.size
    D = dv.DeviceMatrix(Csr(nnz, nnz, np.arange(nnz + 1, dtype=np.int32),
                            np.arange(nnz, dtype=np.int32), np.full(nnz, 2.0)))
    D.spmv_values(torch.from_numpy(val).cuda(), A)
    x2 = torch.zeros_like(b)
    assert S.solve(b, x2, torch.zeros_like(b))["status"] == 0
    assert float((2.0 * x2 - x).abs().max()) <= 1e-10 * float(x.abs().max())
