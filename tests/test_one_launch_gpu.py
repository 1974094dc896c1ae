"""FP64 Jacobi-PCG as one launch: the cluster, grid and streamed forms at the edges of their
ranges, against the oracle's GIP_LinearSolver."""
import numpy as np
import pytest
import torch

from gip_b200.formats import Csr

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _band(n, n_all, far=0, values=0, seed=0, ghost=0.0):
    """SPD band matrix: couplings to i +- 1, i +- 37 and (far > 0) of every far-th row to a
    row across the matrix; `values` > 0 draws the diagonal from that many doubles.  Columns
    past n (ghosts) hold `ghost`."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    rows, cols, vals = [], [], []
    for d in (1, 37):
        a = i[:-d] if d < n else i[:0]
        rows += [a, a + d]
        cols += [a + d, a]
        vals += [np.full(a.size, -1.0)] * 2
    if far:
        a = i[: n // 2 : far]
        b = a + n // 2
        rows += [a, b]
        cols += [b, a]
        vals += [np.full(a.size, -0.5)] * 2
    if n_all > n:
        g = np.arange(min(n_all - n, n))
        rows.append(g)
        cols.append(n + g)
        vals.append(np.full(g.size, ghost))
    diag = 6.5 + (rng.integers(0, values, n) / 16.0 if values else 0.0) * np.ones(n)
    rows.append(i)
    cols.append(i)
    vals.append(diag)
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    r, c, v = r[o], c[o], v[o]
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return Csr(n, n_all, rp.astype(np.int32), c.astype(np.int32), v.astype(np.float64))


def _close(got, want):
    """Within 1e-10 of the scale; NaN where the oracle has NaN (one unknown is solved after
    one iteration, and GIP's fixed iterations then divide 0 by 0)."""
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fine = ~np.isnan(want)
    if fine.any():
        assert np.abs(got - want)[fine].max() <= 1e-10 * np.abs(want[fine]).max()


SIZES = [1, 31, 32, 33, 256, 257, 4096, 4097, 16384, 16385, 37888, 37889, 151552, 151553]


@pytest.mark.parametrize("n", SIZES)
def test_forms_match_oracle_at_their_edges(gpu, oracle_mod, n):
    # fixed iterations from a nonzero start with zero-valued ghost columns; the solver's
    # parity bar (1e-10 of the solution's scale) as for the three-kernel loop
    from gip_b200 import device as dv
    n_all = n + min(n, 40)
    L = _band(n, n_all, far=1000, seed=n)
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n_all)
    xr, it, _ = oracle_mod.pcg(L, b, x0, maxit=9, mode=0)
    S = dv.PcgSolver(dv.DeviceMatrix(L), n_all=n_all, mode="fixed", maxit=9)
    x = _t(np.zeros(n_all))
    for start in (_t(x0), None):   # a separate start, then x = x0 in place
        if start is None:
            x.copy_(_t(x0))
        res = S.solve(_t(b), x, x if start is None else start)
        assert res["iterations"] == it == 9
        got = x.cpu().numpy()
        assert np.array_equal(got[n:], x0[n:])
        _close(got, xr)


@pytest.mark.parametrize("n,far,values", [(151600, 32, 0), (160001, 5000, 100), (160001, 0, 300),
                                          (2300001, 0, 0)])
def test_streamed_form_layouts(gpu, oracle_mod, n, far, values):
    # packed rows beside plain slices (far couplings spread a slot over more than 16 bits), an
    # 8-bit value table, an operator without a table (three kernels), and more rows than the
    # shared memory holds (three kernels on the packed operator)
    from gip_b200 import device as dv
    L = _band(n, n, far=far, values=values, seed=3)
    b = np.random.default_rng(5).standard_normal(n)
    xr, it, rr = oracle_mod.pcg(L, b, np.zeros(n), maxit=500, mode=1, tol=1e-9)
    S = dv.PcgSolver(dv.DeviceMatrix(L), mode="tol", maxit=500, tol=1e-9)
    x = _t(np.zeros(n))
    res = S.solve(_t(b), x, _t(np.zeros(n)))
    assert res["status"] == 0 and abs(res["iterations"] - it) <= 1
    if res["iterations"] == it:
        _close(x.cpu().numpy(), xr)


@pytest.mark.parametrize("n", [100, 5000, 20000, 152000])
def test_forms_follow_the_general_path(gpu, monkeypatch, n):
    # failures and special starts come out as the three-kernel loop has them
    from gip_b200 import device as dv
    L = _band(n, n + 8, seed=1)
    A = dv.DeviceMatrix(L)
    rng = np.random.default_rng(2)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n + 8)
    bad = b.copy()
    bad[n // 3] = np.nan
    inf = x0.copy()
    inf[n + 3] = np.inf          # a ghost entry: its stored zero makes the residual NaN
    out = []
    for general in (False, True):
        if general:
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        got = []
        for mode, maxit, rhs, start in (("tol", 2, b, x0), ("tol", 50, bad, x0), ("tol", 50, b, inf),
                                        ("fixed", 3, bad, x0), ("tol", 50, np.zeros(n), 0 * x0),
                                        ("fixed", 0, b, x0)):
            S = dv.PcgSolver(A, n_all=n + 8, mode=mode, maxit=maxit, tol=1e-9)
            x = _t(np.ones(n + 8))
            r = S.solve(_t(rhs), x, _t(start))
            got.append((r["status"], r["iterations"], bool(torch.isfinite(x[:n]).all())))
        out.append(got)
    assert out[0] == out[1], out


def test_nonzero_ghost_values_keep_the_general_path(gpu, oracle_mod):
    # ghost columns with nonzero values read the start's ghost entries in every product
    from gip_b200 import device as dv
    n = 300
    L = _band(n, n + 20, seed=4, ghost=-0.25)
    rng = np.random.default_rng(6)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n + 20)
    xr, it, _ = oracle_mod.pcg(L, b, x0, maxit=9, mode=0)
    S = dv.PcgSolver(dv.DeviceMatrix(L), n_all=n + 20, mode="fixed", maxit=9)
    x = _t(np.zeros(n + 20))
    S.solve(_t(b), x, _t(x0))
    _close(x.cpu().numpy(), xr)


SOLVES = {
    "mixed": dict(mode="mixed", maxit=5000, tol=1e-10, inner_tol=0.1, max_outer=100),
    "mixed_amg": dict(mode="mixed", maxit=2000, tol=1e-10, inner_tol=1e-2, max_outer=100,
                      precond="amg"),
    "tol_amg": dict(mode="tol", maxit=2000, tol=1e-10, precond="amg"),
}


@pytest.mark.parametrize("solve", sorted(SOLVES))
@pytest.mark.parametrize("n", [11, 16, 17, 27, 28, 40])
def test_preconditioned_solves_as_one_launch(gpu, monkeypatch, solve, n):
    # clusters of 8 (to 4096 rows) and 16 (to 20000) and the cooperative grid, on the cavity's
    # pinned operator with ghost columns from a nonzero start, against the same solver kernel
    # by kernel: the same row sums, dots added in another order, so the iterates agree far
    # below the tolerance's own error (conditioning x 1e-10)
    from gip_b200 import cavity
    from gip_b200 import device as dv
    case, _ = cavity.generate(n, re=100.0)
    L = case.ops["L"]
    A = dv.DeviceMatrix(L)
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(L.nrows), rng.standard_normal(case.n_owned) * 0.1
    S = dv.PcgSolver(A, n_all=case.n_owned, **SOLVES[solve])
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    K = dv.PcgSolver(A, n_all=case.n_owned, **SOLVES[solve])
    xs, xk = _t(np.zeros(case.n_owned)), _t(np.zeros(case.n_owned))
    rk = K.solve(_t(b), xk, _t(x0))
    for alias in (False, True):
        if alias:
            xs.copy_(_t(x0))
        rs = S.solve(_t(b), xs, xs if alias else _t(x0))
        assert rs["status"] == rk["status"] == 0
        assert abs(rs["iterations"] - rk["iterations"]) <= 0.1 * rk["iterations"] + 1
        got, want = xs.cpu().numpy(), xk.cpu().numpy()
        assert np.array_equal(got[L.nrows:], x0[L.nrows:])
        assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
        r = b - L.to_scipy() @ got
        assert np.linalg.norm(r) <= 1.0001e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("solve", sorted(SOLVES))
def test_preconditioned_one_launch_statuses(gpu, monkeypatch, solve):
    from gip_b200 import cavity
    from gip_b200 import device as dv
    L, b = cavity.poisson_problem(14, seed=2)
    A = dv.DeviceMatrix(L)
    bad = b.copy()
    bad[17] = np.nan
    out = []
    for general in (False, True):
        if general:
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        S = dv.PcgSolver(A, **SOLVES[solve])
        T = dv.PcgSolver(A, **dict(SOLVES[solve], maxit=2))
        got = []
        for slv, rhs in ((S, bad), (S, b), (T, b), (S, 0 * b)):
            x = _t(np.ones(L.nrows))
            r = slv.solve(_t(rhs), x, _t(np.zeros(L.nrows)))
            got.append((r["status"], bool(torch.isfinite(x).all())))
        out.append(got)
    assert out[0] == out[1] and out[0][1][0] == 0, out


@pytest.mark.parametrize("values,far", [(0, 32), (100, 700), (300, 0)])
def test_preconditioned_one_launch_layouts(gpu, monkeypatch, values, far):
    # plain slices beside packed ones, an 8-bit value table, and an operator that does not
    # pack: the same solutions kernel by kernel
    from gip_b200 import device as dv
    n = 70000
    A = dv.DeviceMatrix(_band(n, n, far=far, values=values, seed=8))
    b = np.random.default_rng(3).standard_normal(n)
    for solve in sorted(SOLVES):
        monkeypatch.delenv("GIPB200_NO_ONE_LAUNCH", raising=False)
        S = dv.PcgSolver(A, **SOLVES[solve])
        monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        K = dv.PcgSolver(A, **SOLVES[solve])
        xs, xk = _t(np.zeros(n)), _t(np.zeros(n))
        rs, rk = S.solve(_t(b), xs, _t(np.zeros(n))), K.solve(_t(b), xk, _t(np.zeros(n)))
        assert rs["status"] == rk["status"] == 0, (solve, rs, rk)
        assert float((xs - xk).abs().max()) <= 1e-8 * float(xk.abs().max()), solve


@pytest.mark.parametrize("edges", [[12, 17, 16, 24, 9], [10, 10], [40, 8, 20]])
def test_grouped_batch_solves_equal_the_branches(gpu, monkeypatch, edges):
    # a batch's mixed AMG solves in one launch, a CTA group per instance, against the same
    # batch solving inside its graph branches and against single engines: the same steps
    from gip_b200 import cavity
    from gip_b200.device import DnsBatch, DnsEngine, dns_params
    cases = [cavity.generate(n, re=100.0 * (i + 1), permute_seed=i)[0] for i, n in enumerate(edges)]
    kw = dict(pcg_mode="mixed", maxit=2000, tol=1e-8, inner_tol=1e-2, max_outer=100, reorder=True,
              precond="amg")
    prm = [dns_params(gamma=1.0 / (100.0 * (i + 1)), **kw) for i in range(len(edges))]
    G = DnsBatch(cases, prm)
    single = DnsEngine(cases[0], gamma=1.0 / 100.0, **kw)
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    B = DnsBatch(cases, prm)
    for batch in (G, B, single):
        batch.advance(2)
        batch.advance(1)
    assert np.all(G.instances[0].history()["kernels"] == 11)   # one launch, counted once
    assert all(np.all(e.history()["kernels"] == 10) for e in G.instances[1:])
    assert np.all(B.instances[0].history()["kernels"] > 11)
    for e, f in zip(G.instances, B.instances):
        he, hf = e.history(), f.history()
        assert np.all(he["massr"] < 1e-6) and np.all(np.abs(he["iters"] - hf["iters"]) <= 1)
        scale = np.abs(f.field("u")).max()
        for k in ("u", "v", "w"):
            assert np.abs(e.field(k) - f.field(k)).max() <= 1e-9 * scale, k
    for k in ("u", "v", "w"):
        assert np.abs(G.instances[0].field(k) - single.field(k)).max() <= 1e-9 * np.abs(single.field("u")).max()


@pytest.mark.parametrize("mode,n,fewer", [("mixed", 89, True), ("mixed", 100, True),
                                          ("tol", 24, True), ("tol", 36, False)])
def test_small_levels_in_one_launch_are_exact(gpu, monkeypatch, mode, n, fewer):
    # kernel-by-kernel cycles run their small levels in one launch: every row is summed as its
    # own kernel sums it, so the steps are the same bit for bit, in fewer kernels (36^3 in FP64
    # has one level between the finest and the dense one, with more than 1 MB: none)
    from gip_b200 import cavity
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(n, re=400.0)
    kw = dict(gamma=1.0 / 400.0, pcg_mode=mode, maxit=2000, tol=1e-8, inner_tol=1e-2,
              max_outer=100, reorder=True, precond="amg")
    out = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        E = DnsEngine(case, **kw)
        E.advance(2)
        out.append((E.history()["iters"], E.history()["kernels"], {k: E.field(k) for k in "uvwp"}))
        E.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.all((out[0][1] < out[1][1]) == fewer)
    for k in "uvwp":
        assert np.array_equal(out[0][2][k], out[1][2][k]), k


@pytest.mark.parametrize("wide", [False, True])  # rows of at most six and of eight entries
@pytest.mark.parametrize("n", [480, 481, 960, 961, 1440, 1441, 1920, 1921])
def test_block_form_matches_oracle_at_its_edges(gpu, oracle_mod, n, wide):
    # the one-CTA form at one to four rows a thread, and the first size past it; the solver's
    # parity bar (1e-10 of the solution's scale)
    import scipy.sparse as sp
    from gip_b200 import device as dv
    n_all = n + 40
    L = _band(n, n_all, far=50, seed=n)
    if wide:
        M = sp.csr_matrix((L.val, L.col, L.rowptr), shape=(n, n_all)).tolil()
        for i in (0, 50, 100):  # rows with a far coupling, and the last ones with ghost columns
            for j in (i + 5, i + 9):
                M[i, j] = M[j, i] = -0.25
        M = M.tocsr()
        M.sort_indices()
        L = Csr(n, n_all, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
    assert np.diff(L.rowptr).max() == (8 if wide else 6)
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n_all)
    for mode, kw in (("fixed", dict(maxit=9)), ("tol", dict(maxit=500, tol=1e-9))):
        xr, it, _ = oracle_mod.pcg(L, b, x0, mode=0 if mode == "fixed" else 1, **kw)
        S = dv.PcgSolver(dv.DeviceMatrix(L), n_all=n_all, mode=mode, **kw)
        x = _t(np.zeros(n_all))
        res = S.solve(_t(b), x, _t(x0))
        assert res["status"] == 0 and abs(res["iterations"] - it) <= 1
        if res["iterations"] == it:
            _close(x.cpu().numpy(), xr)


@pytest.mark.parametrize("first,second", [(400000, 160001), (160001, 400000)])
def test_streamed_solvers_of_different_sizes_live_side_by_side(gpu, oracle_mod, first, second):
    # each plans its own shared memory on the same kernel: both still launch afterwards, in
    # either order of creation
    from gip_b200 import device as dv
    made = []
    for n in (first, second):
        L = _band(n, n, seed=n)
        b = np.random.default_rng(n).standard_normal(n)
        S = dv.PcgSolver(dv.DeviceMatrix(L), mode="fixed", maxit=5)
        made.append((n, S, b, oracle_mod.pcg(L, b, np.zeros(n), maxit=5, mode=0)[0]))
    for _ in range(2):
        for n, S, b, xr in made:
            x = _t(np.zeros(n))
            assert S.solve(_t(b), x, _t(np.zeros(n)))["iterations"] == 5
            _close(x.cpu().numpy(), xr)
