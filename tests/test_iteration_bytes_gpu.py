"""The bytes an engine reports for one PCG iteration are those of the form its solve runs in."""
import pytest

from gip_b200 import cavity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,form", [(10, "block"), (24, "cluster"), (33, "grid"), (64, "stream")])
def test_iteration_bytes_follow_the_form(gpu, monkeypatch, n, form):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(n, re=100.0)
    L = case.ops["L"]
    rows, slices = L.nrows, (L.nrows + 31) // 32
    kw = dict(gamma=0.01, pcg_mode="fixed", maxit=5)
    got = DnsEngine(case, **kw).info()["iteration_bytes"]
    # on chip; 16-byte pairs written and read; the packed words (16 + 4 bytes a row, bases and a
    # flag a slice) with p twice, dinv, and x and p read and written
    want = {"block": 0.0, "cluster": 0.0, "grid": 32.0 * rows,
            "stream": 20.0 * rows + 33.0 * slices + 48.0 * rows}[form]
    assert got == want
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    loop = DnsEngine(case, **kw).info()["iteration_bytes"]
    assert loop == 12.0 * L.nnz + 104.0 * rows  # three kernels, the sliced operator


def test_mixed_amg_iteration_bytes(gpu, monkeypatch):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(24, re=100.0)
    kw = dict(gamma=0.01, pcg_mode="mixed", maxit=500, tol=1e-6, inner_tol=0.01, max_outer=100,
              precond="amg")
    one = DnsEngine(case, **kw).info()["iteration_bytes"]
    monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
    loop = DnsEngine(case, **kw).info()["iteration_bytes"]
    assert abs(one - loop - 8.0 * case.ops["L"].nrows) <= 1e-6 * loop
