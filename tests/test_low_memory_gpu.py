"""Calls when the device's memory runs out: refused with a status, nothing written, and whole again
once there is memory."""
import contextlib
import gc

import numpy as np
import pytest
import torch

from gip_b200 import _lib, cavity

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory_left(mb):
    """Holds all of the device's memory that can be had but for `mb` (even, at least 10) and what is
    smaller than 10 MB; none of it is touched.  (Blocks from 10 MB on are what they say: the
    caching allocator rounds them to 2 MB.)"""
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    first = 10 + mb % 10          # this one and tens of MB are given back
    give = [torch.empty(size << 20, dtype=torch.uint8, device="cuda")
            for size in [first] + [10] * ((mb - first) // 10)]
    held = []
    try:
        big = torch.cuda.mem_get_info()[0] - (256 << 20)
        held.append(torch.empty(big >> 21 << 21, dtype=torch.uint8, device="cuda"))
        with contextlib.suppress(torch.cuda.OutOfMemoryError):
            while True:
                held.append(torch.empty(10 << 20, dtype=torch.uint8, device="cuda"))
        del give
        torch.cuda.empty_cache()
        yield
    finally:
        del held
        torch.cuda.synchronize()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("left_mb", [10, 24, 48, 70])  # of the 90 MB that the 64^3 state takes
def test_snapshot_that_found_no_memory_can_be_taken_later(gpu, left_mb):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(64, re=100.0)
    E = DnsEngine(case, gamma=0.01, pcg_mode="fixed", maxit=5)
    E.advance(2)
    kept = {k: E.field(k) for k in ("u", "p", "mf")}
    with memory_left(left_mb):
        for _ in range(2):
            with pytest.raises(_lib.GipB200Error) as err:
                E.snapshot()
            assert err.value.status == _lib.ERR_NOMEM
        with pytest.raises(_lib.GipB200Error) as err:
            E.snapshot(restore=True)
        assert err.value.status == _lib.ERR_STATE
        E.advance(1)
    E.snapshot(restore=False)
    later = {k: E.field(k) for k in kept}
    E.advance(2)
    E.snapshot(restore=True)
    for k in kept:
        assert np.array_equal(E.field(k), later[k]), k
        assert not np.array_equal(kept[k], later[k]), k
    E.close()  # not left to the collector: a caught error's frames hold it


def _created(make):
    try:
        return make()
    except _lib.GipB200Error as e:
        assert e.status == _lib.ERR_NOMEM or "out of memory" in str(e), e
        return None


def test_large_handles_need_no_memory_for_the_packed_copy(gpu, monkeypatch):
    # whatever memory the sliced layout fits in is enough for a handle: the packed copy is left
    # out where it does not fit beside it; the products are the same bits
    from gip_b200.device import DeviceMatrix
    from test_one_launch_gpu import _band
    n = 200000
    m = _band(n, n, seed=2)
    x = torch.randn(n, dtype=torch.float64, device="cuda")
    want = DeviceMatrix(m).spmv(x, torch.zeros_like(x)).cpu()
    y = torch.zeros_like(x)
    fits = []
    for left_mb in range(10, 60, 2):
        with memory_left(left_mb):
            monkeypatch.setenv("GIPB200_NO_PACK", "1")
            plain = _created(lambda: DeviceMatrix(m))
            fits.append(plain is not None)
            if plain is not None:
                plain.close()
                monkeypatch.delenv("GIPB200_NO_PACK")
                A = _created(lambda: DeviceMatrix(m))
                assert A is not None, left_mb
                y.zero_()
                assert torch.equal(A.spmv(x, y).cpu(), want)
                A.close()
    assert True in fits and False in fits  # the range crosses what the handle needs


SOLVERS = [("stream", 1500000, dict(mode="fixed", maxit=5), range(32, 120, 4)),
           ("mixed", 1500000, dict(mode="mixed", maxit=500, tol=1e-8, inner_tol=0.1, max_outer=50),
            range(64, 320, 16)),
           ("tol_amg", 150000, dict(mode="tol", maxit=100, tol=1e-8, precond="amg"),
            range(16, 96, 6))]


@pytest.mark.parametrize("name,n,kw,left", SOLVERS, ids=[s[0] for s in SOLVERS])
def test_solvers_need_no_memory_for_one_launch(gpu, monkeypatch, name, n, kw, left):
    # where the kernel-by-kernel solver fits, the solver can be created and solves
    from gip_b200.device import DeviceMatrix, PcgSolver
    from test_one_launch_gpu import _band
    A = DeviceMatrix(_band(n, n, seed=2))
    b = torch.randn(n, dtype=torch.float64, device="cuda")
    x, x0 = torch.zeros_like(b), torch.zeros_like(b)
    fits, forms = [], set()
    for left_mb in left:
        with memory_left(left_mb):
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
            K = _created(lambda: PcgSolver(A, **kw))
            fits.append(K is not None)
            if K is not None:
                K.close()
                monkeypatch.delenv("GIPB200_NO_ONE_LAUNCH")
                S = _created(lambda: PcgSolver(A, **kw))
                assert S is not None, left_mb
                forms.add(S.solve_form())
                assert S.solve(b, x, x0)["status"] == 0
                S.close()
    assert True in fits and False in fits, fits  # the range crosses what the solver needs
    assert len(forms - {"loop"}) == 1, forms


def test_engines_hold_no_buffers_of_forms_they_never_run(gpu, monkeypatch):
    # an engine with mixed Jacobi keeps the kernel-by-kernel loop: it takes the memory of an engine
    # that plans nothing else (at 100^3 the unused pairs and residual would be 16 MB; a difference
    # of one 2 MB granule of the allocator is allowed)
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(100, re=100.0)
    kw = dict(gamma=0.01, pcg_mode="mixed", maxit=500, tol=1e-6, inner_tol=0.3, max_outer=100)
    DnsEngine(case, **kw).close()
    used = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        E = DnsEngine(case, **kw)
        torch.cuda.synchronize()
        used.append(before - torch.cuda.mem_get_info()[0])
        E.close()
    assert abs(used[0] - used[1]) <= 2 << 20, used
