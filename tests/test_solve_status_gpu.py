"""The pressure solves' statuses in the step history, and solves whose waits give up: the step
history and the calls that follow say so, and a restored snapshot brings the engine back."""
import ctypes as C

import numpy as np
import pytest

from gip_b200 import _lib, cavity

pytestmark = pytest.mark.gpu

SOLVES = [("fixed", dict(pcg_mode="fixed", maxit=3), 0),
          ("tol", dict(pcg_mode="tol", maxit=3, tol=1e-12), _lib.ERR_NOT_CONVERGED),
          ("tol_amg", dict(pcg_mode="tol", maxit=2, tol=1e-14, precond="amg"), _lib.ERR_NOT_CONVERGED),
          ("mixed", dict(pcg_mode="mixed", maxit=3, tol=1e-12, inner_tol=0.1, max_outer=50),
           _lib.ERR_NOT_CONVERGED),
          ("mixed_amg", dict(pcg_mode="mixed", maxit=2, tol=1e-14, inner_tol=0.01, max_outer=50,
                             precond="amg"), _lib.ERR_NOT_CONVERGED),
          ("mixed_amg_ok", dict(pcg_mode="mixed", maxit=500, tol=1e-8, inner_tol=0.01, max_outer=50,
                                precond="amg"), 0)]


@pytest.mark.parametrize("name,kw,status", SOLVES, ids=[s[0] for s in SOLVES])
@pytest.mark.parametrize("graph", [True, False])
def test_history_has_the_solves_status(gpu, name, kw, status, graph):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(13, re=100.0)
    E = DnsEngine(case, gamma=0.01, use_graph=graph, **kw)
    E.advance(2)
    assert E.history()["status"].tolist() == [status, status]
    E.advance(1030)  # past the first history arrays
    assert len(E.history()["status"]) == 1032 and E.history()["status"][1] == status


def test_wait_that_gives_up_is_reported(gpu):
    # solves and a barrier of a group that claims a CTA it does not have: each gives up and says
    # so; the engine then refuses steps until a valid state is restored
    from gip_b200.device import DnsBatch, DnsEngine, dns_params
    kw = dict(pcg_mode="mixed", maxit=500, tol=1e-8, inner_tol=0.01, max_outer=50, precond="amg")
    case, _ = cavity.generate(13, re=100.0)
    E = DnsEngine(case, gamma=0.01, **kw)
    E.advance(2)
    E.snapshot()
    E.advance(2)
    want = E.field("u")
    st = C.c_int(-1)

    def give_up(e):
        _lib.call("gipb200_dns_check_bounded_wait", e.handle, None, C.byref(st))
        assert st.value == _lib.ERR_TIMEOUT
        for call in (lambda: e.advance(1), e.step_phases):
            with pytest.raises(_lib.GipB200Error) as err:
                call()
            assert err.value.status == _lib.ERR_TIMEOUT

    give_up(E)
    E.snapshot(restore=True)
    E.advance(2)
    assert np.array_equal(E.field("u"), want)
    B = DnsBatch([case, case], [dns_params(gamma=0.01, **kw)] * 2)
    B.advance(1)
    assert B.solver_status() == 0
    give_up(B.instances[1])
    with pytest.raises(_lib.GipB200Error):
        B.advance(1)
    assert B.solver_status() != 0 and B.solver_status() == 0
    B.close()  # not left to the collector: a caught error's frames hold them
    E.close()
