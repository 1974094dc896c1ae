"""The V-cycle's profile lists the launches of the cycle that runs."""
import pytest

from gip_b200 import cavity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,n", [("mixed", 100), ("tol", 24)])
def test_small_levels_are_one_entry(gpu, monkeypatch, mode, n):
    # kernel-by-kernel engines: the small levels' one launch in place of its products, with their
    # bytes; level 0 and the total are those of the cycle of one kernel per product
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(n, re=400.0)
    kw = dict(gamma=1.0 / 400.0, pcg_mode=mode, maxit=2000, tol=1e-8, inner_tol=1e-2, max_outer=100,
              reorder=True, precond="amg")
    prof = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("GIPB200_NO_ONE_LAUNCH", "1")
        E = DnsEngine(case, **kw)
        E.advance(1)
        prof.append(E.vcycle_profile(reps=3))
        E.close()
    one, each = prof
    small = [c for c in one if c["kind"] == "small"]
    assert len(small) == 1 and small[0]["kernel"] == "k_amg_small" and small[0]["ms"] > 0
    assert not any(c["kind"] in ("small", "tail") for c in each)
    assert "dense" in [c["kind"] for c in each] and "dense" not in [c["kind"] for c in one]
    top = [(c["level"], c["kind"], c["kernel"], c["bytes"]) for c in each if c["level"] < small[0]["level"]]
    assert [(c["level"], c["kind"], c["kernel"], c["bytes"]) for c in one if c["kind"] != "small"] == top
    total = sum(c["bytes"] for c in each)
    assert abs(sum(c["bytes"] for c in one) - total) <= 1e-9 * total
