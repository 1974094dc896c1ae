"""launch_count counts what a grouped batch step launches."""
import pytest

from gip_b200 import cavity

pytestmark = pytest.mark.gpu


def test_grouped_batch_counts_every_kernel(gpu):
    # per step and instance ten kernels of its own and the one that takes the
    # ghost columns' part off the right-hand side; the grouped solve is counted on the first instance
    from gip_b200.device import DnsBatch, dns_params
    kw = dict(gamma=0.01, pcg_mode="mixed", maxit=500, tol=1e-6, inner_tol=0.01, max_outer=50,
              precond="amg")
    cases = [cavity.generate(n, re=100.0)[0] for n in (12, 16)]
    B = DnsBatch(cases, [dns_params(**kw)] * 2)
    B.advance(1)
    before = [e.launch_count() for e in B.instances]
    B.advance(3)
    got = [e.launch_count() - c for e, c in zip(B.instances, before)]
    assert B.instances[0].history()["kernels"][0] == 11  # solved in a group
    assert got == [36, 33]
