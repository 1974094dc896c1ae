"""Snapshot and restore of the timestep state: one kernel copies every array of it."""
import numpy as np
import pytest

from gip_b200 import cavity

FIELDS = ("u", "v", "w", "p", "mf", "rhs", "ax", "ax0", "gpx")


@pytest.mark.gpu
@pytest.mark.parametrize("edge", [2, 7, 13, 16])  # arrays below, across and at a chunk's end
@pytest.mark.parametrize("reorder", [False, True])
def test_restore_brings_every_array_back(gpu, edge, reorder):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(edge, re=100.0)
    E = DnsEngine(case, gamma=0.01, pcg_mode="fixed", maxit=20, reorder=reorder)
    E.advance(2)
    E.snapshot()
    kept = {k: E.field(k) for k in FIELDS}
    sc = E.scalars()
    E.advance(3)
    after = {k: E.field(k) for k in FIELDS}
    assert any(not np.array_equal(after[k], kept[k]) for k in FIELDS)
    E.snapshot(restore=True)
    for k in FIELDS:
        assert np.array_equal(E.field(k), kept[k]), k
    assert E.scalars() == sc
    E.advance(3)
    for k in FIELDS:
        assert np.array_equal(E.field(k), after[k]), k
