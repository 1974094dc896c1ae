"""Calls when the device's memory runs out: refused with a status, nothing written, and whole again
once there is memory."""
import contextlib

import numpy as np
import pytest
import torch

from gip_b200 import _lib, cavity

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory_left(nbytes):
    """Holds the device's free memory but for about `nbytes` (nothing of it is touched)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        for _ in range(4):
            take = torch.cuda.mem_get_info()[0] - nbytes
            if take > (2 << 20):
                held.append(torch.empty(take >> 21 << 21, dtype=torch.uint8, device="cuda"))
        yield
    finally:
        del held
        torch.cuda.synchronize()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("left_mb", [4, 24, 48, 80])  # of the 90 MB that the 64^3 state takes
def test_snapshot_that_found_no_memory_can_be_taken_later(gpu, left_mb):
    from gip_b200.device import DnsEngine
    case, _ = cavity.generate(64, re=100.0)
    E = DnsEngine(case, gamma=0.01, pcg_mode="fixed", maxit=5)
    E.advance(2)
    kept = {k: E.field(k) for k in ("u", "p", "mf")}
    with memory_left(left_mb << 20):
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
