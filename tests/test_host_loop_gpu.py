"""host_loop_pcg refuses what its fused calls refuse one by one."""
import numpy as np
import pytest
import torch

from gip_b200.formats import Csr

pytestmark = pytest.mark.gpu


def test_start_shorter_than_the_operators_columns_is_refused(gpu):
    # x0 broadcasts to a two-dimensional x, so x has the operator's columns and x0 has not: the
    # search direction, a copy of x0, is too short for the product
    from gip_b200 import device as dv
    n, ncols = 64, 120
    col = np.stack([np.arange(n), np.arange(n) + ncols - n], 1).ravel()
    val = np.tile([4.0, 0.0], n)
    A = dv.DeviceMatrix(Csr(n, ncols, np.arange(0, 2 * n + 1, 2, dtype=np.int32),
                            col.astype(np.int32), val))
    D = dv.DeviceMatrix(Csr(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                            np.full(n, 0.25)))
    f = dict(dtype=torch.float64, device="cuda")
    x0, x, b, dinv = torch.zeros(n, **f), torch.zeros(2, n, **f), torch.ones(n, **f), torch.full((n,), 0.25, **f)
    with pytest.raises(ValueError):
        dv.host_loop_pcg(A, D, dinv, b, x, x0, 3)
    A.close()  # not left to the collector: the caught error's frames hold them
    D.close()
