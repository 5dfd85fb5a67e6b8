"""The adjoint object's forward sweep keeps no pairs, and needs no memory for
them."""
import numpy as np
import pytest

import conftest
from scenarios import adjoint_problem

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def test_forward_has_no_room_for_pairs(gpu_lib, abi):
    kw, x0, _ = adjoint_problem(abi, N=300, L=15.0)
    ref = cbm.Adjoint(abi.make_config(**kw)).forward(x0, 5)
    # rows of 2^29 partners would take 644 GB
    adj = cbm.Adjoint(abi.make_config(**dict(kw, n_max_neighbors=1 << 29)))
    for a, b in zip(adj.forward(x0, 5), ref):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(cbm.CbmError):
        adj.run(x0, x0, 5)
