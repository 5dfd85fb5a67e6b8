"""DGADI lines against the CPU checker, bit for bit, at the lengths where the
grouped reads end (4 to 13 nodes) and where blocks hold lines of several
fields, and for media whose field is mostly zero and subnormal."""
import numpy as np
import pytest

import conftest
from _oracle import OracleMedium

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims,n,fields", [(3, (4, 5, 6), 1), (3, (7, 8, 9), 3), (3, (10, 11, 70), 2),
                                           (2, (400, 13, 1), 8), (2, (12, 420, 1), 5),
                                           (2, (330, 310, 1), 2), (3, (66, 60, 50), 2)])
def test_dgadi_lines_bitexact(gpu_lib, abi, dims, n, fields, prec):
    rng = np.random.default_rng(sum(n))
    nodes = int(np.prod(n[:dims]))
    cfg = abi.make_medium_config(dims, n, (0.0,) * 3, (1.0, 1.3, 0.8), 0.003,
                                 list(rng.uniform(0.2, 3.0, fields)),
                                 list(rng.uniform(0.0, 0.4, fields)), c_max=1.2,
                                 precision=abi.F32 if prec == "f32" else abi.F64)
    u = rng.uniform(0.0, 1.0, (fields, nodes))
    if fields == 2:
        u[1] = 0.0  # grows from the source: zeros, subnormals, then values
    src = np.zeros(nodes)
    src[rng.integers(0, nodes, 3)] = 0.7
    g, o = abi.DGADIMedium(cfg), OracleMedium(abi, cfg)
    g.upload(u, src)
    o.upload(u, src)
    g.step(1)
    g.step(4)
    o.step(5)
    np.testing.assert_array_equal(g.download()[0].reshape(fields, -1),
                                  np.asarray(o.download()[0]).reshape(fields, -1))
