"""The ordered exchange by lists (fields with many nodes per agent) and the
3D vector stencils against the CPU checker, bit for bit: nodes shared by more
agents than one pass orders, clamped stencils on the border, rows that are and
are not whole vectors, in one call of chained steps and step by step."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext
from scenarios import medium_colony

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("uptake", [0.0, 0.05])
@pytest.mark.parametrize("dims,nodes,n", [(3, 40, 1900), (3, 42, 1), (3, 37, 1200), (2, 120, 800),
                                          (1, 900, 100)])
def test_exchange_lists_bitexact(gpu_lib, abi, prec, uptake, dims, nodes, n):
    kw, st = medium_colony(abi, dims, N=n, L=float(nodes), n_medium=nodes, uptake=uptake,
                           precision=abi.F32 if prec == "f32" else abi.F64)
    rng = np.random.default_rng(5)
    for d, k in enumerate("xyz"[:dims]):
        x = np.array(st[k])
        x[: n // 4] = nodes / 3 + rng.uniform(0, 1.2, n // 4)   # dozens on a node
        x[n // 4: n // 3] = rng.uniform(-0.4, 0.4, n // 3 - n // 4)  # clamped stencils
        st[k] = x
    st["c"] = rng.uniform(0, 1, nodes ** dims)
    cfg = abi.make_config(**kw)
    assert n * 2 ** dims * 4 <= nodes ** dims  # the rule that takes the lists
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    g.upload(st)
    o.upload(st)
    g.step(1)
    g.step(19)
    o.step(20)
    a, b = g.download(), o.download()
    for k in ("x", "y", "z")[:dims] + ("c",) + ("gx", "gy", "gz")[:dims]:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
