"""The ordered exchange by lists where thousands of agents meet on one node:
the CPU checker's bits, and a time that grows with the agents, not with their
square."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext
from scenarios import medium_colony

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def crowd(abi, dims, nodes, n, where, prec, **kw):
    """n agents on one node: inside (one stencil), or beyond a corner of the
    field, whose node then has all 2^dims entries of each."""
    kw, st = medium_colony(abi, dims, N=n, L=float(nodes), n_medium=nodes,
                           precision=abi.F32 if prec == "f32" else abi.F64, **kw)
    rng = np.random.default_rng(15)
    for k in "xyz"[:dims]:
        st[k] = rng.uniform(0.51, 1.49, n) + nodes // 3 if where == "node" else rng.uniform(-9, -2, n)
    if dims == 1:  # no two agents at the same Float32 place, where the pair force is undefined
        st["x"] = rng.permutation(np.linspace(0.51, 1.49, n)) + nodes // 3
    st["c"] = rng.uniform(0, 1, nodes ** dims)
    assert n * 2 ** dims * 4 <= nodes ** dims  # the rule that takes the lists
    return kw, st


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("uptake", [0.0, 0.05])
@pytest.mark.parametrize("dims,nodes,n,where", [
    (3, 40, 16, "node"), (3, 40, 17, "node"), (3, 40, 33, "node"), (3, 40, 1999, "node"),
    (3, 40, 1999, "corner"), (2, 120, 900, "corner"), (1, 9000, 1000, "node")])
def test_crowded_node_bitexact(gpu_lib, abi, prec, uptake, dims, nodes, n, where):
    kw, st = crowd(abi, dims, nodes, n, where, prec, uptake=uptake)
    cfg = abi.make_config(**kw)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    g.upload(st)
    o.upload(st)
    g.step(2)
    o.step(2)
    a, b = g.download(), o.download()
    for k in ("x", "y", "z")[:dims] + ("c",):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("where", ["node", "corner"])
def test_crowded_node_time(gpu_lib, abi, where):
    """4000 agents: a node's list has m = 4000 entries (32000 at the corner).
    Read m / 4 times over it is at least 4e6 (2.6e8) dependent reads, 80 ms (5
    s) at 40 cycles each; searched and sorted it is some 32000 reads spread
    over a block and 120 network steps of at most 16 rounds a thread, a few
    milliseconds for the eight nodes."""
    kw, st = crowd(abi, 3, 64, 4000, where, "f32", dt=1e-9)
    g = cbm.Context(abi.make_config(**kw))
    g.upload(st)
    g.set_kernel_timing(True)
    g.step(1)
    g.step(1)
    times = dict(g.kernel_times())
    assert times["k_medium_apply"] < 40.0, times
