"""The Verlet-list walk and its list-writing walk against the CPU checker, bit
for bit: rows shorter than a group of four, remainders, rows that overrun the
walk's queue, agents near the skin, coincident agents, stiffnesses outside the
branch-free form's range, agents far outside the box."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def layout(name, dims, rng):
    n = 7001
    if name == "few":  # zero to a few partners
        return rng.uniform(0, 60.0 if dims == 3 else 200.0, (dims, n)), 200.0
    if name == "dense":  # 60 to 110 partners
        L = 24.0 if dims == 3 else 60.0
        return rng.uniform(0, L, (dims, n)), L
    if name == "grid":  # partners exactly at the skin
        m = 20 if dims == 3 else 84
        g = np.stack(np.meshgrid(*[np.arange(m) * 1.5 + 0.75] * dims), 0).reshape(dims, -1)
        return g[:, :n], m * 1.5
    p = rng.uniform(0, 30.0 if dims == 3 else 100.0, (dims, n))  # "odd"
    p[:, 1::500] = p[:, 0:-1:500]
    p[0, 2::700] += 2.0e6
    return p, 100.0


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("name,k_rep", [("few", 10.0), ("dense", 0.5), ("grid", 10.0),
                                        ("odd", 10.0), ("dense", 1e-15)])
def test_list_steps_bitexact(gpu_lib, abi, prec, dims, name, k_rep):
    rng = np.random.default_rng(5)
    p, L = layout(name, dims, rng)
    cfg = abi.make_config(
        dims=dims, precision=abi.F32 if prec == "f32" else abi.F64, n_max=p.shape[1],
        box_lo=(0.0,) * dims, box_hi=(L,) * dims, dt=0.002, neighbors=abi.NEIGH_CLVD,
        cell_edge=3.0, skin=3.0, rebuild_threshold=0.01, n_max_neighbors=256,
        k_rep=k_rep, r_rep=2.0, k_att=k_rep / 10, r_att=2.8)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    st = {k: p[d] for d, k in enumerate("xyz"[:dims])}
    g.upload(st)
    o.upload(st)
    steps = 1 if name == "odd" else 6
    g.step(steps)
    o.step(steps)
    a, b = g.download(), o.download()
    for k in st:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
