"""The tiled 3D force walk in other units of length, and with cells of many
cutoffs, against the CPU checker, bit for bit; and the adjoint, whose recorded
pairs come from the same walk.  Every length of a community is multiplied by
the same factor: the pairs within the cutoff stay the same ones."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext, oracle_adjoint_dual

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def ball(rng, n, radius, centre):
    u = rng.normal(size=(3, n))
    u *= radius * rng.uniform(size=n) ** (1 / 3) / np.linalg.norm(u, axis=0)
    return u + np.asarray(centre, float)[:, None]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("unit", [1e-3, 2e-4, 6e-5, 1e-5, 1e-19])
@pytest.mark.parametrize("name", ["ring", "rows", "wide cells", "wider cells"])
def test_other_units(gpu_lib, abi, prec, unit, name):
    rng = np.random.default_rng(21)
    L, edge = 60.0, 3.3
    if name == "rows":  # a few agents a cell: tiles span rows of cells
        p, L = rng.uniform(4, 40, (3, 9000)), 44.0
    else:
        p = ball(rng, 3000, 4.5, (31.3, 29.2, 30.1))
        edge = {"ring": 3.3, "wide cells": 20.0, "wider cells": 60.0}[name]  # cutoff 3, or 1
    cut = 3.0 if name in ("ring", "rows") else 1.0
    cfg = abi.make_config(
        dims=3, precision=abi.F32 if prec == "f32" else abi.F64, n_max=p.shape[1],
        box_lo=(0.0,) * 3, box_hi=(L * unit,) * 3, dt=0.002, neighbors=abi.NEIGH_CELL_LINKED,
        cell_edge=edge * unit, k_rep=10.0, r_rep=cut * unit * 2 / 3, k_att=1.0, r_att=cut * unit)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    st = dict(x=p[0] * unit, y=p[1] * unit, z=p[2] * unit)
    g.upload(st)
    o.upload(st)
    for _ in range(3):
        g.step(1)
        o.step(1)
    a, b = g.download(), o.download()
    for k in "xyz":
        assert np.any(b[k] != st[k].astype(b[k].dtype))
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("unit", [1.0, 2e-4])
def test_adjoint_in_other_units(gpu_lib, abi, unit):
    rng = np.random.default_rng(22)
    n, steps = 700, 10
    x0 = list(ball(rng, n, 3.5, (15, 15, 15)) * unit)
    target = [x + 0.1 * unit * rng.normal(size=n) for x in x0]
    kw = dict(dims=3, precision=abi.F64, n_max=n, box_lo=(0.0,) * 3, box_hi=(30.0 * unit,) * 3,
              dt=1e-4, neighbors=abi.NEIGH_CELL_LINKED, cell_edge=3.3 * unit,
              integrator=abi.INT_EULER, k_rep=10.0, r_rep=2.0 * unit, k_att=1.0, r_att=3.0 * unit,
              att_form=abi.ATT_FROM_REP, n_max_neighbors=n)
    cfg = abi.make_config(**kw)
    adj, o = cbm.Adjoint(cfg), OracleContext(abi, cfg, threads=4)
    o.upload(dict(x=x0[0], y=x0[1], z=x0[2]))
    o.step(steps)
    s = o.download()
    for d, x in enumerate(adj.forward(x0, steps)):
        np.testing.assert_array_equal(x, s["xyz"[d]])
    res = adj.run(x0, target, steps, checkpoint_every=4)
    seeds = [(5, 0), (123, 1), (699, 2)]
    loss, grad, dx = oracle_adjoint_dual(abi, cfg, x0, target, steps, seeds=seeds)
    assert abs(res["loss"] - loss) <= 1e-10 * abs(loss)
    # the adjoint's Float64 sums against dual numbers: 1e-6, as for its other problems
    np.testing.assert_allclose(res["dtheta"], grad, rtol=1e-6)
    scale = max(np.max(np.abs(d)) for d in res["dx0"])
    for (i, ax), v in zip(seeds, dx):
        assert abs(res["dx0"][ax][i] - v) <= 1e-6 * scale
