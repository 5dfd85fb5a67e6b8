"""The tiled 3D force walk against the CPU checker, bit for bit, at the sizes
and layouts where a tile goes wrong: counts around a warp, tiles over several
rows of cells, rings that wrap, cells beyond the box, agents far from their
tile, coincident agents, stiffnesses outside the branch-free form's range."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def ball(rng, n, radius, centre):
    u = rng.normal(size=(3, n))
    u *= radius * rng.uniform(size=n) ** (1 / 3) / np.linalg.norm(u, axis=0)
    return u + np.asarray(centre, float)[:, None]


def layout(name, rng):
    """(positions, box side) of a community."""
    if name.startswith("n"):  # a dense handful
        return ball(rng, int(name[1:]), 2.5, (30, 30, 30)), 60.0
    if name == "ring":  # about 300 agents a cell: several hundred words a tile
        return ball(rng, 4000, 4.5, (31.3, 29.2, 30.1)), 60.0
    if name == "rows":  # a few agents a cell: tiles span rows
        return rng.uniform(0, 40, (3, 9000)), 40.0
    if name == "mixed":  # a dense core in a sparse box
        return np.concatenate([ball(rng, 2000, 5.0, (11, 40, 40)),
                               rng.uniform(0, 80, (3, 2000))], axis=1), 80.0
    if name == "outside":  # agents beyond the box, in its last cells
        return rng.uniform(-6, 36, (3, 6000)), 30.0
    if name == "far":  # a second group a million units outside
        p = ball(rng, 800, 4.0, (15, 15, 15))
        q = ball(rng, 200, 3.0, (1.0e6, 15, 15))
        return np.concatenate([p, q], axis=1), 30.0
    p = ball(rng, 900, 4.0, (15, 15, 15))  # coincident pairs
    p[:, 1::90] = p[:, 0:-1:90]
    return p, 30.0


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("name", ["n1", "n31", "n32", "n33", "n129", "ring", "rows", "mixed",
                                  "outside", "far", "coincident"])
def test_tile_walk_bitexact(gpu_lib, abi, prec, name):
    rng = np.random.default_rng(11)
    p, L = layout(name, rng)
    cfg = abi.make_config(
        dims=3, precision=abi.F32 if prec == "f32" else abi.F64, n_max=p.shape[1],
        box_lo=(0.0,) * 3, box_hi=(L,) * 3, dt=0.002, neighbors=abi.NEIGH_CELL_LINKED,
        cell_edge=3.3, k_rep=10.0, r_rep=2.0, k_att=1.0, r_att=3.0)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    st = dict(x=p[0], y=p[1], z=p[2])
    g.upload(st)
    o.upload(st)
    for _ in range(1 if name == "coincident" else 3):
        g.step(1)
        o.step(1)
    a, b = g.download(), o.download()
    for k in "xyz":
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("k_rep,k_att,r_rep,r_att,to_att",
                         [(10.0, 1.0, 2.0, 3.0, True), (1e-15, 1e-16, 2.0, 3.0, False),
                          (1e13, 0.0, 2.0, 3.0, False), (10.0, 0.0, 2.0, 0.0, False),
                          (0.0, 3.0, 0.0, 2.9, False), (10.0, 1.0, 60.0, 61.0, False)])
def test_tile_walk_models(gpu_lib, abi, prec, k_rep, k_att, r_rep, r_att, to_att):
    rng = np.random.default_rng(12)
    p = ball(rng, 1500, 5.0, (20, 20, 20))
    cfg = abi.make_config(
        dims=3, precision=abi.F32 if prec == "f32" else abi.F64, n_max=1500,
        box_lo=(0.0,) * 3, box_hi=(40.0,) * 3, dt=0.001, neighbors=abi.NEIGH_CELL_LINKED,
        cell_edge=3.0, k_rep=k_rep, r_rep=r_rep, k_att=k_att, r_att=r_att,
        att_form=abi.ATT_TO_ATT if to_att else abi.ATT_FROM_REP)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=4)
    st = dict(x=p[0], y=p[1], z=p[2])
    g.upload(st)
    o.upload(st)
    g.step(2)
    o.step(2)
    a, b = g.download(), o.download()
    for k in "xyz":
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
