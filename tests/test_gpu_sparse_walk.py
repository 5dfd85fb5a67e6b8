"""The choice between the 3D walk by tiles and by threads, which follows the
community's density: sparse communities of many agents are walked by threads,
dense ones and few agents by tiles, with the CPU checker's bits either way,
across uploads that change the density and steps that make it."""
import numpy as np
import pytest

import conftest
from _oracle import OracleContext

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def state(rng, n, rho, L):
    """n agents at rho a unit volume around the middle of [0, L]^3."""
    side = (n / rho) ** (1 / 3)
    p = rng.uniform(-side / 2, side / 2, (3, n)) + L / 2
    return dict(x=p[0], y=p[1], z=p[2])


def walks(g):
    """Names of the force kernels of one step."""
    g.set_kernel_timing(True)
    g.step(1)
    names = [k for k, _ in g.kernel_times()]
    assert len(names) == g.kernels_per_step()
    g.set_kernel_timing(False)
    return {k for k in names if k.startswith("k_agent_de")}


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("alg", ["cell", "clvd"])
def test_walk_follows_density(gpu_lib, abi, prec, alg):
    n, L = 66000, 110.0
    rng = np.random.default_rng(3)
    kw = dict(dims=3, precision=abi.F32 if prec == "f32" else abi.F64, n_max=n + 4000,
              box_lo=(0.0,) * 3, box_hi=(L,) * 3, dt=0.001, cell_edge=3.3, k_rep=10.0, r_rep=2.0,
              k_att=1.0, r_att=3.0, neighbors=abi.NEIGH_CELL_LINKED)
    extra = {}
    if alg == "clvd":  # births and deaths: its steps walk the cells
        kw.update(neighbors=abi.NEIGH_CLVD, skin=3.3, rebuild_threshold=0.15, n_max_neighbors=400,
                  growth=1, fate=abi.FATE_VOLUME, v_div=2.0, div_sep=0.5, p_death=1e-3)
        extra = dict(v=rng.uniform(1, 2, n), g=rng.uniform(0.8, 1.2, n))
    cfg = abi.make_config(**kw)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=8)
    tiles = {"k_agent_de_tile"} if alg == "cell" else {"k_agent_de_tile", "k_agent_de"}
    # agents a cell: 4.6, 36 and 4.6 again
    for rho, want in ((0.1, {"k_agent_de"}), (1.0, tiles), (0.1, {"k_agent_de"})):
        st = dict(state(rng, n, rho, L), **extra)
        g.upload(st)
        o.upload(st)
        assert walks(g) == want
        g.step(2)
        o.step(3)
        a, b = g.download(), o.download()
        for k in "xyz":
            np.testing.assert_array_equal(a[k], b[k], err_msg=f"{rho} {k}")


def test_few_agents_stay_with_tiles(gpu_lib, abi):
    cfg = abi.make_config(dims=3, precision=abi.F64, n_max=60000, box_lo=(0.0,) * 3,
                          box_hi=(110.0,) * 3, dt=0.001, cell_edge=3.3, k_rep=10.0, r_rep=2.0,
                          k_att=1.0, r_att=3.0, neighbors=abi.NEIGH_CELL_LINKED)
    g = cbm.Context(cfg)
    g.upload(state(np.random.default_rng(4), 60000, 0.1, 110.0))
    assert walks(g) == {"k_agent_de_tile"}


def test_walk_changes_between_calls(gpu_lib, abi):
    """A sparse community that a drift to the origin makes dense (0.95 a step
    and axis): the walk changes with the counters of a later call."""
    n, L = 66000, 110.0
    cfg = abi.make_config(dims=3, precision=abi.F64, n_max=n, box_lo=(-L / 2,) * 3,
                          box_hi=(L / 2,) * 3, dt=0.05, cell_edge=3.3, k_rep=0.1, r_rep=2.0,
                          k_att=0.0, r_att=3.0, neighbors=abi.NEIGH_CELL_LINKED, drift_linear=1.0)
    st = state(np.random.default_rng(5), n, 0.1, 0.0)
    g, o = cbm.Context(cfg), OracleContext(abi, cfg, threads=8)
    g.upload(st)
    o.upload(st)
    assert walks(g) == {"k_agent_de"}
    for _ in range(3):
        g.step(4)
    assert walks(g) == {"k_agent_de_tile"}
    o.step(14)
    a, b = g.download(), o.download()
    for k in "xyz":
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
