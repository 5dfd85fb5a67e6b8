"""Batched communities: positions in and out through the page-locked ring
(empty and single-agent communities, more bytes than the ring holds, repeated
uploads before a step), and the branch-free force on lists of every remainder,
against the plain path, bit for bit."""
import numpy as np
import pytest

import conftest
from scenarios import make_descs, plain_config_for

cbm = conftest.cbm
pytestmark = pytest.mark.gpu


def test_exchange_roundtrip(gpu_lib, abi):
    rng = np.random.default_rng(3)
    sizes = [0, 1, 2, 255, 256, 257, 5000] + [9000] * 60  # 6.6 MB of positions
    base = abi.make_config(dims=3, precision=abi.F32, n_max=1, dt=0.01, neighbors=abi.NEIGH_CLVD,
                           integrator=abi.INT_EM, n_max_neighbors=64, skin=4.0, cell_edge=4.0)
    descs = [dict(n=n, box_lo=(0.0,) * 3, box_hi=(50.0,) * 3, k_rep=1.0, r_rep=2.0, k_att=0.1,
                  r_att=3.0, sigma=0.0, community=c) for c, n in enumerate(sizes)]
    b = cbm.Batch(base, make_descs(abi, descs))
    pos = [rng.uniform(0, 50, (3, n)).astype(np.float32) for n in sizes]
    for _ in range(2):
        for c, p in enumerate(pos):
            b.upload(c, p[0], p[1], p[2], step=7 + c)
    for c, p in enumerate(pos):
        got = b.download(c)
        assert got["step"] == 7 + c
        for k, want in zip("xyz", p):
            np.testing.assert_array_equal(got[k], want)


@pytest.mark.parametrize("n,L", [(1, 3.0), (2, 2.0), (5, 2.5), (37, 5.0), (300, 9.0), (2000, 20.0)])
def test_lists_match_plain(gpu_lib, abi, n, L):
    rng = np.random.default_rng(n)
    base = dict(dims=3, precision=abi.F32, n_max=1, dt=0.01, seed=5, neighbors=abi.NEIGH_CLVD,
                integrator=abi.INT_EM, n_max_neighbors=256, skin=3.6, cell_edge=3.6,
                rebuild_threshold=0.3, k_rep=10.0, r_rep=2.0, k_att=1.0, r_att=3.0)
    d = dict(n=n, box_lo=(0.0,) * 3, box_hi=(L,) * 3, k_rep=7.0, r_rep=2.0, k_att=1.3, r_att=3.0,
             sigma=0.05, community=3)
    p = rng.uniform(0, L, (3, n)).astype(np.float32)
    if n > 30:
        p[:, 5] = p[:, 6]  # a coincident pair
    b = cbm.Batch(abi.make_config(**base), make_descs(abi, [d]))
    b.set_tuning(threads=256, ctas_per_sm=1, skin=0.6)
    plain = cbm.Context(abi.make_config(**plain_config_for(abi, base, d, b.tuning().as_dict())))
    b.upload(0, *p)
    plain.upload(dict(x=p[0], y=p[1], z=p[2]))
    for steps in (1, 1, 9):
        b.step(steps)
        plain.step(steps)
        got, want = b.download(0), plain.download()
        for k in "xyz":
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
