"""The rods' step against the checker, bit for bit, at the sizes where its
lanes a rod change and where a block's last rods are missing, and on piles so
dense that a rod's queue of near candidates fills in the middle of its walk;
rods of zero length, rods in one line, NaN."""
import math

import numpy as np
import pytest

from test_gpu_rods import PARAMS, _colony, _compare

pytestmark = pytest.mark.gpu


def _config(abi, n, half, prec, full=False):
    return abi.make_rods_config(
        n, (-half - 2, -half - 2), (half + 2, half + 2), cell_edge=4.0,
        neighbors=abi.NEIGH_FULL if full else abi.NEIGH_CELL_LINKED,
        precision=abi.F32 if prec == "f32" else abi.F64, **PARAMS)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n", [7, 33, 2999, 7001, 21003])
def test_rods_lane_counts(gpu_lib, abi, prec, n):
    from conftest import cbm
    half = math.sqrt(n) * 0.9 + 1
    _compare(abi, cbm, _config(abi, n, half, prec), _colony(abi, n, 21, half), [1, 4])


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n,full", [(900, False), (700, True), (12000, False)])
def test_rods_piles(gpu_lib, abi, prec, n, full):
    """About eight rods per unit area: a hundred near candidates a rod."""
    from conftest import cbm
    half = math.sqrt(n / 8.0) / 2
    _compare(abi, cbm, _config(abi, n, half, prec, full), _colony(abi, n, 22, half), [1, 2])


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_rods_odd_shapes(gpu_lib, abi, prec):
    from conftest import cbm
    n, half = 1001, 30.0
    st = _colony(abi, n, 23, half)
    st["theta"][:300] = 0.3 + 1e-7 * np.arange(300)  # one direction, mostly one line
    st["x"][:300] = np.linspace(-28, 28, 300)
    st["y"][:300] = st["x"][:300] * math.tan(0.3)
    st["l"][300:400] = 0.0
    st["x"][500:510] = st["x"][510:520]  # coincident centres
    st["y"][500:510] = st["y"][510:520]
    st["vx"][600] = np.nan
    _compare(abi, cbm, _config(abi, n, half, prec), st, [1, 2])
