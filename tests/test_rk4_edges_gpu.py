"""The RK4 step of both precisions on the smallest grid and on ragged ones.

The stage kernels work on tiles of 128 cells (FP64 32 x 4, mixed 128 x 1) with operands staged
or prefetched by the tile, so the rows that end inside a tile, just after one, and the smallest
grid, with two interior levels, are where an index can go wrong.  A batch's other tile shapes
are test_batch_gpu.py's.  Tolerances, from the states and forces of one step on the
grids of test_parity_gpu.py and test_mixed_gpu.py: FP64 1e-12; mixed 1e-8 for the
prognostic fields and 1e-4 for the acting forces.  The time-level copy is exact.
"""
import numpy as np
import pytest

from athad_cond_b200 import GpuAtmosphere, make_state
from athad_cond_b200._abi import Precision, config_params
from oracle_binding import OracleState

pytestmark = pytest.mark.gpu

PROG = ["t", "u", "v", "w", "c", "cloud", "ice", "gr", "co2", "tke", "dis"]


def relerr(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.mark.parametrize("precision", [Precision.FP64, Precision.MIXED])
@pytest.mark.parametrize("grid", [(4, 5, 5), (5, 7, 33), (9, 17, 129), (6, 9, 131), (7, 11, 257)])
def test_rk4_step_on_ragged_grids(grid, precision):
    p = config_params()
    st = make_state(*grid, seed=31)
    rng = np.random.default_rng(31)
    st["P_rain"] = 1e-4 * rng.random(grid)
    st["P_snow"] = 1e-4 * rng.random(grid)
    o = OracleState(st, p)
    o.rk4(dt=4e-5, buoyancy_ramp=0.5)
    p.precision = int(precision)
    state_tol, force_tol = (1e-12, 1e-12) if precision == Precision.FP64 else (1e-8, 1e-4)
    with GpuAtmosphere(*grid, p) as g:
        g.upload_state(st)
        g.solveRungeKutta_Atmosphere_Turb(4e-5, 1.0, 0.5, store_n_level=True)
        for n in PROG:
            new = g.download(n)
            assert relerr(new, o.f[n]) <= state_tol, n
            assert np.array_equal(g.download(n + "n"), new), n
        for n in ("aux_u", "aux_v", "aux_w"):
            assert relerr(g.download(n), o.f[n]) <= force_tol, n
        for n in ("P_rain", "P_snow"):
            assert np.array_equal(g.download(n + "n"), st[n]), n
