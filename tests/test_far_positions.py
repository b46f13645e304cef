"""Grid coordinates beyond 2^31 cells, where the cell index saturates: a periodic
power-of-two grid (index by addition, wrapped with a mask) against the same
field in a grid of three periods (index by conversion, wrapped by division)."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, protons, random_grid

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")


@pytest.mark.gpu
# (the mixed fixed-step push over grids that are not powers of two rounds its cell
# fractions differently: its adaptive step stands for it)
@pytest.mark.parametrize("precision,prop", [(_abi.PRECISION_FP64, (_abi.PROP_BP, 1, 1)),
                                            (_abi.PRECISION_FP64, (_abi.PROP_CK, 0.5, 5)),
                                            (_abi.PRECISION_MIXED, (_abi.PROP_BP, 0.5, 5)),
                                            (_abi.PRECISION_MIXED, (_abi.PROP_CK, 0.5, 5))])
def test_saturated_cell_indices(precision, prop):
    from crpropa3_b200.engine import Plan
    grid = random_grid(np.random.default_rng(8), 16, 3e-13)
    rng = np.random.default_rng(9)
    n = 96
    c = protons(rng, n, emin=0.1 * U.EeV)
    cells = rng.uniform(1, 2, (n, 3)) * rng.choice([-1, 1], (n, 3)) * 2.0 ** rng.uniform(29, 40, (n, 1))
    cells[::3, 1:] = rng.uniform(-8, 8, (len(cells[::3]), 2))  # far on one axis only
    c.set_position(cells * 10 * U.kpc)
    got = []
    for values in (grid, np.tile(grid, (3, 3, 3, 1))):
        plan = Plan(P.ChainSpec([P.GridField(values, (0, 0, 0), (10 * U.kpc,) * 3)],
                                [P.Propagation(prop[0], 1e-4, prop[1] * U.kpc, prop[2] * U.kpc),
                                 P.MaxTrajectoryLength(20 * U.kpc)], precision=precision))
        dev = c.to_device()
        plan.run(dev)
        got.append(dev.to_host())
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got[0], name), getattr(got[1], name), err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("far", [1e6, 1e12])
def test_persistent_fixed_push_rounds_its_coordinates(far):
    """Persistent launches of the mixed fixed push over a general grid: the cell fractions of
    the periodic power-of-two grid, far from the origin too, and no NaN at 10^300 m."""
    from crpropa3_b200.engine import Plan
    grid = random_grid(np.random.default_rng(8), 16, 3e-13)
    rng = np.random.default_rng(10)
    c = protons(rng, 500, emin=0.1 * U.EeV)
    c.set_position(rng.uniform(-far, far, (500, 3)) * 10 * U.kpc)
    got = []
    for values in (grid, np.tile(grid, (3, 3, 3, 1))):
        plan = Plan(P.ChainSpec([P.GridField(values, (0, 0, 0), (10 * U.kpc,) * 3)],
                                [P.Propagation(_abi.PROP_BP, 0.42, 1 * U.kpc, 1 * U.kpc), P.MaxTrajectoryLength(60 * U.kpc)],
                                precision=_abi.PRECISION_MIXED))
        dev = c.to_device()
        plan.run(dev, mode=_abi.MODE_PERSISTENT)
        got.append(dev.to_host())
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got[0], name), getattr(got[1], name), err_msg=name)
    c.x[::3] = 1e300
    plan.run(c, mode=_abi.MODE_PERSISTENT)
    assert np.isfinite(c.position()).all()
