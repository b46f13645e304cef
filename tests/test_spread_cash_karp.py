"""Cash-Karp launches that fill their warps however few candidates they have
(fixed steps over one field) or spread only small runs (tricubic grids): a
candidate's results are those of a run that fills the GPU."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, protons, random_grid

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("low", [1, 0.2])
@pytest.mark.parametrize("interpolation", [_abi.INTERPOLATION_TRILINEAR, _abi.INTERPOLATION_TRICUBIC])
def test_results_do_not_depend_on_how_warps_are_filled(precision, low, interpolation):
    from crpropa3_b200.engine import Plan
    grid = random_grid(np.random.default_rng(6), 8, 3e-13)
    plan = Plan(P.ChainSpec([P.GridField(grid, (0, 0, 0), (10 * U.kpc,) * 3, interpolation=interpolation)],
                            [P.Propagation(_abi.PROP_CK, 1e-4, low * U.kpc, 1 * U.kpc), P.MaxTrajectoryLength(6 * U.kpc)],
                            precision=precision))
    c = protons(np.random.default_rng(7), 592 * 32, emin=0.05 * U.EeV)
    full = c.to_device()
    plan.run(full)
    full = full.to_host()
    for n in (1, 592 * 8, 592 * 8 + 1):  # 8 and 9 candidates per warp
        dev = c.head(n).to_device()
        plan.run(dev)
        got = dev.to_host()
        for name in NAMES:
            np.testing.assert_array_equal(getattr(got, name), getattr(full, name)[:n], err_msg=f"{n} {name}")
