"""PlaneWaveTurbulence evaluated by a block for its candidates: the same bits as
the thread-by-thread sum (the persistent kernels), for every propagator, odd
mode counts, partial blocks and phases beyond the fixed-point range."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P, workloads as W
from helpers import U, protons

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("prop", [(_abi.PROP_BP, 1, 1), (_abi.PROP_BP, 0.1, 5), (_abi.PROP_CK, 0.1, 5)])
@pytest.mark.parametrize("n,modes", [(1, 33), (33, 50), (129, 8), (700, 301), (19000, 40), (40000, 33)])
def test_block_sums_match_the_thread_by_thread_sums(precision, prop, n, modes):
    from crpropa3_b200.engine import Plan
    spectrum = (1 * U.nG, 20 * U.kpc, 200 * U.kpc, 200 * U.kpc, 5.0 / 3.0, 4.0)
    waves = P.PlaneWaveField(*W.plane_wave_modes(*spectrum, modes, 11), spectrum=spectrum, seed=11)
    mods = [P.Propagation(prop[0], 1e-4, prop[1] * U.kpc, prop[2] * U.kpc), P.MaxTrajectoryLength(12 * U.kpc),
            P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0.0, 0.0, 0.0), 60 * U.kpc, True, False)]
    plan = Plan(P.ChainSpec([waves], mods[:2 + n % 2], precision=precision))
    c = protons(np.random.default_rng(n), n, emin=0.1 * U.EeV)
    c.charge[::9] = 0
    if modes == 50:
        c.x[5] = 1e13 * U.kpc  # beyond the fixed-point phase
    a, b = c.to_device(), c.to_device()
    plan.run(a)
    plan.run(b, mode=_abi.MODE_PERSISTENT)
    a, b = a.to_host(), b.to_host()
    for name in NAMES:
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name), err_msg=name)
