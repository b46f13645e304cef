"""Chains over lists of fields: kernels with the field sum inlined (full warps,
Boris push) and called (few candidates per warp, adaptive Cash-Karp, persistent
launches) give the same bits."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, protons, random_grid

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")
PROPS = [(_abi.PROP_CK, 1, 1), (_abi.PROP_CK, 0.5, 5), (_abi.PROP_BP, 1, 1), (_abi.PROP_BP, 0.5, 5)]


def _spec(fields, prop, precision):
    kind, lo, hi = prop
    return P.ChainSpec(fields, [P.Propagation(kind, 1e-4, lo * U.kpc, hi * U.kpc), P.MaxTrajectoryLength(15 * U.kpc),
                                P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0, 0, 0), 55 * U.kpc, True, False),
                                P.BoundarySpec(_abi.BOUNDARY_SPHERICAL, (0, 0, 0), size=70 * U.kpc)],
                       precision=precision)


def _fields(kind):
    grid = random_grid(np.random.default_rng(2), 8, 3e-13)
    if kind == "wrapped":
        return [P.GridField(grid, (0, 0, 0), (10 * U.kpc,) * 3, periodic=((0, 0, 0), (80 * U.kpc,) * 3, False))]
    return [P.UniformField((1e-13, -2e-13, 0)), P.GridField(grid, (0, 0, 0), (10 * U.kpc,) * 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("prop", PROPS)
@pytest.mark.parametrize("kind", ["list", "wrapped"])
def test_results_do_not_depend_on_the_launch(precision, prop, kind):
    """31 and 32 candidates per warp (592 schedulers), a partial block, one warp, persistent."""
    from crpropa3_b200.engine import Plan
    plan = Plan(_spec(_fields(kind), prop, precision))
    c = protons(np.random.default_rng(3), 592 * 31 + 1, emin=0.1 * U.EeV, emax=20 * U.EeV)
    c.charge[::17] = 0
    full = c.to_device()
    plan.run(full)
    full = full.to_host()
    for n, options in ((592 * 31, {}), (33, {}), (700, {"mode": _abi.MODE_PERSISTENT})):
        dev = c.head(n).to_device()
        plan.run(dev, **options)
        got = dev.to_host()
        for name in NAMES:
            np.testing.assert_array_equal(getattr(got, name), getattr(full, name)[:n], err_msg=f"{n} {name}")


@pytest.mark.gpu
@pytest.mark.parametrize("prop", PROPS)
def test_full_warps_match_the_oracle(oracle_crpow, prop):
    from crpropa3_b200.engine import Plan
    spec = _spec(_fields("list"), prop, _abi.PRECISION_FP64)
    c = protons(np.random.default_rng(4), 592 * 32, emin=0.1 * U.EeV, emax=20 * U.EeV)
    dev = c.to_device()
    Plan(spec).run(dev)
    got, ref = dev.to_host(), c.head(400)
    oracle_crpow.run(spec, ref)
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got, name)[:400], getattr(ref, name), err_msg=name)
