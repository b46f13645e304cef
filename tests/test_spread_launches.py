"""Chunked launches that spread few candidates over many warps, the adaptive
chains' loop over tries, and the pair-record gathers: bit for bit against the
oracle (FP64) and against the same candidates inside a larger run (mixed)."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, grid_chain, protons, random_grid

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "current_step", "next_step",
         "active", "flags", "step_count")


def _chain(shape, prop, precision, reflective=False, origin=(0, 0, 0)):
    rng = np.random.default_rng(17)
    grid = (rng.standard_normal(shape + (3,)) * 3e-13).astype(np.float32)
    kind, lo, hi = prop
    return grid_chain(grid, 10 * U.kpc, P.Propagation(kind, 1e-4, lo * U.kpc, hi * U.kpc), 300 * U.kpc,
                      observer_radius=150 * U.kpc, precision=precision, reflective=reflective, origin=origin)


CHAINS = [((16, 16, 16), (_abi.PROP_CK, 0.1, 20), False), ((16, 16, 16), (_abi.PROP_BP, 0.1, 20), False),
          ((16, 8, 4), (_abi.PROP_BP, 1, 1), False), ((5, 7, 3), (_abi.PROP_CK, 0.1, 20), False),
          ((5, 7, 3), (_abi.PROP_BP, 0.1, 20), True), ((1, 2, 9), (_abi.PROP_BP, 1, 1), True)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,prop,reflective", CHAINS)
@pytest.mark.parametrize("n", [1, 33, 593])
def test_small_runs_match_the_oracle(oracle_crpow, shape, prop, reflective, n):
    from crpropa3_b200.engine import Plan
    rng = np.random.default_rng(n)
    spec = _chain(shape, prop, _abi.PRECISION_FP64, reflective)
    c = protons(rng, n, emin=0.05 * U.EeV, emax=50 * U.EeV, spread=100 * U.kpc)
    c.charge[: n // 8] = 0  # neutral candidates beside charged ones
    ref = c.copy()
    oracle_crpow.run(spec, ref)
    dev = c.to_device()
    Plan(spec).run(dev)
    got = dev.to_host()
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got, name), getattr(ref, name), err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,prop,reflective", CHAINS)
def test_mixed_results_do_not_depend_on_the_launch(shape, prop, reflective):
    """The first candidates of a run that fills the GPU, alone and one by one."""
    from crpropa3_b200.engine import Plan
    plan = Plan(_chain(shape, prop, _abi.PRECISION_MIXED, reflective))
    c = protons(np.random.default_rng(3), 40000, emin=0.05 * U.EeV, emax=50 * U.EeV, spread=100 * U.kpc)
    full = c.to_device()
    plan.run(full)
    full = full.to_host()
    for n in (1, 31, 700):
        dev = c.head(n).to_device()
        plan.run(dev)
        got = dev.to_host()
        for name in NAMES:
            np.testing.assert_array_equal(getattr(got, name), getattr(full, name)[:n], err_msg=name)


@pytest.mark.gpu
def test_positions_many_periods_away(oracle):
    """Grid coordinates up to 2^30 cells: the cell index keeps its low bits."""
    from crpropa3_b200.engine import Plan
    rng = np.random.default_rng(9)
    spec = _chain((16, 16, 16), (_abi.PROP_BP, 1, 1), _abi.PRECISION_FP64, origin=(3 * U.kpc, -7 * U.kpc, 0))
    c = protons(rng, 64, spread=1.0)
    c.set_position(rng.uniform(-1, 1, (64, 3)) * 2.0 ** np.arange(64)[:, None].clip(0, 30) * 10 * U.kpc)
    ref = c.copy()
    oracle.run(spec, ref)
    dev = c.to_device()
    Plan(spec).run(dev)
    got = dev.to_host()
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got, name), getattr(ref, name), err_msg=name)
