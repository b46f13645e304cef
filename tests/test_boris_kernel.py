"""The kernel of the chain [fixed-step PropagationBP, MaximumTrajectoryLength]
over a periodic power-of-two grid: FP64 bit for bit against the oracle, the
mixed form against the module-list kernel of the same chain."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from crpropa3_b200.state import RecordArrays
from helpers import U, protons

NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")


def _spec(precision, brms=3e-13, per_candidate=False, length=700, extra=False):
    rng = np.random.default_rng(5)
    grid = (rng.standard_normal((16, 8, 4, 3)) * brms).astype(np.float32)
    grid[3:5] = 0  # field-free cells
    grid[9, :, :, 1] = 0  # and one vanishing component
    mods = [P.Propagation(_abi.PROP_BP, 0.42, 1 * U.kpc, 1 * U.kpc),
            P.MaxTrajectoryLength(length * U.kpc, per_candidate=per_candidate, record=True)]
    if extra:  # a fourth module that never acts: the module-list kernel
        mods += [P.ObserverSpec(features=[P.Feature(_abi.OBSERVER_PARTICLE_ID_VETO, particle_id=77)])] * 2
    return P.ChainSpec([P.GridField(grid, (1 * U.kpc, 0, 0), (10 * U.kpc,) * 3)], mods, precision=precision)


def _candidates(n):
    rng = np.random.default_rng(n)
    c = protons(rng, n, emin=0.02 * U.EeV, emax=50 * U.EeV, spread=300 * U.kpc)
    c.charge[::7] = 0
    c.active[3::11] = 0
    k = np.arange(n)
    for axis, name in enumerate(("dx", "dy", "dz")):  # directions with vanishing components
        getattr(c, name)[k % 5 == 2] = float(axis == 1)
    far = k % 13 == 4  # directions away from unit length
    for name in ("dx", "dy", "dz"):
        getattr(c, name)[far] *= 1.5
    return c


def _run(spec, c, **kw):
    from crpropa3_b200.engine import Plan
    rec = RecordArrays(c.n)
    got = c.copy()
    stats = Plan(spec).run(got, records=rec, **kw)
    return got, rec.sorted(), stats


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 129, 700])
@pytest.mark.parametrize("per_candidate", [False, True])
@pytest.mark.parametrize("steps_per_launch", [0, 1, 64])
def test_fp64_matches_the_oracle(oracle, n, per_candidate, steps_per_launch):
    spec = _spec(_abi.PRECISION_FP64, per_candidate=per_candidate)
    c = _candidates(n)
    if per_candidate:
        c.max_length = np.random.default_rng(1).uniform(0, 600, n) * U.kpc
    ref = c.copy()
    rec = RecordArrays(n)
    oracle.run(spec, ref, records=rec)
    got, records, _ = _run(spec, c, steps_per_launch=steps_per_launch)
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got, name), getattr(ref, name), err_msg=name)
    for name, want in rec.sorted().items():
        np.testing.assert_array_equal(records[name], want, err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("n,cap", [(701, 0), (701, 1), (701, 130), (24001, 0)])  # with and without asking ahead
def test_same_as_the_module_list_kernel(precision, n, cap):
    c = _candidates(n)
    a, ra, sa = _run(_spec(precision), c, max_steps=cap)
    b, rb, sb = _run(_spec(precision, extra=True), c, max_steps=cap)
    for name in NAMES:
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name), err_msg=name)
    for name in ra:
        np.testing.assert_array_equal(ra[name], rb[name], err_msg=name)
    assert (sa.particle_steps, sa.tries, sa.field_evaluations) == (sb.particle_steps, sb.tries, sb.field_evaluations)


@pytest.mark.gpu
def test_extreme_charges_and_energies(oracle):
    """Beyond the range of the division-free push the chain is run as elsewhere."""
    c = _candidates(64)
    c.charge[:] = np.geomspace(1e-90, 1e90, 64)
    c.energy[32:] = np.geomspace(1e-70, 1e80, 32)
    spec = _spec(_abi.PRECISION_FP64, length=40)
    ref = c.copy()
    oracle.run(spec, ref)
    got, _, _ = _run(spec, c)
    for name in NAMES:
        np.testing.assert_array_equal(getattr(got, name), getattr(ref, name), err_msg=name)
