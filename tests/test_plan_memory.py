"""What a plan's grids take of the device memory."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, bp_fixed, protons

SHAPE = (256, 256, 128)
CELLS = 256 * 256 * 128


def _spec(precision, interpolation=_abi.INTERPOLATION_TRILINEAR, values=None, extra=()):
    values = np.zeros(SHAPE + (3,), np.float32) if values is None else values
    return P.ChainSpec([P.GridField(values, (0, 0, 0), (10 * U.kpc,) * 3, interpolation=interpolation)],
                       [bp_fixed(1 * U.kpc), P.MaxTrajectoryLength(100 * U.kpc), *extra], precision=precision)


def _plan_and_bytes(spec):
    import torch
    from crpropa3_b200.engine import Plan
    Plan(_spec(_abi.PRECISION_FP64, values=np.zeros((2, 2, 2, 3), np.float32)))  # the context's own memory
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = Plan(spec)
    return plan, before - torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("interpolation", [_abi.INTERPOLATION_TRICUBIC, _abi.INTERPOLATION_NEAREST_NEIGHBOUR])
def test_grids_that_no_kernel_gathers_in_pairs_hold_their_values_only(precision, interpolation):
    _, used = _plan_and_bytes(_spec(precision, interpolation))
    assert 12 * CELLS <= used <= 12 * CELLS + (8 << 20)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("n_extra", [0, 1, 2])
def test_same_results_where_the_pair_records_find_no_room(precision, n_extra):
    """[fixed BP, MaximumTrajectoryLength], with an observer and with two, over a periodic
    power-of-two grid: free memory decides the kernel, never the trajectories."""
    import torch
    from crpropa3_b200.engine import Plan
    rng = np.random.default_rng(3)
    values = (rng.standard_normal(SHAPE + (3,)) * 3e-13).astype(np.float32)
    extra = [P.ObserverSpec(features=[P.Feature(_abi.OBSERVER_PARTICLE_ID_VETO, particle_id=77)])] * n_extra
    spec = _spec(precision, values=values, extra=extra)
    c = protons(rng, 500, emin=0.1 * U.EeV, spread=1e7 * U.kpc)  # fractions of coordinates near 10^6
    small = _spec(precision, values=np.zeros((5, 3, 2, 3), np.float32), extra=extra)
    Plan(small).run(c.copy())  # the general grid's kernel, loaded while there is room for it
    want, got = c.copy(), c.copy()
    plan = Plan(spec)
    plan.run(want)
    del plan
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    room = 12 * CELLS + 32 * CELLS - (64 << 20)  # for the values, not for their records beside them
    fill = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        plan, used = _plan_and_bytes(spec)
        plan.run(got)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert used < 16 * CELLS
    for name, a in want.members().items():
        np.testing.assert_array_equal(getattr(got, name), a, err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
def test_pair_records_leave_room_for_the_rest_of_the_program(precision):
    """Free memory for a grid's values, its records and little more: the values only."""
    import torch
    torch.cuda.empty_cache()
    _plan_and_bytes(_spec(precision, values=np.zeros((2, 2, 2, 3), np.float32)))  # the context's own memory
    free = torch.cuda.mem_get_info()[0]
    room = 12 * CELLS + 48 * CELLS
    fill = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        _, used = _plan_and_bytes(_spec(precision))
    finally:
        del fill
        torch.cuda.empty_cache()
    assert 12 * CELLS <= used < 16 * CELLS
    _, used = _plan_and_bytes(_spec(precision))  # with the whole device free
    assert used >= 44 * CELLS
