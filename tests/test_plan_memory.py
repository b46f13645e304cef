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
