"""A single galactic field is called directly, a list of fields through the sum
over its components: the same bits with a vanishing uniform field beside it."""
import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from helpers import U, protons

FIELDS = {"jf12": lambda: P.JF12Field(), "uf23": lambda: P.UF23Field(_abi.UF23_TWISTX), "pt11": lambda: P.PT11Field(),
          "tf17": lambda: P.TF17Field(), "kst24": lambda: P.KST24Field()}


@pytest.mark.gpu
@pytest.mark.parametrize("field", sorted(FIELDS))
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("prop", [(_abi.PROP_CK, 1e-4, 100), (_abi.PROP_BP, 100, 100)])
def test_single_field_matches_the_component_sum(field, precision, prop):
    from crpropa3_b200.engine import Plan
    mods = [P.Propagation(prop[0], 1e-4, prop[1] * U.pc, prop[2] * U.pc), P.MaxTrajectoryLength(12 * U.kpc),
            P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0.0, 0.0, 0.0), 15 * U.kpc, True, False)]
    c = protons(np.random.default_rng(2), 300, spread=9 * U.kpc, origin=(-1 * U.kpc, 0, 0))
    got = []
    for fields in ([FIELDS[field]()], [FIELDS[field](), P.UniformField((0.0, 0.0, 0.0))]):
        d = c.to_device()
        Plan(P.ChainSpec(fields, mods, precision=precision)).run(d)
        got.append(d.to_host())
    for name in ("x", "y", "z", "dx", "dy", "dz", "trajectory_length", "next_step", "flags", "step_count"):
        np.testing.assert_array_equal(getattr(got[0], name), getattr(got[1], name), err_msg=name)
