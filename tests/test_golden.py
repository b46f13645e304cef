"""The oracle (CPU) and the device (GPU) against golden fixtures generated
from the reference itself by tests/golden/make_golden.py."""
import os

import numpy as np
import pytest

from helpers import P, RecordArrays, U, _abi, bp_fixed, ck, grid_chain, random_grid
from crpropa3_b200.state import CandidateArrays

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reference_golden.npz")
STATE = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time",
         "current_step", "next_step", "active", "flags")
PROPS = {
    "bp_fixed": (lambda: bp_fixed(1 * U.kpc), False),
    "bp_fixed_reflective": (lambda: bp_fixed(1 * U.kpc), True),
    "bp_adaptive": (lambda: P.Propagation(_abi.PROP_BP, 1e-3, 0.1 * U.kpc, 10 * U.kpc), False),
    "ck_fixed": (lambda: ck(1e-4, 1 * U.kpc, 1 * U.kpc), False),
    "ck_adaptive": (lambda: ck(1e-4, 0.1 * U.kpc, 10 * U.kpc), False),
}


@pytest.fixture(scope="module")
def golden():
    return dict(np.load(GOLDEN))


def _case(golden, name):
    rng = np.random.default_rng(sum(map(ord, name)))
    grid = random_grid(rng, 16)
    prop, refl = PROPS[name]
    spec = grid_chain(grid, 10 * U.kpc, prop(), 1 * U.Mpc, observer_radius=0.4 * U.Mpc, reflective=refl)
    n = golden[f"{name}/in_x"].shape[0]
    c = CandidateArrays(n)
    for m in STATE + ("id", "charge", "energy"):
        getattr(c, m)[:] = golden[f"{name}/in_{m}"]
    return spec, c


@pytest.mark.parametrize("name", list(PROPS))
def test_oracle_reproduces_golden(oracle, golden, name):
    spec, c = _case(golden, name)
    rec = RecordArrays(256)
    steps, _ = oracle.run(spec, c, rec)
    assert steps == golden[f"{name}/steps"][0]
    for m in STATE:
        np.testing.assert_array_equal(getattr(c, m), golden[f"{name}/out_{m}"], err_msg=m)
    for k, v in rec.sorted().items():
        np.testing.assert_array_equal(v, golden[f"{name}/rec_{k}"], err_msg=k)


def test_oracle_fields_random_source_charge_golden(oracle, golden):
    grid, pos = golden["field/grid"], golden["field/pos"]
    for key, f in (("periodic", dict()), ("reflective", dict(reflective=True)), ("clip", dict(clip_volume=True))):
        spec = P.ChainSpec([P.GridField(grid, (0, 0, 0), (10 * U.kpc,) * 3, **f)], [bp_fixed(U.kpc)])
        np.testing.assert_array_equal(oracle.field(spec, pos), golden[f"field/B_{key}"])
    spectrum = tuple(golden["planewave/spectrum"])
    modes = oracle.plane_wave_modes(*spectrum, 64, 4321)
    spec = P.ChainSpec([P.PlaneWaveField(*modes, spectrum=spectrum, seed=4321)], [bp_fixed(U.kpc)])
    np.testing.assert_array_equal(oracle.field(spec, golden["planewave/pos"]), golden["planewave/B"])
    for key in [k for k in golden if k.startswith("random/")]:
        kind, *args = key.split("/")[1].split("_")
        a = [float(x) for x in args if x] + [0.0] * (3 - len([x for x in args if x]))
        np.testing.assert_array_equal(oracle.random(2024, int(kind), 500, *a), golden[key])
    ids = [1000010010, 1000020040, 1000070140, 1000260560]
    sid, se, sd = oracle.sample_source(11, 400, ids, None, 0.1 * U.EeV, 100 * U.EeV, -2.0)
    np.testing.assert_array_equal(sid, golden["source/id"])
    np.testing.assert_array_equal(se, golden["source/energy"])
    np.testing.assert_array_equal(sd, golden["source/dir"])
    from crpropa3_b200.workloads import charge_of
    assert [charge_of(int(i)) for i in golden["charge/ids"]] == list(golden["charge/q"])


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(PROPS))
def test_device_fp64_against_golden(golden, name):
    """Fixed-step chains bit-identical to the reference's results; adaptive
    chains bit-identical for >= 80 % of candidates (glibc pow, see
    test_gpu_parity.py)."""
    from crpropa3_b200.engine import Plan
    spec, c = _case(golden, name)
    rec = RecordArrays(256)
    Plan(spec).run(c, records=rec)
    if "adaptive" in name:
        same = np.all([getattr(c, m) == golden[f"{name}/out_{m}"] for m in ("x", "y", "z")], axis=0)
        assert same.mean() >= 0.8
    else:
        for m in STATE:
            np.testing.assert_array_equal(getattr(c, m), golden[f"{name}/out_{m}"], err_msg=m)
        for k, v in rec.sorted().items():
            np.testing.assert_array_equal(v, golden[f"{name}/rec_{k}"], err_msg=k)


def test_correctly_rounded_pow_of_the_controllers(tmp_path):
    """cr_pow (csrc/crmath.cuh) against 40-digit arithmetic: the quick evaluation
    and the full one that takes over where it cannot round."""
    import ctypes
    import subprocess
    from decimal import Decimal, localcontext
    src = tmp_path / "p.cpp"
    src.write_text('#include "crmath.cuh"\n'
                   'extern "C" double cr(double x, double y) { return crp::cr_pow(x, y); }\n'
                   'extern "C" int quick(double x, double y, double *r) { return crp::pow_quick(x, y, *r); }\n')
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-w",
                    "-I" + os.path.join(root, "crpropa3_b200", "csrc"), str(src), "-o", str(tmp_path / "p.so")],
                   check=True)
    lib = ctypes.CDLL(str(tmp_path / "p.so"))
    lib.cr.restype = ctypes.c_double
    lib.cr.argtypes = lib.quick.argtypes = [ctypes.c_double, ctypes.c_double]
    lib.quick.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.POINTER(ctypes.c_double)]
    rng = np.random.default_rng(8)
    x = np.concatenate([np.exp(rng.uniform(-12, 12, 600)), np.exp(rng.uniform(-690, 690, 200)),
                        1 + rng.uniform(-1, 1, 200) * 2.0 ** rng.integers(-52, 0, 200), [0.5, 2.0, 1024.0, 1e-307]])
    y = rng.choice([-0.2, 1 / 3, 0.5, 1.0, -1.0, 0.2371], len(x))
    declined = 0
    with localcontext() as ctx:
        ctx.prec = 40
        for a, b in zip(x.tolist(), y.tolist()):
            value = (Decimal(a).ln() * Decimal(b)).exp()
            exact = float(value)
            if any(abs((Decimal(exact) + Decimal(float(np.nextafter(exact, to)))) / 2 - value) < value * Decimal(2) ** -98
                   for to in (0.0, np.inf)):
                continue  # closer to a midpoint than the evaluation's 100 bits tell
            assert lib.cr(a, b) == exact, (a, b)
            r = ctypes.c_double()
            if lib.quick(a, b, ctypes.byref(r)):
                assert r.value == exact, (a, b)
            else:
                declined += 1
    assert declined < 0.05 * len(x)
