"""Runs over host arrays: one staged copy each way for small runs, separate
copies above; the states and records of the device run."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P
from crpropa3_b200.state import RecordArrays
from helpers import U, bp_fixed, protons, random_grid


def _spec(per_candidate):
    grid = random_grid(np.random.default_rng(4), 16)
    return P.ChainSpec([P.GridField(grid, (0, 0, 0), (10 * U.kpc,) * 3)],
                       [bp_fixed(1 * U.kpc), P.MaxTrajectoryLength(30 * U.kpc, per_candidate=per_candidate, record=True)])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 700, 1 << 15, (1 << 15) + 1])
@pytest.mark.parametrize("per_candidate,options", [(False, {}), (True, {"steps_per_launch": 7}),
                                                   (True, {"mode": _abi.MODE_PERSISTENT})])
def test_host_and_device_runs_agree(n, per_candidate, options):
    from crpropa3_b200.engine import Plan
    c = protons(np.random.default_rng(n), n)
    if per_candidate:
        c.max_length = np.random.default_rng(1).uniform(1, 30, n) * U.kpc
    plan = Plan(_spec(per_candidate))
    dev, dev_rec = c.to_device(), RecordArrays(n, device="cuda")
    plan.run(dev, records=dev_rec, **options)
    want, want_rec = dev.to_host(), dev_rec.to_host().sorted()
    for _ in range(2):  # the second run finds its buffers laid out
        got, rec = c.copy(), RecordArrays(n)
        plan.run(got, records=rec, **options)
        for name, a in want.members().items():
            np.testing.assert_array_equal(getattr(got, name), a, err_msg=name)
        for name, a in want_rec.items():
            np.testing.assert_array_equal(rec.sorted()[name], a, err_msg=name)


@pytest.mark.gpu
def test_missing_host_array_is_refused():
    from crpropa3_b200.engine import Plan
    plan = Plan(_spec(False))
    c = protons(np.random.default_rng(0), 8)
    s = c.struct()
    s.dy = C.POINTER(C.c_double)()
    assert plan.lib.crp_run(plan.handle, C.byref(s), 8, None, None) != _abi.OK


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 700])
def test_pinned_arrays_follow_the_stream(n):
    """A copy queued on the run's stream before the run is in the arrays the run reads."""
    import torch
    from crpropa3_b200.engine import Plan
    plan = Plan(_spec(False))
    c = protons(np.random.default_rng(n), n)
    want = c.copy()
    plan.run(want)
    keep, got = {}, c.copy()
    for name, a in c.members().items():
        keep[name] = torch.from_numpy(a.view(f"i{a.itemsize}")).pin_memory()
        setattr(got, name, keep[name].numpy().view(a.dtype))
    x = torch.from_numpy(c.x).cuda()
    got.x[:] = 0
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(40_000_000)
        keep["x"].view(torch.float64).copy_(x, non_blocking=True)
    plan.run(got, stream=stream.cuda_stream)
    for name, a in want.members().items():
        np.testing.assert_array_equal(getattr(got, name), a, err_msg=name)


DEVICE_POINTER = """
import ctypes as C, numpy as np, torch
from crpropa3_b200 import _abi
from crpropa3_b200.engine import Plan
from helpers import protons
from test_host_runs import _spec
plan, c = Plan(_spec(False)), protons(np.random.default_rng(0), 8)
x, s = torch.from_numpy(c.x).cuda(), c.struct()
s.x = C.cast(C.c_void_p(x.data_ptr()), C.POINTER(C.c_double))
print("status", plan.lib.crp_run(plan.handle, C.byref(s), 8, None, None))
"""


@pytest.mark.gpu
def test_device_memory_is_the_runtimes_to_judge():
    """A device array among host arrays is copied or refused, never read by the host."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = {**os.environ, "PYTHONPATH": os.pathsep.join([here, os.path.dirname(here)])}
    r = subprocess.run([sys.executable, "-c", DEVICE_POINTER], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "status" in r.stdout, (r.returncode, r.stderr[-2000:])
