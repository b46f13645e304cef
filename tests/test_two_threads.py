"""Plans of different sizes run from two host threads at once."""
import glob
import os
import re
import threading

import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P, workloads as W
from helpers import ROOT, U, protons


def _plan(kind, modes, precision):
    from crpropa3_b200.engine import Plan
    spectrum = (1 * U.nG, 20 * U.kpc, 200 * U.kpc, 200 * U.kpc, 5.0 / 3.0, 4.0)
    waves = P.PlaneWaveField(*W.plane_wave_modes(*spectrum, modes, 11), spectrum=spectrum, seed=11)
    prop = P.Propagation(kind, 1e-4, 1 * U.kpc, 1 * U.kpc)
    return Plan(P.ChainSpec([waves], [prop, P.MaxTrajectoryLength(1000 * U.kpc)], precision=precision))


def test_shared_memory_limits_are_constants():
    """A kernel's shared-memory limit is one for all plans: only the helper that
    takes it as a template argument sets it."""
    calls = []
    for path in glob.glob(os.path.join(ROOT, "crpropa3_b200", "csrc", "*")):
        with open(path) as f:
            calls += re.findall(r"cudaFuncSetAttribute\(.*?\)", f.read().replace("(int)MOST", "MOST"), re.S)
    assert calls == ["cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST)"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,modes,precision", [(_abi.PROP_BP, (40, 1200), _abi.PRECISION_FP64),
                                                  (_abi.PROP_BP, (40, 1365), _abi.PRECISION_MIXED),
                                                  (_abi.PROP_SDE, (1100, 2200), _abi.PRECISION_MIXED)])
def test_mode_tables_of_different_sizes(kind, modes, precision):
    """A kernel's shared-memory limit holds for both plans' tables at any moment."""
    import torch
    errors, done = [], []

    def work(m):
        try:
            plan = _plan(kind, m, precision)
            stream = torch.cuda.Stream()
            c = protons(np.random.default_rng(1), 1).to_device()
            torch.cuda.synchronize()
            start.wait()
            for k in range(1500):
                plan.run(c, max_steps=k + 1, stream=stream.cuda_stream)
            done.append(m)
        except Exception as e:
            errors.append((m, str(e)))
            start.abort()

    start = threading.Barrier(2)
    threads = [threading.Thread(target=work, args=(m,)) for m in modes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and sorted(done) == sorted(modes), errors
