"""The rule that decides how many candidates a block sums PlaneWaveTurbulence
modes for (csrc/engine_internal.h), and the kernels at its edges."""
import os
import subprocess

import numpy as np
import pytest

from crpropa3_b200 import _abi, plan as P, workloads as W
from helpers import ROOT, U, protons

PROGRAM = r"""
#include "engine_internal.h"
#include <cstdio>
int main() {
    for (int sms : {1, 148, 160})
        for (int fp64 = 0; fp64 < 2; fp64++)
            for (int ck = 0; ck < 2; ck++)
                for (int m = 1; m <= 2700; m += m < 70 ? 1 : 7)
                    for (uint64_t n = 1; n < 400000; n += 1 + n / 23) {
                        const int w = crp::wave_block_warps(n, m, sms, fp64, ck, n % 2);
                        const uint64_t blocks = w ? (n + 32 * w - 1) / (32 * w) : 0;
                        const size_t table = fp64 ? 72 * (size_t)m : 80 * (size_t)((m + 1) / 2);
                        const size_t block = table + (fp64 ? 11264 : 9216) + 1024;
                        if (w && block > 227 * 1024) { printf("%d modes do not fit\n", m); return 1; }
                        if (w && fp64 && (w > 2 || blocks > (uint64_t)sms * (228 * 1024 / block))) {
                            printf("FP64, %d modes, %llu candidates: %d warps wait for room\n", m, (unsigned long long)n, w);
                            return 1;
                        }
                    }
    return 0;
}
"""


def test_fp64_blocks_never_wait_for_shared_memory(tmp_path):
    """Sums by the block only where every block has its table at once."""
    src = tmp_path / "rule.cpp"
    src.write_text(PROGRAM)
    include = [os.path.join(ROOT, "crpropa3_b200", "csrc"), os.path.join(ROOT, "include"), "/usr/local/cuda/include"]
    subprocess.run(["g++", "-std=c++17", "-w", *("-I" + d for d in include), str(src), "-o", str(tmp_path / "rule")],
                   check=True)
    r = subprocess.run([str(tmp_path / "rule")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


NAMES = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time", "current_step",
         "next_step", "active", "flags", "step_count")
BLOCKS = [(_abi.PRECISION_FP64, 129, 32), (_abi.PRECISION_FP64, 18945, 101), (_abi.PRECISION_FP64, 65, 1365),
          (_abi.PRECISION_FP64, 9473, 1365), (_abi.PRECISION_MIXED, 129, 8), (_abi.PRECISION_MIXED, 65, 1365),
          (_abi.PRECISION_MIXED, 18945, 200), (_abi.PRECISION_MIXED, 37889, 33),
          (_abi.PRECISION_MIXED, 65, 2600),
          # thread by thread: one mode more than the largest table, and one fewer than the least
          (_abi.PRECISION_FP64, 65, 1366), (_abi.PRECISION_MIXED, 65, 2601), (_abi.PRECISION_FP64, 65, 31)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n,modes", BLOCKS)
@pytest.mark.parametrize("prop", [(_abi.PROP_BP, 1, 1), (_abi.PROP_BP, 0.1, 5), (_abi.PROP_CK, 0.1, 5)])
def test_sums_at_the_edges_of_the_rule(precision, n, modes, prop):
    """The same bits as the persistent kernels, which sum thread by thread."""
    from crpropa3_b200.engine import Plan
    spectrum = (1 * U.nG, 20 * U.kpc, 200 * U.kpc, 200 * U.kpc, 5.0 / 3.0, 4.0)
    waves = P.PlaneWaveField(*W.plane_wave_modes(*spectrum, modes, 11), spectrum=spectrum, seed=11)
    mods = [P.Propagation(prop[0], 1e-4, prop[1] * U.kpc, prop[2] * U.kpc), P.MaxTrajectoryLength(3 * U.kpc)]
    plan = Plan(P.ChainSpec([waves], mods, precision=precision))
    c = protons(np.random.default_rng(n), n, emin=0.1 * U.EeV)
    c.charge[::9] = 0
    a, b = c.to_device(), c.to_device()
    plan.run(a)
    plan.run(b, mode=_abi.MODE_PERSISTENT)
    a, b = a.to_host(), b.to_host()
    for name in NAMES:
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name), err_msg=name)
