"""The division-free quotients and unit vectors of the FP64 form
(csrc/crmath.cuh), compiled for the host: every result is the IEEE one."""
import os
import subprocess

from helpers import ROOT

PROGRAM = r"""
#include "crmath.cuh"
#include <cstdio>
#include <cstdint>
#include <cstring>
using namespace crp;
static uint64_t state = 88172645463325252ull;
static uint64_t next() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static double bits(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
// a mantissa: random, or within 3 units of a power of two or of the middle
static uint64_t mantissa() {
    const uint64_t m = next() >> 12, r = next();
    if (r % 4) return m;
    const uint64_t edge = (r >> 2) % 3 == 0 ? 0 : (r >> 2) % 3 == 1 ? (1ull << 51) : (1ull << 52) - 1;
    return (edge + (r >> 8) % 7 - 3) & ((1ull << 52) - 1);
}
static double operand(int emin, int emax) {
    const int e = 1023 + emin + (int)(next() % (uint64_t)(emax - emin + 1));
    return bits((next() & 1) << 63 | (uint64_t)e << 52 | mantissa());
}
int main() {
    for (int i = 0; i < 3000000; i++) {
        const double b = operand(-200, 200);
        double a = operand(-200, 200);
        if (i % 3 == 0) {  // a product of b, and its neighbours: quotients next to a double and to a midpoint
            a = b * operand(-50, 50);
            a = bits(([&] { uint64_t u; memcpy(&u, &a, 8); return u; })() + next() % 5 - 2);
        }
        if (quotient(a, b, 1.0 / b) != a / b) { printf("%a / %a\n", a, b); return 1; }
    }
    for (int i = 0; i < 3000000; i++) {
        // |n2 - 1| < 2^-27, every size of the difference
        const double d = ldexp((double)(next() >> 11), -53 - 27 - (int)(next() % 26));
        const double n2 = next() & 1 ? 1.0 + d : 1.0 - d;
        if (!(fabs(n2 - 1) < 0x1p-27)) continue;
        const double r = root_near_1(n2);
        if (r != sqrt(n2)) { printf("sqrt %a: %a\n", n2, r); return 1; }
        if (reciprocal_near_1(r) != 1.0 / r) { printf("1 / %a\n", r); return 1; }
    }
    return 0;
}
"""


def test_quotients_roots_and_reciprocals_are_rounded_correctly(tmp_path):
    src = tmp_path / "q.cpp"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I" + os.path.join(ROOT, "crpropa3_b200", "csrc"),
                    str(src), "-o", str(tmp_path / "q")], check=True)
    r = subprocess.run([str(tmp_path / "q")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
