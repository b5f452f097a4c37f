"""The rounding shift of the fixed-point apply kernel (csrc/mw_fx_round.h), compiled for the host, against exact
integers: every count, zero, the largest magnitudes and the halves."""
import os
import random
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include "mw_fx_round.h"
int main() {
    long long v;
    int s;
    while (std::scanf("%lld %d", &v, &s) == 2) std::printf("%lld\n", mwg::fx_round(v, s));
}
"""


def test_rounding_shift(tmp_path):
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "mrchem_gb300", "csrc"), str(src), "-o", str(exe)])
    rng = random.Random(3)
    cases = []
    for s in list(range(0, 64)) + [70, 127, 20000, 1000000]:
        values = {0, 1, -1, 2 ** 62, -2 ** 62, 2 ** 61 - 1, -2 ** 61}
        for _ in range(40):
            m = rng.getrandbits(rng.randint(1, 62))
            values |= {m, -m}
        if 1 <= s <= 62:
            values |= {2 ** (s - 1), -2 ** (s - 1), 2 ** (s - 1) - 1, -2 ** (s - 1) - 1}
        cases += [(v, s) for v in values if abs(v) <= 2 ** 62]
    out = subprocess.run([str(exe)], input="\n".join("%d %d" % c for c in cases), capture_output=True, text=True, check=True)
    for (v, s), r in zip(cases, map(int, out.stdout.split()), strict=True):
        if s <= 62:
            assert r == (v + (1 << s >> 1)) >> s, (v, s, r)  # Python's integers: exact
        elif abs(v) < 2 ** 61:
            assert r == 0, (v, s, r)  # above all, zero stays zero
        else:
            assert abs(r) <= 1
