"""const_divisor (csrc/divisor.h): whether a / h = fma(a, inv, a lo) for every
float a is decided from a handful of dividends; here every significand of a is
tried (a quotient's rounding does not depend on the exponent), for spacings the
configurations use, powers of two, significands near 1 and 2, even and odd ones,
and one that the two operations do not divide by."""
import subprocess
from pathlib import Path

from mixedprecisionfaracoustic_b200 import build as B

PROGRAM = r"""
#include "divisor.h"
#include <cstdio>
#include <cstdlib>
int main(int n, char** v) {
    for (int i = 1; i < n; i++) {
        const float h = strtof(v[i], nullptr), inv = 1.0f / h;
        float lo = 0;
        const bool said = bpk::const_divisor(h, inv, &lo);
        bool all = true;
        for (int A = 1 << 23; A < 1 << 24 && all; A++) {
            const float a = (float)A, t = a * lo;
            all = std::fma(a, inv, t) == a / h;
        }
        double lod = 0;
        printf("%d %d %d\n", said, all, bpk::const_divisor((double)h, 1.0 / h, &lod));
    }
}
"""
# REFUSED: found by search; its significand leaves a quotient within 2^-47 of a midpoint
REFUSED = "0x1.4193fep+2"
SPACINGS = ["0.01", "5", "10", "12.5", "4", "0.1", "7.7", "0x1.fffffep0", "0x1.000002p2", "0x1.8p-3", "0x1.234568p3", REFUSED]


def test_decision_matches_every_dividend(tmp_path):
    (tmp_path / "d.cpp").write_text(PROGRAM)
    exe = tmp_path / "d"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(B.CSRC), "-o", str(exe),
                    str(tmp_path / "d.cpp")], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe), *SPACINGS], check=True, capture_output=True, text=True, timeout=600).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == len(SPACINGS)
    for h, (said, exact, _) in zip(SPACINGS, rows):
        assert said == exact, h
    assert rows[SPACINGS.index(REFUSED)][0] == 0
    assert all(r[0] for r in rows[:6])
