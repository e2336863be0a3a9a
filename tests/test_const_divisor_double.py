"""const_divisor (csrc/divisor.h) for doubles.  A spacing arrives as a float, so
as a double its significand ends in 29 or more zero bits: the decision must come
at once for every such count, without undefined shifts.  Doubles with full
significands have dividends that divide wrongly; there the decision is held
against exact rational arithmetic: a / h = fma(a, inv, a lo) fails for some a
exactly where it fails for one whose quotient lies next to a midpoint."""
import random
import subprocess
import time
from fractions import Fraction

import numpy as np

from mixedprecisionfaracoustic_b200 import build as B

PROGRAM = r"""
#include "divisor.h"
#include <cstdio>
#include <cstdlib>
int main(int n, char** v) {
    for (int i = 1; i < n; i++) {
        const double h = strtod(v[i], nullptr);
        double lo = -1;
        const bool said = bpk::const_divisor(h, 1.0 / h, &lo);
        printf("%d %a\n", said, lo);
        fflush(stdout);
    }
}
"""
FLOATS = [0.011, 0.022, 0.037, 0.051, 0.13, 0.26, 0.52, 0.0033, 0.0044, 0.0097, 0.01, 0.1, 5.0, 7.7, 12.5, 4.0]
# doubles the two operations do not divide by, found by search
REFUSED = [float.fromhex(x) for x in ("0x1.cd613d8f16adfp+0", "0x1.afbd6619699cfp+0", "0x1.e8e5b7589a82bp+3")]


def decisions(tmp_path, hs):
    """[(decision, lo)] of const_divisor, compiled with every undefined operation an error."""
    (tmp_path / "d.cpp").write_text(PROGRAM)
    exe = tmp_path / "d"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    "-I", str(B.CSRC), "-o", str(exe), str(tmp_path / "d.cpp")], check=True, capture_output=True, timeout=300)
    t = time.monotonic()
    r = subprocess.run([str(exe), *(h.hex() for h in hs)], check=True, capture_output=True, text=True, timeout=20)
    assert time.monotonic() - t < 5
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == len(hs)
    return [(int(a), float.fromhex(b)) for a, b in rows]


def rounds_right(A, h, inv, lo):
    rn = lambda x: x.numerator / x.denominator            # int / int rounds correctly
    return rn(Fraction(A) * Fraction(inv) + Fraction(float(A) * lo)) == rn(Fraction(A) / Fraction(h))


def near_midpoints(h, reach=8):
    """Integer dividends in [2^52, 2^53) whose quotient by h lies within
    reach 2^-53 units of a midpoint, h's significand odd or nearly so."""
    n, d = h.as_integer_ratio()
    Bi = n
    while Bi < 1 << 52:
        Bi *= 2
    assert Bi < 1 << 53
    out = []
    for E in (53, 54):
        for J in range(-reach, reach + 1):
            s = (Bi & -Bi).bit_length() - 1
            if J % (1 << s):
                continue
            Bo = Bi >> s
            a = (J >> s) * pow(pow(2, E - s, Bo), -1, Bo) % Bo
            out += [A for A in range(a, 1 << 53, Bo) if A >= 1 << 52]
    return out


def test_spacings_are_decided_at_once(tmp_path):
    hs = [float(np.float32(x)) for x in FLOATS]
    ends = [int(np.frexp(h)[0] * 2 ** 53) for h in hs]
    assert {(m & -m).bit_length() - 1 for m in ends} >= {29, 30, 32, 33, 34, 35, 48, 50, 52}    # zero bits
    rng = random.Random(3)
    for h, (said, lo) in zip(hs, decisions(tmp_path, hs)):
        assert said == 1, h
        for _ in range(2000):
            assert rounds_right(rng.getrandbits(52) | 1 << 52, h, 1.0 / h, lo), h


def test_full_significands_against_exact_arithmetic(tmp_path):
    rng = random.Random(5)
    hs = REFUSED + [(rng.getrandbits(52) | 1 << 52 | 1) / 2.0 ** 50 for _ in range(200)]
    said = decisions(tmp_path, hs)
    for h, (ok, lo) in zip(hs, said):
        assert bool(ok) == all(rounds_right(A, h, 1.0 / h, lo) for A in near_midpoints(h)), h.hex()
    assert [ok for ok, _ in said[:3]] == [0, 0, 0] and sum(ok for ok, _ in said) > 150
