"""The packed terms of the dependency gathers (csrc/xf64.cuh: xg_pack,
xg_add_packed, xg_packed_sum) on the host against exact arithmetic: a word is
within 2^-56 of its value (half a unit of 56 bits; 2^-55 in the last 128 units
below a power of two, where it is truncated), and each of a sum's n adds and
n / 32 renormalisations truncates less than 2^-56 of the sum."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BIAS = 1085  # of the extended format: m 2^(e - BIAS)
TWO = Fraction(2)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("packed") / "packed_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-w", "-I", os.path.join(ROOT, "lightgraphs.jl_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "packed_check.cpp")], check=True)
    return exe


def run(exe, sums):
    text = "\n".join("%d %s" % (len(x), " ".join("%d %d" % t for t in x)) for x in sums) + "\n"
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    return [[int(t) for t in ln.split()] for ln in out.strip().split("\n")]


def value(m, e):
    return Fraction(m) * TWO ** (e - BIAS)


# exponents of 2^-64 (the reciprocal of the largest path count) to 2^31 (every vertex)
LOW, HIGH = 1085 - 62 - 64, 1085 - 62 + 31


def terms(rng, n, low=LOW, high=HIGH):
    m = rng.integers(2**62, 2**63, n, dtype=np.uint64)
    m[rng.random(n) < 0.2] = np.uint64(2**62)
    m[rng.random(n) < 0.2] = np.uint64(2**63 - 1)
    return [(int(a), int(b)) for a, b in zip(m, rng.integers(low, high + 1, n))]


def test_words(harness):
    edge = [(m, e) for e in (LOW, HIGH) for k in (0, 1, 30, 60, 64, 70, 126, 127, 128, 129, 200)
            for m in (2**62 + k, 2**63 - 1 - k)]
    cases = edge + terms(np.random.default_rng(1), 3000)
    for (m, e), r in zip(cases, run(harness, [[t] for t in cases])):
        w = r[0]
        got, exact = Fraction(w) * TWO ** ((w & 255) - 186), value(m, e)
        bound = TWO ** -55 if m >= 2**63 - 128 else TWO ** -56
        assert abs(got - exact) <= exact * bound, (m, e)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 600])
@pytest.mark.parametrize("low,high", [(LOW, HIGH), (1023, 1023), (1000, 1030)])
def test_sums(harness, n, low, high):
    rng = np.random.default_rng(n + high)
    sums = [terms(rng, n, low, high) for _ in range(60)]
    for x, r in zip(sums, run(harness, sums)):
        exact = sum(value(*t) for t in x)
        m, e = r[-2:]
        assert 2**61 <= m < 2**63
        bound = TWO ** -55 + (n + n // 32 + 1) * TWO ** -56
        assert abs(value(m, e) - exact) <= exact * bound
