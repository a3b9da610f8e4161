"""The psi words and row sums of the shared-memory sweeps (csrc/xf64.cuh:
psi_pack, psi_add, psi_norm, psi_value) on the host against exact arithmetic.
A word is within 2^-56 of its value (half a unit of 56 bits).  Each of a sum's n
adds and n / 32 renormalisations is off by less than one unit of at least 58
bits, 2^-57 of the sum, and long rows must not be biased."""
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
    exe = str(tmp_path_factory.mktemp("psi") / "psi_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-w", "-I", os.path.join(ROOT, "lightgraphs.jl_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "psi_check.cpp")], check=True)
    return exe


def run(exe, sums):
    text = "\n".join("%d %s" % (len(x), " ".join("%d %d" % t for t in x)) for x in sums) + "\n"
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    return [[int(t) for t in ln.split()] for ln in out.strip().split("\n")]


def value(m, e):
    return Fraction(m) * TWO ** (e - BIAS)


# exponents of values in (2^-48, 2^15]
LOW, HIGH = BIAS - 62 - 48, BIAS - 62 + 14


def terms(rng, n, low=LOW, high=HIGH):
    m = rng.integers(2**62, 2**63, n, dtype=np.uint64)
    m[rng.random(n) < 0.2] = np.uint64(2**62)
    m[rng.random(n) < 0.2] = np.uint64(2**63 - 1)
    return [(int(a), int(b)) for a, b in zip(m, rng.integers(low, high + 1, n))]


def of_doubles(x):
    """{m, e} of positive doubles, 10 random bits added below them."""
    b = np.asarray(x, np.float64).view(np.uint64)
    m = ((b & np.uint64(2**52 - 1)) | np.uint64(2**52)) << np.uint64(10)
    return list(zip(m.tolist(), (b >> np.uint64(52)).astype(int).tolist()))


def test_words(harness):
    edge = [(m, e) for e in (LOW, HIGH) for k in (0, 1, 30, 31, 32, 33, 63, 64, 65, 95, 96, 127, 128, 192)
            for m in (2**62 + k, 2**63 - 1 - k)]
    cases = edge + terms(np.random.default_rng(1), 3000)
    for (m, e), r in zip(cases, run(harness, [[t] for t in cases])):
        w = r[0]
        assert 2**61 <= w < 2**62  # the two top bits are flags of the sweeps
        got, exact = Fraction(w & ~63) * TWO ** ((w & 63) - 109), value(m, e)
        assert abs(got - exact) <= exact * TWO ** -56, (m, e)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 470, 1000])
@pytest.mark.parametrize("low,high", [(LOW, HIGH), (1023, 1023), (1000, 1030)])
def test_sums(harness, n, low, high):
    rng = np.random.default_rng(n + high)
    sums = [terms(rng, n, low, high) for _ in range(40)]
    for x, r in zip(sums, run(harness, sums)):
        exact = sum(value(*t) for t in x)
        m, e = r[-2:]
        assert 2**62 <= m < 2**63
        bound = TWO ** -56 + (n + n // 32 + 1) * TWO ** -57
        assert abs(value(m, e) - exact) <= exact * bound


@pytest.mark.parametrize("n,bias", [(64, 2e-17), (470, 2.0**-54)])
def test_long_rows_are_not_biased(harness, n, bias):
    # random psi in [0.2, 1.2): the mean error over many rows, against -1.5e-16
    # and -2.2e-15 of sums in 56 bits that drop what does not fit
    rng = np.random.default_rng(n)
    sums = [[(m + int(t), e) for (m, e), t in zip(of_doubles(0.2 + rng.random(n)), rng.integers(0, 1024, n))]
            for _ in range(400)]
    off = []
    for x, r in zip(sums, run(harness, sums)):
        exact = sum(value(*t) for t in x)
        off.append(float((value(*r[-2:]) - exact) / exact))
    assert abs(np.mean(off)) < bias, np.mean(off)


@pytest.mark.parametrize("n", [1, 2, 64, 470, 2000])
def test_short_terms_stay_exact(harness, n):
    # psi = 1 of leaves, whole numbers and halves of trees and grids
    rng = np.random.default_rng(n)
    for pick in (lambda: np.ones(n), lambda: rng.choice([0.25, 0.5, 1.0], n), lambda: rng.integers(1, 20000, n)):
        x = of_doubles(np.asarray(pick(), np.float64))
        r = run(harness, [x])[0]
        assert value(*r[-2:]) == sum(value(*t) for t in x)
