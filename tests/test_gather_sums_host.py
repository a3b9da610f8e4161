"""Sums of the dependency gathers as the kernels form them (csrc/xf64.cuh with
kXgPsiBias) on the host against exact arithmetic: rows of random terms are not
biased, rows of terms of few bits (psi = 1 of leaves, whole numbers of trees)
keep all but the last of 57 bits."""
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
    exe = str(tmp_path_factory.mktemp("gather") / "gather_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-w", "-I", os.path.join(ROOT, "lightgraphs.jl_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "gather_check.cpp")], check=True)
    return exe


def run(exe, sums):
    text = "\n".join("%d %s" % (len(x), " ".join("%d %d" % t for t in x)) for x in sums) + "\n"
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    return [[int(t) for t in ln.split()] for ln in out.strip().split("\n")]


def value(m, e):
    return Fraction(m) * TWO ** (e - BIAS)


def of_doubles(x):
    b = np.asarray(x, np.float64).view(np.uint64)
    m = ((b & np.uint64(2**52 - 1)) | np.uint64(2**52)) << np.uint64(10)
    return list(zip(m.tolist(), (b >> np.uint64(52)).astype(int).tolist()))


@pytest.mark.parametrize("n,bias", [(64, 2e-17), (256, 2.0**-54)])
@pytest.mark.parametrize("spread", ["narrow", "wide"])
def test_long_rows_are_not_biased(harness, n, bias, spread):
    rng = np.random.default_rng(n)
    draw = (lambda: 0.2 + rng.random(n)) if spread == "narrow" else (lambda: np.exp2(-20 * rng.random(n)))
    sums = [[(m + int(t), e) for (m, e), t in zip(of_doubles(draw()), rng.integers(0, 1024, n))]
            for _ in range(400)]
    off = []
    for x, r in zip(sums, run(harness, sums)):
        exact = sum(value(*t) for t in x)
        off.append(float((value(*r[1:]) - exact) / exact))
    assert abs(np.mean(off)) < bias, np.mean(off)


@pytest.mark.parametrize("n", [1, 2, 32, 64, 256, 2000])
def test_terms_of_few_bits(harness, n):
    # a word of the largest exponent is above its value by its exponent byte,
    # less than one unit of the term's 57 bits; the others lose that byte
    rng = np.random.default_rng(n)
    for pick in (lambda: np.ones(n), lambda: rng.choice([0.25, 0.5, 1.0], n), lambda: rng.integers(1, 1 << 20, n),
                 lambda: rng.integers(1, 1 << 31, n) if n < 3 else np.full(n, 2.0**30)):
        x = of_doubles(np.asarray(pick(), np.float64))
        top, m, e = run(harness, [x])[0]
        exact = sum(value(*t) for t in x)
        assert top < 128
        assert abs(value(m, e) - exact) <= exact * TWO ** -56
