"""The integer-pipe FP64 arithmetic of the dipole mover and the tracer
(csrc/fp64_int.cuh), run on the host against the host's FP64 operations (bit
for bit) and, for a^2.5, against exact rational bounds. The device's FP32
estimates are replaced by the exact values with errors over their bounds."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("fp64_int")
    exe = str(d / "check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(HERE, "cpp", "fp64_int_check.cpp")])

    def run(a, b, c, err):
        src = d / "in.bin"
        np.stack([a, b, c, err], 1).astype(np.float64).tofile(src)
        out = subprocess.run([exe, str(src)], capture_output=True, check=True).stdout
        return np.frombuffer(out, np.float64).reshape(-1, 3)

    return run


def significands(rng, n, kind):
    """Doubles in [1, 2) of one kind of significand."""
    if kind == "random":
        m = rng.integers(0, 1 << 52, n)
    elif kind == "edges":  # all zeros, all ones and their neighbours
        m = rng.choice(np.array([0, 1, 2, 3, (1 << 52) - 1, (1 << 52) - 2, 1 << 51, (1 << 51) - 1]), n)
    elif kind == "few_bits":  # products and sums land on exact ties
        m = rng.integers(0, 1 << 27, n) << 25
    else:  # long runs of ones or zeros below a random top
        m = (rng.integers(0, 1 << 20, n) << 32) | rng.choice(np.array([0, (1 << 32) - 1, 1 << 31, 1]), n)
    return (m.astype(np.uint64) | np.uint64(1023 << 52)).view(np.float64)


@pytest.mark.parametrize("kind", ["random", "edges", "few_bits", "runs"])
@pytest.mark.parametrize("spread", [0, 2, 60, 150])
def test_operations_round_as_fp64(check, kind, spread):
    rng = np.random.default_rng(7 + spread)
    n = 60000
    a, b, c = (significands(rng, n, kind) * rng.choice([-1.0, 1.0], n) *
               2.0 ** rng.integers(-spread, spread + 1, n) for _ in range(3))
    out = check(a, b, c, rng.choice([-1.0, 0.0, 1.0], n) * rng.random(n) ** 0.25)
    bad = np.nonzero(out[:, 0])[0]
    assert len(bad) == 0, [(a[i].hex(), b[i].hex(), c[i].hex()) for i in bad[:5]]


def test_pow25_is_correctly_rounded_where_sure(check):
    rng = np.random.default_rng(11)
    a = np.concatenate([significands(rng, 30000, "random") * 2.0 ** rng.integers(-150, 151, 30000),
                        significands(rng, 2000, "edges") * 2.0 ** rng.integers(-5, 6, 2000),
                        np.floor(rng.uniform(1, 1e6, 4000)) ** 2, rng.integers(1, 10 ** 6, 4000).astype(float)])
    err = rng.choice([-1.0, 0.0, 1.0], len(a))
    out = check(a, np.ones_like(a), np.ones_like(a), err)
    sure = out[:, 2] != 0
    assert sure[:30000].mean() > 0.999
    for x, r in zip(a[sure], out[sure, 1]):
        # r rounds x^2.5 to nearest: (r - ulp/2)^2 < x^5 < (r + ulp/2)^2
        r = float(r)
        h = Fraction(np.spacing(r)) / 2
        lo = Fraction(r) - (h if np.frexp(r)[0] != 0.5 else h / 2)
        assert lo * lo < Fraction(float(x)) ** 5 < (Fraction(r) + h) ** 2, float(x).hex()
