"""The reciprocal of the FP64 push's rotation (csrc/fp64_int.cuh:
refine_reciprocal) on the host, from approximations up to its error bound off:
within an ulp of the exact value."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_reciprocal_is_within_an_ulp(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe, src = str(tmp_path / "check"), str(tmp_path / "in.bin")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(HERE, "cpp", "reciprocal_check.cpp")])
    rng = np.random.default_rng(1)
    d = np.concatenate([1.0 + rng.random(6000) ** 8, 2.0 ** rng.uniform(0, 220, 6000),
                        np.nextafter(2.0 ** np.arange(1, 60), np.inf), np.nextafter(2.0 ** np.arange(1, 60), 0.0)])
    e = rng.choice([-1.0, 0.0, 1.0, 0.5], len(d)) * 2.0 ** -20
    np.stack([d, e], 1).tofile(src)
    got = np.frombuffer(subprocess.run([exe, src], capture_output=True, check=True).stdout, np.float64)
    for x, r in zip(d, got):
        assert abs(Fraction(float(r)) - 1 / Fraction(float(x))) <= Fraction(float(np.spacing(r))), float(x).hex()
