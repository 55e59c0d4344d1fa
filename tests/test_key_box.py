"""The tracer's quick box test (csrc/fp64_int.cuh: key_box, in_key_box) on the
host, with signed overflow trapped: a position it takes lies inside the box
(no wrap), and one it does not take lies outside or shares a high word with a
face (then the full comparison decides)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_key_box_is_inside(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe, src = str(tmp_path / "check"), str(tmp_path / "in.bin")
    subprocess.check_call([cxx, "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow",
                           "-fsanitize-undefined-trap-on-error", "-o", exe,
                           os.path.join(HERE, "cpp", "key_box_check.cpp")])
    big = np.finfo(np.float64).max
    faces = [(-32.0, 32.0), (-4.0, 4.0), (-0.0, 1.0), (0.0, 1e-310), (-1e-310, -0.0), (-big, big), (-8.0, -2.0),
             (3.0, 3.5), (-1e300, 2.0), (1.0, 1.0)]
    rng = np.random.default_rng(1)
    rows = []
    for low, high in faces:
        x = np.concatenate([rng.uniform(-40, 40, 2000), rng.normal(0, 1, 500) * 10.0 ** rng.uniform(-320, 300, 500),
                            np.array([low, high, 0.0, -0.0, np.inf, -np.inf, np.nan, -np.nan, big, -big, 5e-324]),
                            np.nextafter(low, [-1.0, 1.0]), np.nextafter(high, [-1.0, 1.0])])
        rows.append(np.stack([np.full_like(x, low), np.full_like(x, high), x], 1))
    rows = np.concatenate(rows)
    rows.tofile(src)
    out = np.frombuffer(subprocess.run([exe, src], capture_output=True, check=True).stdout, np.uint8)
    assert len(out) == len(rows)
    took, inside = (out & 1) != 0, (out & 2) != 0
    assert not (took & ~inside).any()
    on_face = np.zeros(len(rows), bool)
    for r in (rows, rows + 0.0):  # + 0.0: either sign of zero
        high_word = r.view(np.uint64) >> np.uint64(32)
        on_face |= (high_word[:, 2] == high_word[:, 0]) | (high_word[:, 2] == high_word[:, 1])
    assert (took | ~inside | on_face).all()
