"""Uploads into a known layout (the cell kernel of csrc/upload.cu) of 1 to 16
populations, through a second upload that fits, one that overflows its slots
and one of few particles: what comes back is what went up, bit for bit (FP32:
positions to 1e-7 cell widths, velocities as FP32), and the fused deposit's J
and rho are the projection's to 1e-5 of their peak."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import gpu_sim

pytestmark = pytest.mark.gpu

SPECIES = [(-1.0, -1.0), (1.0, 0.1), (-1.0, 0.1), (0.0, 1.0), (2.0, 0.0)] + [(3.0 + k, -2.0 - k) for k in range(11)]


def load(size, width, per, species, seed):
    rng = np.random.default_rng(seed)
    counts = rng.poisson(per, int(np.prod(size)))
    cell = np.repeat(np.arange(len(counts)), counts)
    c = np.stack(np.unravel_index(cell, size), 1)
    p = np.zeros(len(cell), abi.PARTICLE_DTYPE)
    p["position"] = (c + rng.random((len(c), 3))) * width
    p["velocity"] = rng.normal(0.0, 0.1, (len(c), 3))
    p["q"], p["qom"] = np.array(SPECIES[:species])[rng.integers(0, species, len(c))].T
    if species > 3:  # either sign of zero is the same species
        zero = (p["q"] == 0.0) & (rng.random(len(p)) < 0.5)
        p["q"][zero] = -0.0
    return p, counts.astype(np.uint64)


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("species", [1, 2, 3, 4, 5, 9, 16])
def test_uploads_come_back(species, prec):
    size, width = (5, 4, 6), np.array([0.7, 1.0, 1.5])
    props = abi.Props.make(size=size, cell_width=width, dt=0.1)
    cfg = dict(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC, flags=abi.F_TRACK_IDS)
    sim, ref = (gpu_sim(props, abi.Config.make(precision=k, **cfg)) for k in (prec, abi.FP64))
    for s in (sim, ref):
        s.upload_fields(np.zeros(abi.field_shape(props)))
    first = load(size, width, 30, species, 1)
    first[0]["q"][:species], first[0]["qom"][:species] = np.array(SPECIES[:species]).T  # every species is known
    for p, counts in (first, load(size, width, 30, species, 2), load(size, width, 300, species, 3),
                      load(size, width, 0.5, species, 4)):
        sim.upload_particles(p, counts)
        q, back, ids = sim.download_particles()
        np.testing.assert_array_equal(back, counts)
        np.testing.assert_array_equal(np.sort(ids), np.arange(len(p)))
        p = p[ids]
        for k in ("q", "qom"):
            np.testing.assert_array_equal(q[k], p[k])
        if prec == abi.FP64:
            np.testing.assert_array_equal(q["position"], p["position"])
            np.testing.assert_array_equal(q["velocity"], p["velocity"])
        else:
            assert np.abs((q["position"] - p["position"]) / width).max(initial=0) <= 1e-7
            np.testing.assert_array_equal(q["velocity"], p["velocity"].astype(np.float32))
            cell = np.repeat(np.arange(len(counts)), counts.astype(int))
            assert np.all(np.diff(cell) >= 0)
        if prec == abi.FP32:
            ref.upload_particles(p, counts)
            ref.project()
            sim.project()
            for x, y in zip(sim.download_fields()[2:], ref.download_fields()[2:]):
                np.testing.assert_allclose(x, y, rtol=0, atol=1e-5 * np.abs(y).max())
    sim.close()
    ref.close()
