"""The FP64 dipole mover without a dipole moment (csrc/push64.cuh: no_field):
free flight, bit for bit the oracle's -- zeros of either sign, tiny, huge and
subnormal values included."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import OracleSim, align_by_id, gpu_sim
from test_gpu_dipole64 import KINDS, edge_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bz", [0.0, -0.0])
@pytest.mark.parametrize("kind", KINDS)
def test_free_flight_matches_oracle(kind, bz):
    n = 8
    parts = edge_particles(kind, 3000, 5, 4.0)
    parts["qom"] = np.resize(parts["qom"][:12], len(parts))  # a universe has at most 16 species
    rng = np.random.default_rng(1)
    parts["velocity"][rng.random(len(parts)) < 0.2, 1] = -0.0
    parts["velocity"][rng.random(len(parts)) < 0.2, 2] = 0.0
    cell = np.clip(np.floor(parts["position"] + 4.0).astype(np.int64), 0, n - 1)
    flat = (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2]
    parts = parts[np.argsort(flat, kind="stable")]
    counts = np.bincount(flat, minlength=n ** 3).astype(np.uint64)
    props = abi.Props.make(size=(n,) * 3, dt=0.05, planet_radius=0.5, origin=(-4.0,) * 3, external_b=(0.0, 0.0, bz))
    sim = gpu_sim(props, abi.Config.make(flags=abi.F_TRACK_IDS))
    orc = OracleSim(props, abi.Config.make())
    for s in (sim, orc):
        s.upload_particles(parts, counts)
        s.step(4)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    for f in ("position", "velocity"):
        np.testing.assert_array_equal(np.ascontiguousarray(a[f]).view(np.uint64),
                                      np.ascontiguousarray(b[f]).view(np.uint64))
    sim.close()
