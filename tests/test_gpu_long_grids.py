"""Universes with one very long axis (more rows than a launch's second and
third grid dimension hold): one step with deposit against the oracle. States
to 1e-12, densities to 1e-11 of their peak (a handful of terms per node)."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import OracleSim, align_by_id, assert_states_close, gpu_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_long_axis_matches_oracle(axis):
    size = np.array([1, 1, 1])
    size[axis] = 70000
    rng = np.random.default_rng(axis)
    n = 70000
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    cell = np.zeros((n, 3))
    cell[:, axis] = np.arange(n)
    p["position"] = cell + rng.random((n, 3))
    p["velocity"] = rng.normal(0.0, 0.05, (n, 3))
    p["q"], p["qom"] = -0.5, -1.0
    props = abi.Props.make(size=size, dt=0.1)
    cfg = dict(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC)
    sim = gpu_sim(props, abi.Config.make(flags=abi.F_TRACK_IDS, **cfg))
    orc = OracleSim(props, abi.Config.make(**cfg))
    field = rng.normal(0.0, 0.1, abi.field_shape(props))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(p, np.ones(n, np.uint64))
        s.step(1)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    assert_states_close(a, b, rtol=1e-12, atol=1e-12, what=str(axis))
    orc.project()
    for x, y in zip(sim.download_fields()[2:], orc.download_fields()[2:]):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * np.abs(y).max())
    sim.close()
