"""The FP64 field mover with the dipole term where its factor mft / r^5 leaves
the integer path: lengths of 2^-110 and 2^110 (r^2 beyond 2^+-200), no dipole
moment, and the ordinary scale beside them. Against the oracle, relative to
the scale, to 1e-12."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import OracleSim, align_by_id, gpu_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moment", [1.5, 0.0])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 110, 2.0 ** -110])
def test_dipole_scales_match_oracle(scale, moment):
    n, ppc = 6, 30
    rng = np.random.default_rng(7)
    cell = np.stack(np.unravel_index(np.repeat(np.arange(n ** 3), ppc), (n,) * 3), 1)
    p = np.zeros(len(cell), abi.PARTICLE_DTYPE)
    p["position"] = (cell + rng.random((len(cell), 3)) - 3.0) * scale
    p["velocity"] = rng.normal(0.0, 0.4, (len(cell), 3)) * scale
    p["q"], p["qom"] = 1.0, -1.0
    props = abi.Props.make(size=(n,) * 3, cell_width=(scale,) * 3, origin=(-3.0 * scale,) * 3, dt=0.1,
                           planet_radius=0.8 * scale, external_b=(0.0, 0.0, moment))
    field = np.zeros(abi.field_shape(props))
    field[..., :3] = rng.normal(0.0, 0.1, field.shape[:3] + (3,)) * scale  # q/m E is an acceleration
    field[..., 3:6] = rng.normal(0.0, 0.1, field.shape[:3] + (3,))
    kw = dict(mover=abi.MOVER_FIELD, bc=abi.BC_PERIODIC)
    sim = gpu_sim(props, abi.Config.make(flags=abi.F_DIPOLE_IN_GATHER | abi.F_TRACK_IDS, **kw))
    orc = OracleSim(props, abi.Config.make(flags=abi.F_DIPOLE_IN_GATHER, **kw))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(p, np.full(n ** 3, ppc, np.uint64))
        s.step(3)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    for k in ("position", "velocity"):
        np.testing.assert_allclose(a[k] / scale, b[k] / scale, rtol=0, atol=1e-12)
    sim.close()
