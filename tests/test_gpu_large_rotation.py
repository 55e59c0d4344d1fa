"""The FP64 field mover with rotations |t| = |q/m dt B / 2| up to 10^163, whose
squares overflow: the reference's operations stay finite and leave the
velocity all but unchanged. Against the oracle, to 1e-12."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import OracleSim, align_by_id, assert_states_close, gpu_sim, scenario

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qom,b,c,v", [
    (1e300, 1e-133, 1e30, 0.1),   # 100 sub-cycles, |t|^2 infinite
    (-1e300, 1e-140, 1e18, 0.1),
    (1e200, 1e-95, 1e8, 0.1),     # |t| 1e102
    (1e250, 1e-110, 1e40, 1e-3),
    (1.0, 0.3, 1.0, 0.1),         # an ordinary one beside them
])
def test_large_rotations_match_oracle(qom, b, c, v):
    props, parts, counts = scenario(7501, (4, 4, 4), dt=0.1, ppc=20, vscale=v, c=c, species=((1.0, qom),))
    field = np.zeros(abi.field_shape(props))
    field[..., 3:6] = np.array([1.0, -0.5, 0.25]) * b
    kw = dict(mover=abi.MOVER_FIELD, bc=abi.BC_PERIODIC)
    sim, orc = gpu_sim(props, abi.Config.make(flags=abi.F_TRACK_IDS, **kw)), OracleSim(props, abi.Config.make(**kw))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(parts, counts)
        s.step(2)
    p, q = align_by_id(sim.download_particles(), orc.download_particles())
    assert np.isfinite(q["velocity"]).all() and not np.array_equal(q["position"], parts["position"])
    assert_states_close(p, q, rtol=1e-12, atol=1e-12, what=str(qom))
    sim.close()
