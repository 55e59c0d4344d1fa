"""Graph runs of 24 steps and more against eager steps: with injection, the
particles that wait for a slot have to be looked at often enough."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import gpu_sim

pytestmark = pytest.mark.gpu


def pair(props, cfg, flags=0):
    sims = [gpu_sim(props, abi.Config.make(flags=flags | g, **cfg)) for g in (abi.F_USE_GRAPH, 0)]
    if cfg["precision"] == abi.FP32:
        for s in sims:  # no autotuner trials: the same steps in both
            s.set_push_shape(256, 32, 2)
    return sims


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("size,steps", [((8, 8, 8), 24), ((8, 8, 8), 60), ((4, 64, 64), 24)])
def test_injection_into_an_empty_universe(prec, size, steps):
    """8 particles per face cell and step into cells that were laid out for
    none: no particle is lost however many steps a call takes, and the
    particles are those of eager steps."""
    props = abi.Props.make(size=size, dt=0.1)
    run, eager = pair(props, dict(precision=prec, mover=abi.MOVER_FIELD, inject_per_cell=8.0, inject_q=-1e-3,
                                  inject_qom=-1.0, inject_drift=(1.0, 0.0, 0.0), inject_vth=(0.1, 0.1, 0.1), seed=11,
                                  bc_low=(abi.BC_OPEN, abi.BC_PERIODIC, abi.BC_PERIODIC),
                                  bc_high=(abi.BC_OPEN, abi.BC_PERIODIC, abi.BC_PERIODIC)), abi.F_INJECT_LOW_X)
    got = []
    for s in (run, eager):
        s.upload_fields(np.zeros(abi.field_shape(props)))
        s.upload_particles(np.zeros(0, abi.PARTICLE_DTYPE), np.zeros(props.ncells, np.uint64))
        s.step(steps)
        p, c, _ = s.download_particles()
        cell = np.repeat(np.arange(props.ncells), c.astype(np.int64))
        key = [p["velocity"][:, a] for a in range(3)] + [p["position"][:, a] for a in range(3)] + [cell]
        got.append((p[np.lexsort(key)], c))
        s.close()
    assert len(got[0][0]) > 8 * size[1] * size[2] * min(steps, 9) // 2
    np.testing.assert_array_equal(got[0][1], got[1][1])
    for k in ("position", "velocity"):
        np.testing.assert_array_equal(got[0][0][k], got[1][0][k])
