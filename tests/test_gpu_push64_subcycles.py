"""The FP64 push's short items where the dipole can ask for many sub-cycles
(csrc/particles_fp64.cu many_sub_cycles): fields below and far above the line
at 8 (the loads below ask for dt 4 |q/m| B^2 / pi = 5.7 and 90), against the
oracle, and in a batch in which one universe is above it.

Tolerances: a sub-cycle adds at most 32 eps of the speed, up to 100 of them
4e-13; the position's share of that turns the field by 3 dx / r over 20 rad,
60 * 0.1 * 4e-13 = 2e-12; 1e-11 for states, and for densities of up to 4000
terms."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import Batch, abi
from common import OracleSim, align_by_id, assert_states_close, gpu_sim
from test_gpu_push64_large import BC, load

pytestmark = pytest.mark.gpu


def universe(size, mean, seed, bz):
    props, parts, counts = load(size, mean, seed)
    props.external_b[2] = bz
    return props, parts, counts


# 0.06, 0.97 and 3.8 million slots: items of 8, and of 64 and 256 below the line, 32 above it
@pytest.mark.parametrize("size,mean", [((6, 6, 5), 200), ((13, 14, 14), 350), ((20, 19, 21), 440)])
@pytest.mark.parametrize("mover,flags", [(abi.MOVER_DIPOLE, 0), (abi.MOVER_FIELD, abi.F_DIPOLE_IN_GATHER)])
@pytest.mark.parametrize("bz", [1.5, 6.0])
def test_matches_oracle(size, mean, mover, flags, bz):
    props, parts, counts = universe(size, mean, mean, bz)
    field = np.random.default_rng(3).normal(0.0, 0.5, abi.field_shape(props))
    kw = dict(mover=mover, projector=abi.PROJECT_CIC, **BC)
    sim = gpu_sim(props, abi.Config.make(flags=flags | abi.F_TRACK_IDS, **kw))
    orc = OracleSim(props, abi.Config.make(flags=flags, **kw))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(parts, counts)
        s.step(1)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    assert_states_close(a, b, rtol=1e-11, atol=1e-11, what=str((size, bz)))
    orc.project()  # the GPU's J is of the moved particles
    for x, y in zip(sim.download_fields()[2:], orc.download_fields()[2:]):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * np.abs(y).max())
    sim.close()


def test_batch_with_one_strong_dipole_matches_single_universes():
    loads = [universe(s, m, 20 + i, bz) for i, (s, m, bz) in enumerate([
        ((10, 10, 9), 450, 1.5), ((9, 10, 8), 500, 6.0), ((8, 9, 10), 480, 0.0)])]
    cfg = abi.Config.make(mover=abi.MOVER_DIPOLE, projector=abi.PROJECT_CIC, flags=abi.F_TRACK_IDS, **BC)
    batch = Batch([p for p, _, _ in loads], cfg)
    singles = [gpu_sim(p, cfg) for p, _, _ in loads]
    for i, (_, parts, counts) in enumerate(loads):
        for s in (batch.universe(i), singles[i]):
            s.upload_particles(parts, counts)
    batch.step(2)
    for i, s in enumerate(singles):
        s.step(2)
        u = batch.universe(i)
        a, b = align_by_id(u.download_particles(), s.download_particles())
        for k in ("position", "velocity"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=str(i))
        for x, y in zip(u.download_fields()[2:], s.download_fields()[2:]):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * np.abs(y).max())
        s.close()
    batch.close()
