"""Graph runs of 24 steps and more, which replay several steps at a time
(the moves with the next step's field solve among them), against eager steps:
bit for bit where no sum depends on the order of additions, with re-layouts on
the way, and with injection, where the particles that wait for a slot have to
be looked at often enough."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import align_by_id, gpu_sim, scenario
from test_gpu_fieldstep import sparse_particles

pytestmark = pytest.mark.gpu


def pair(props, cfg, flags=0):
    sims = [gpu_sim(props, abi.Config.make(flags=flags | g, **cfg)) for g in (abi.F_USE_GRAPH, 0)]
    if cfg["precision"] == abi.FP32:
        for s in sims:  # no autotuner trials: the same steps in both
            s.set_push_shape(256, 32, 2)
    return sims


@pytest.mark.parametrize("steps", [24, 25, 33])
@pytest.mark.parametrize("prec,solver,flags", [
    (abi.FP64, abi.SOLVER_LEAPFROG, abi.F_J_DIV8),
    (abi.FP64, abi.SOLVER_FORWARD, 0),
    (abi.FP64, abi.SOLVER_STATIC, 0),
    (abi.FP32, abi.SOLVER_LEAPFROG, abi.F_REFRESH_NODE_B)])
def test_long_graph_runs_match_eager_steps(prec, solver, flags, steps):
    props, _, _ = scenario(7401, (8, 8, 8), width=(0.6, 0.5, 0.7), dt=0.05, ppc=1)
    parts, counts = sparse_particles(props, [(0, 0, 0), (7, 3, 0), (3, 7, 5), (5, 0, 7), (2, 4, 3)], 7402)
    parts["q"][1::2], parts["qom"][1::2] = 0.25, 0.1  # two species
    rng = np.random.default_rng(7403)
    run, eager = pair(props, dict(precision=prec, mover=abi.MOVER_FIELD, solver=solver, projector=abi.PROJECT_CIC,
                                  bc=abi.BC_PERIODIC), abi.F_TRACK_IDS | flags)
    f, bc = rng.normal(0.0, 0.02, abi.field_shape(props)), rng.normal(0.0, 0.02, abi.bcfield_shape(props))
    for s in (run, eager):
        s.upload_fields(f, bc, None)
        s.upload_particles(parts, counts)
        s.step(steps)
    for a, b in zip(run.download_fields(), eager.download_fields()):
        np.testing.assert_array_equal(a, b)
    a, b = align_by_id(run.download_particles(), eager.download_particles())
    np.testing.assert_array_equal(a["position"], b["position"])
    np.testing.assert_array_equal(a["velocity"], b["velocity"])
    for k in ("steps", "particles", "migrated_last", "removed_last", "pending_last"):
        assert run.stats()[k] == eager.stats()[k], k
    run.close()
    eager.close()


@pytest.mark.parametrize("solver", [abi.SOLVER_STATIC, abi.SOLVER_LEAPFROG])
def test_long_graph_runs_relayout(solver):
    """A converging flow of 16,000 particles: the middle cells run out of
    slots again and again. Without fields of their own the particles agree bit
    for bit; with them (J's additions in any order) to 1e-10."""
    props, parts, counts = scenario(7411, (8, 8, 8), dt=0.05, ppc=32, vscale=0.01, species=((-1e-4, -1.0),))
    parts["velocity"] -= 0.5 * (parts["position"] - 4.0)
    run, eager = pair(props, dict(precision=abi.FP64, mover=abi.MOVER_FIELD, solver=solver, slack_min=1,
                                  projector=abi.PROJECT_CIC if solver else abi.PROJECT_NONE, bc=abi.BC_PERIODIC),
                      abi.F_TRACK_IDS)
    for s in (run, eager):
        s.upload_fields(np.zeros(abi.field_shape(props)), np.zeros(abi.bcfield_shape(props)), None)
        s.upload_particles(parts, counts)
        s.step(45)
        assert s.stats()["rebuilds"] >= 2 and s.particle_count() == len(parts)
    tol = 1e-10 if solver else 0.0
    for a, b in zip(run.download_fields(), eager.download_fields()):
        np.testing.assert_allclose(a, b, rtol=0, atol=tol)
    a, b = align_by_id(run.download_particles(), eager.download_particles())
    for k in ("position", "velocity"):
        np.testing.assert_allclose(a[k], b[k], rtol=0, atol=tol)
    run.close()
    eager.close()


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
