"""The FP64 push (csrc/push64.cuh) with the work splits of larger launches:
items of 16 to 256 particles that end in a ragged round, spans of 4 tiles cut
at the capacity's end, blocks that take several rounds (no deposit, 3,648
tiles and more), and batches whose universes end inside a span. Against the
oracle (counts and ids exact, states to 1e-12, densities to 1e-11 of their
peak: sums of up to 4000 terms, 4000 eps / 2 < 1e-12), and a batch against
single universes bit for bit."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import Batch, abi
from common import OracleSim, align_by_id, assert_states_close, gpu_sim

pytestmark = pytest.mark.gpu

BC = dict(bc_low=[abi.BC_PERIODIC, abi.BC_REFLECT, abi.BC_OPEN],
          bc_high=[abi.BC_PERIODIC, abi.BC_REFLECT, abi.BC_REFLECT])


def load(size, mean, seed):
    """Uneven cells: empty ones, single particles, a few of several tiles."""
    rng = np.random.default_rng(seed)
    nc = int(np.prod(size))
    counts = rng.choice([0, 1, mean // 3, mean, mean + 7, 2 * mean], nc, p=[0.05, 0.05, 0.1, 0.5, 0.2, 0.1])
    counts[rng.integers(0, nc, 3)] = [2500, 1030, 4000]
    cell = np.repeat(np.arange(nc), counts)
    n = len(cell)
    c = np.stack([cell // (size[1] * size[2]), (cell // size[2]) % size[1], cell % size[2]], 1)
    w, org = np.array([0.75, 1.0, 1.5]), np.array([-2.0, 1.0, 0.5])
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    p["position"] = org + (c + rng.random((n, 3))) * w
    p["velocity"] = rng.normal(0.0, 1.0, (n, 3))
    p["q"], p["qom"] = np.array([(-0.5, -1.0), (0.25, 2.0)])[rng.integers(0, 2, n)].T
    props = abi.Props.make(size=size, cell_width=w, dt=0.1, planet_radius=1.3, object_center=(-1.0, 2.0, 1.5),
                           origin=org, external_b=(0.0, 0.0, 1.5))
    return props, p, counts.astype(np.uint64)


# 0.35, 0.97 and 3.8 million slots: items of 16, 64 (32 without deposit), 256 (32)
@pytest.mark.parametrize("size,mean", [((11, 10, 10), 270), ((13, 14, 14), 350), ((20, 19, 21), 440)])
@pytest.mark.parametrize("mover,project,flags", [
    (abi.MOVER_FIELD, abi.PROJECT_CIC, abi.F_GATHER_DIV_VOL),
    (abi.MOVER_DIPOLE, abi.PROJECT_CIC, 0),
    (abi.MOVER_DIPOLE, abi.PROJECT_NONE, 0)])
def test_large_splits_match_oracle(size, mean, mover, project, flags):
    props, parts, counts = load(size, mean, mean)
    field = np.random.default_rng(3).normal(0.0, 0.5, abi.field_shape(props))
    kw = dict(mover=mover, projector=project, **BC)
    sim = gpu_sim(props, abi.Config.make(flags=flags | abi.F_TRACK_IDS, **kw))
    orc = OracleSim(props, abi.Config.make(flags=flags, **kw))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(parts, counts)
        s.step(1)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    assert_states_close(a, b, rtol=1e-12, atol=1e-12, what=str(size))
    if project == abi.PROJECT_CIC:  # the GPU's J is of the moved particles
        orc.project()
        for x, y in zip(sim.download_fields()[2:], orc.download_fields()[2:]):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * np.abs(y).max())
    sim.close()


def test_batch_of_partial_spans_matches_single_universes():
    loads = [load(s, m, 10 + i) for i, (s, m) in enumerate([((7, 6, 5), 350), ((5, 9, 6), 300), ((8, 7, 6), 290),
                                                          ((4, 5, 6), 620), ((6, 6, 6), 330), ((7, 7, 7), 240)])]
    cfg = abi.Config.make(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC, flags=abi.F_TRACK_IDS, **BC)
    batch = Batch([p for p, _, _ in loads], cfg)
    singles = [gpu_sim(p, cfg) for p, _, _ in loads]
    rng = np.random.default_rng(5)
    for i, (props, parts, counts) in enumerate(loads):
        field = rng.normal(0.0, 0.5, abi.field_shape(props))
        for s in (batch.universe(i), singles[i]):
            s.upload_fields(field)
            s.upload_particles(parts, counts)
    batch.step(2)
    tiles = 0
    for i, s in enumerate(singles):
        s.step(2)
        tiles += s.stats()["capacity"] // 1024
        u = batch.universe(i)
        a, b = align_by_id(u.download_particles(), s.download_particles())
        for k in ("position", "velocity"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=str(i))
        for x, y in zip(u.download_fields()[2:], s.download_fields()[2:]):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-12 * np.abs(y).max())
        s.close()
    assert tiles >= 304
    batch.close()
