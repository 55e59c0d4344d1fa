"""The FP64 push (csrc/push64.cuh) where its work split can go wrong: cells
longer than a tile (cut at span boundaries), cells that start in one tile and
end in the next, empty and single-particle cells, item lengths that leave a
ragged last round, several populations, every policy pair; against the
oracle. Counts and ids exact, states to 1e-12, densities to 1e-11 of their
peak (sums of up to 4000 terms in another order: 4000 eps / 2 < 1e-12)."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import OracleSim, align_by_id, assert_states_close, gpu_sim
from test_gpu_dipole64 import KINDS, edge_particles

pytestmark = pytest.mark.gpu

LOADS = {
    "ragged": ((5, 4, 3), lambda r, nc: r.integers(0, 40, nc)),
    "single": ((4, 4, 4), lambda r, nc: r.integers(0, 2, nc)),
    "rounds": ((3, 3, 3), lambda r, nc: np.arange(nc) + 1),
    "tiles": ((7, 5, 6), lambda r, nc: r.choice([120, 250, 511, 3], nc)),
    "long": ((2, 2, 2), lambda r, nc: np.array([2500, 0, 1, 1030, 4000, 7, 900, 64])),
}


def load(name, species):
    size, per = LOADS[name]
    rng = np.random.default_rng(len(name))
    nc = int(np.prod(size))
    counts = np.asarray(per(rng, nc)).astype(np.int64)
    cell = np.repeat(np.arange(nc), counts)
    n = len(cell)
    c = np.stack([cell // (size[1] * size[2]), (cell // size[2]) % size[1], cell % size[2]], 1)
    w, org = np.array([0.75, 1.0, 1.5]), np.array([-2.0, 1.0, 0.5])
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    p["position"] = org + (c + rng.random((n, 3))) * w
    p["velocity"] = rng.normal(0.0, 1.5, (n, 3))
    which = rng.integers(0, len(species), n)
    p["q"], p["qom"] = np.array(species)[which].T
    props = abi.Props.make(size=size, cell_width=w, dt=0.1, planet_radius=0.4, object_center=(-1.0, 2.0, 1.5),
                           origin=org, external_b=(0.0, 0.0, 1.5))
    return props, p, counts.astype(np.uint64)


@pytest.mark.parametrize("name", list(LOADS))
@pytest.mark.parametrize("mover,project,flags", [
    (abi.MOVER_FIELD, abi.PROJECT_CIC, 0),
    (abi.MOVER_FIELD, abi.PROJECT_CIC, abi.F_DIPOLE_IN_GATHER | abi.F_GATHER_DIV_VOL | abi.F_J_DIV8),
    (abi.MOVER_FIELD, abi.PROJECT_NONE, abi.F_DIPOLE_IN_GATHER),
    (abi.MOVER_DIPOLE, abi.PROJECT_CIC, 0),
    (abi.MOVER_DIPOLE, abi.PROJECT_NONE, 0)])
def test_fp64_push_splits_match_oracle(name, mover, project, flags):
    props, parts, counts = load(name, [(-0.5, -1.0), (0.25, 2.0)])
    rng = np.random.default_rng(3)
    field = rng.normal(0.0, 0.5, abi.field_shape(props))
    kw = dict(mover=mover, projector=project, bc_low=[abi.BC_PERIODIC, abi.BC_REFLECT, abi.BC_OPEN],
              bc_high=[abi.BC_PERIODIC, abi.BC_REFLECT, abi.BC_REFLECT])
    sim = gpu_sim(props, abi.Config.make(flags=flags | abi.F_TRACK_IDS, **kw))
    orc = OracleSim(props, abi.Config.make(flags=flags, **kw))
    for s in (sim, orc):
        s.upload_fields(field)
        s.upload_particles(parts, counts)
        s.step(3)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    assert_states_close(a, b, rtol=1e-12, atol=1e-12, what=name)
    if project == abi.PROJECT_CIC:  # the GPU's J is of the moved particles
        orc.project()
        for x, y in zip(sim.download_fields()[2:], orc.download_fields()[2:]):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * np.abs(y).max())
    sim.close()


@pytest.mark.parametrize("kind", KINDS)
def test_fp64_dipole_push_edges_match_oracle(kind):
    n = 8
    parts = edge_particles(kind, 4000, 9, 4.0)
    parts["qom"] = np.resize(parts["qom"][:12], len(parts))  # a universe has at most 16 species
    cell = np.clip(np.floor(parts["position"] + 4.0).astype(np.int64), 0, n - 1)
    flat = (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2]
    parts = parts[np.argsort(flat, kind="stable")]
    counts = np.bincount(flat, minlength=n ** 3).astype(np.uint64)
    props = abi.Props.make(size=(n,) * 3, dt=0.05, planet_radius=0.5, origin=(-4.0,) * 3,
                           external_b=(0.0, 0.0, 2.0))
    sim = gpu_sim(props, abi.Config.make(flags=abi.F_TRACK_IDS))
    orc = OracleSim(props, abi.Config.make())
    for s in (sim, orc):
        s.upload_particles(parts, counts)
        s.step(8)
    a, b = align_by_id(sim.download_particles(), orc.download_particles())
    # the smoke run's bar: the host's pow is not correctly rounded for about
    # one argument in 10^4, so single bits may differ
    assert_states_close(a, b, rtol=1e-12, atol=1e-12, what=kind)
    sim.close()
