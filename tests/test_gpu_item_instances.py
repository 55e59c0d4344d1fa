"""The FP32 push's instance for launches whose tiles all have at most
`item_cells` cells (no slot mode) at the edges of that rule: the shape's limit
one below, at and above the most cells of a tile, two populations of different
density in one launch, single and batched. Particles are equal bit for bit
whichever instance and mode runs; J and rho, whose sums the modes order
differently, to 1e-5 of their peak (FP32 moments of up to 200 terms: 200 eps /
2)."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import Batch, abi
from common import align_by_id, gpu_sim

pytestmark = pytest.mark.gpu

N = 10


def load(dense):
    """`dense` particles per cell and species (the second has a fifth)."""
    rng = np.random.default_rng(dense)
    nc = N ** 3
    per = [dense, max(1, dense // 5)]
    cell = np.repeat(np.arange(nc), sum(per))
    c = np.stack(np.unravel_index(cell, (N,) * 3), 1)
    p = np.zeros(len(cell), abi.PARTICLE_DTYPE)
    p["position"] = c + rng.random((len(c), 3))
    p["velocity"] = rng.normal(0.0, 0.3, (len(c), 3))
    second = np.tile(np.arange(sum(per)) >= per[0], nc)
    p["q"], p["qom"] = np.where(second, 1e-3, -1e-3), np.where(second, 0.1, -1.0)
    return p, np.full(nc, sum(per), np.uint64)


@pytest.mark.parametrize("flags", [0, abi.F_DIPOLE_IN_GATHER | abi.F_USE_GRAPH])
@pytest.mark.parametrize("dense", [25, 110, 160])
def test_item_instance_matches_slot_mode(dense, flags):
    props = abi.Props.make(size=(N,) * 3, dt=0.1, origin=(-5.0,) * 3, planet_radius=0.5, external_b=(0.0, 0.0, 0.5))
    cfg = abi.Config.make(precision=abi.FP32, mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC, bc=abi.BC_PERIODIC,
                          flags=abi.F_TRACK_IDS | flags)
    parts, counts = load(dense)
    parts["position"] -= 5.0
    field = np.random.default_rng(1).normal(0.0, 0.1, abi.field_shape(props))
    sims = []
    # slot mode everywhere, then items in the tiles of at most so many cells;
    # the two populations' tiles have up to 27 and 64, 9 and 32, or 6 and 22
    for item_cells in (0, 6, 9, 21, 22, 23, 27, 31, 32):
        sim = gpu_sim(props, cfg)
        sim.set_push_shape(64, item_cells, 2)
        sim.upload_fields(field)
        sim.upload_particles(parts, counts)
        sim.step(6)
        sims.append((sim.download_particles(), sim.download_fields()[2:]))
        sim.close()
    for got in sims[1:]:
        a, b = align_by_id(got[0], sims[0][0])
        for k in ("position", "velocity"):
            np.testing.assert_array_equal(a[k], b[k])
        for x, y in zip(got[1], sims[0][1]):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-5 * np.abs(y).max())


def test_batch_of_full_and_sparse_universes():
    props = abi.Props.make(size=(N,) * 3, dt=0.1)
    cfg = abi.Config.make(precision=abi.FP32, mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC, bc=abi.BC_PERIODIC,
                          flags=abi.F_TRACK_IDS, block_size=256)
    field = np.random.default_rng(2).normal(0.0, 0.1, abi.field_shape(props))
    loads = [load(110), load(150), load(3)]
    for pick in ((0, 1), (0, 1, 2)):  # full cells only, then a sparse universe among them
        batch = Batch([props] * len(pick), cfg)
        singles = [gpu_sim(props, cfg) for _ in pick]
        for i, j in enumerate(pick):
            for s in (batch.universe(i), singles[i]):
                s.upload_fields(field)
                s.upload_particles(*loads[j])
        batch.step(5)
        for i, s in enumerate(singles):
            s.step(5)
            a, b = align_by_id(batch.universe(i).download_particles(), s.download_particles())
            for k in ("position", "velocity"):
                np.testing.assert_array_equal(a[k], b[k])
            for x, y in zip(batch.universe(i).download_fields()[2:], s.download_fields()[2:]):
                np.testing.assert_allclose(x, y, rtol=0, atol=1e-5 * np.abs(y).max())
            s.close()
        batch.close()
