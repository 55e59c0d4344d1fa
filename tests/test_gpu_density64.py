"""The FP64 deposit's charge density (csrc/push64.cuh: Moments64) where a sum
of weights is next to nothing: the particles of a cell that share a face or
an edge of it leave their opposite nodes empty; against exact rational sums,
at the shortest and the longest work items.

Tolerance. A weight (1 - r) or r, r = (x - middle) / w + 1/2, is off by a few
2^-53 on widths that are no powers of two (the start of the cell, the
difference and 1 / w round), a product of three by less than 2^-49, and the
sums round below N 2^-53 more per addition (at most one per 8 particles):
|q| N (N / 8 + 32) 2^-53."""
from fractions import Fraction

import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import gpu_sim

pytestmark = pytest.mark.gpu

Q = -0.5


def project(size, width, filler, places):
    """J and rho of a universe (origin 0) whose cell `places[i][0]` holds the
    positions and velocities places[i][1:], every other cell `filler`
    particles without charge (the longest work items need 4M slots)."""
    size = np.array(size)
    flat = [int((c[0] * size[1] + c[1]) * size[2] + c[2]) for c, _, _ in places]
    counts = np.full(int(np.prod(size)), filler)
    counts[flat] = [len(x) for _, x, _ in places]
    start = np.concatenate([[0], np.cumsum(counts)])
    p = np.zeros(start[-1], abi.PARTICLE_DTYPE)
    cell = np.repeat(np.arange(len(counts)), counts)
    at = np.stack([cell // (size[1] * size[2]), cell // size[2] % size[1], cell % size[2]], 1)
    p["position"] = (at + 0.5) * width
    p["qom"] = 1.0
    for f, (_, x, v) in zip(flat, places):
        mine = slice(start[f], start[f + 1])
        p["position"][mine], p["velocity"][mine], p["q"][mine] = x, v, Q
    props = abi.Props.make(size=size, cell_width=width, dt=0.1)
    sim = gpu_sim(props, abi.Config.make(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC))
    sim.upload_fields(np.zeros(abi.field_shape(props)))
    sim.upload_particles(p, counts.astype(np.uint64))
    sim.project()
    J, rho = sim.download_fields()[2:]
    sim.close()
    return J, rho


def corners():
    return np.array([(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)])


def exact_weights(cell, width, x):
    """The eight corners' weights of position x in `cell`, as fractions."""
    r = [Fraction(float(t)) / Fraction(float(w)) - int(c) for t, w, c in zip(x, width, cell)]
    return [np.prod([r[a] if k[a] else 1 - r[a] for a in range(3)]) for k in corners()]


@pytest.mark.parametrize("long_items", [False, True])
def test_empty_corners_of_cells_with_all_particles_on_an_edge(long_items):
    width = np.array([0.75, 0.75, 0.75])
    size, filler = ((17, 17, 17), 800) if long_items else ((6, 6, 6), 0)
    top = 1.5  # the upper faces of the cells at index 1
    places = []
    for i, (x, n) in enumerate([((1.27734375, top, top), 256), ((top, 0.80859375, 1.34765625), 256),
                                ((top, top, 1.0546875), 250), ((top, top, top), 256), ((0.75, 0.75, 0.75), 256),
                                ((1.27734375, top, top - 2.0 ** -52), 31), ((top, top, 1.0546875), 9),
                                ((0.75, top, 1.125), 1)]):
        c = np.array([1 + 2 * (i % 2), 1 + 2 * (i // 2 % 2), 1 + 2 * (i // 4)])
        places.append((c, np.tile(np.array(x) + (c - 1) * width, (n, 1)), np.zeros((n, 3))))
    _, rho = project(size, width, filler, places)
    for c, x, _ in places:
        n = len(x)
        for k, w in zip(corners(), exact_weights(c, width, x[0])):
            got = float(rho[tuple(c + k)]) * float(np.prod(width))
            assert abs(Fraction(got) - Fraction(Q) * w * n) <= abs(Q) * n * (n / 8 + 32) * 2.0 ** -53, (n, c, k)
