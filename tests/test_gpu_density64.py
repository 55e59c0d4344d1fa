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


# Tolerance of the sums of N particles of a cell, V the largest velocity
# component among them (1 for the density), on widths that are powers of two
# and positions whose difference from the cell's middle is exact. With items
# of I particles a lane adds up to r = ceil(min(N, I) / 8) of them in units of
# 2^(room - 63) of the power of two above V, room = ceil(log2 r): at most 32
# units a particle over the eight corners' sums (products, weights and shifts
# round down, by less than 4 units a moment). The lanes' sums are then shifted
# by at most 2 + log2(N) - room bits, half a unit each: 2 N 2^-63 for each of
# min(N, 32) lanes. Last, each of A = ceil(N / I) items rounds its product with
# the charge and its addition to the node by 2^-53 of a sum below S = sum |Q v
# w|, and the finalisation by nothing (the volume is a power of two):
# 2 V N (32 2^room + 2 min(N, 32)) 2^-63 |Q| + 2 A 2^-53 S.
SPARSE = [1, 2, 3, 4, 7, 8, 9, 16, 40, 255, 256, 600]


@pytest.mark.parametrize("kind", ["plain", "far", "faces"])
@pytest.mark.parametrize("long_items", [False, True])
def test_sums_keep_their_last_places(long_items, kind):
    """However long the launch's work items are, the sums of a cell with few
    particles are as fine as their number allows."""
    width = np.array([0.5, 1.0, 2.0])
    size, filler, item = ((17, 17, 17), 800, 256) if long_items else ((8, 8, 8), 0, 8)
    rng = np.random.default_rng(["plain", "far", "faces"].index(kind))
    places = []
    for i, n in enumerate(SPARSE):
        c = np.array([1 + 2 * (i % 3), 1 + 2 * (i // 3 % 2), 1 + 2 * (i // 6)])
        r = rng.integers(1, 2 ** 20, (n, 3)) / 2.0 ** 20
        if kind == "far":
            r = r / 64.0  # the far node gets 2^-18 or less of a particle
        elif kind == "faces":
            r = rng.choice([0.0, 0.25, 1.0, 2.0 ** -20, 1.0 - 2.0 ** -30], (n, 3))
        places.append((c, (c + r) * width, rng.normal(0.0, 1.5, (n, 3))))
    J, rho = project(size, width, filler, places)
    for c, x, v in places:
        n = len(x)
        rounds = -(-min(n, item) // 8)
        fine = 2.0 * n * (32 * 2 ** (rounds - 1).bit_length() + 2 * min(n, 32)) * 2.0 ** -63
        weights = [exact_weights(c, width, t) for t in x]
        comps = [[Fraction(float(t)) for t in v[:, a]] for a in range(3)] + [[Fraction(1)] * n]
        for i, k in enumerate(corners()):
            got = [float(t) for t in J[tuple(c + k)]] + [float(rho[tuple(c + k)])]
            for a, q in enumerate(comps):
                terms = [t * w[i] for t, w in zip(q, weights)]
                top, total = max(abs(t) for t in q), sum(abs(t) for t in terms)
                tol = abs(Q) * (Fraction(fine) * top + 2 * -(-n // item) * total / 2 ** 53)
                assert abs(Fraction(got[a]) - Fraction(Q) * sum(terms)) <= tol, (n, k, a, got[a], float(tol))


def test_cells_reach_their_nodes_in_one_addition():
    """Work items of 8, cells of 16 items each, no two of which share a node:
    the items' sums are added in a fixed order and reach the nodes in one
    addition each, so every projection gives the same bits (several additions
    to a node round by their order)."""
    n, per = 9, 128
    rng = np.random.default_rng(9)
    c = np.array([(x, y, z) for x in range(0, n, 2) for y in range(0, n, 2) for z in range(0, n, 2)])
    counts = np.zeros(n ** 3, np.uint64)
    counts[(c[:, 0] * n + c[:, 1]) * n + c[:, 2]] = per
    p = np.zeros(len(c) * per, abi.PARTICLE_DTYPE)
    p["position"] = np.repeat(c, per, 0) + rng.random((len(p), 3))
    p["velocity"] = rng.normal(0.0, 1.0, (len(p), 3))
    p["q"], p["qom"] = Q, 1.0
    props = abi.Props.make(size=(n,) * 3, dt=0.1)
    sim = gpu_sim(props, abi.Config.make(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC))
    sim.upload_fields(np.zeros(abi.field_shape(props)))
    sim.upload_particles(p, counts)
    sim.project()
    first = sim.download_fields()[2:]
    for _ in range(15):
        sim.project()
        for a, b in zip(sim.download_fields()[2:], first):
            np.testing.assert_array_equal(a, b)
    sim.close()
