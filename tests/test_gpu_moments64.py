"""The FP64 deposit's fixed-point moments (csrc/push64.cuh: Moments64) where
they can go wrong: cells that end a round or a work item early, particles on
faces and corners (the largest sums: all of a cell in one corner), components
of zero, of widely spread and of out-of-range magnitudes, particles outside
their cell, at the shortest and the longest work items; against exact
rational sums.

Tolerance. N particles of a cell, V the largest |Q w| among them: a term is
off by less than 2^-55 V, the reduction of a work item of 8 or more particles
by less than 2^-51 V, and every addition to a node (at most one per 8
particles and cell, one per particle for those on the FP64 path) and the
final products by 2^-53 of a partial sum below N V: N V (N / 4 + 32) 2^-53
covers them, N V (N + 32) 2^-53 where particles take the FP64 path."""
from fractions import Fraction
from itertools import product

import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import gpu_sim

pytestmark = pytest.mark.gpu

WIDTH = np.array([0.5, 1.0, 2.0])
ORIGIN = np.array([-2.0, 1.0, 0.5])
Q = -0.5
COUNTS = {"short": [1, 7, 8, 9, 16, 17, 250], "long": [3, 31, 255, 256, 257, 600]}
KINDS = ["plain", "corner", "faces", "zero", "spread", "range", "outside"]


def particles(kind, n, rng):
    """Positions in the cell (in cell widths) and velocities of n particles."""
    r, v = rng.random((n, 3)), rng.normal(0.0, 1.5, (n, 3))
    if kind == "corner":
        r[:] = rng.choice([0.0, 1.0], 3)
    elif kind == "faces":
        r = rng.choice([0.0, 0.5, 1.0, 2.0 ** -60, 1.0 - 2.0 ** -50], (n, 3))
    elif kind == "zero":
        v[:, 1] = 0.0
        v[rng.random(n) < 0.5] *= -0.0
    elif kind == "spread":
        v = rng.choice([-1.0, 1.0], (n, 3)) * 10.0 ** rng.uniform(-30, 30, (n, 3))
    elif kind == "range":
        v[:, 0] = rng.choice([1e250, -3e240, 1.0], n)
        v[:, 1] = rng.choice([2e-270, -5e-324, 1e-308], n)
    elif kind == "outside":
        r = np.where(rng.random((n, 1)) < 0.3, rng.uniform(-1.0, 2.0, (n, 3)), r)
    return r, v


@pytest.mark.parametrize("items", list(COUNTS))
@pytest.mark.parametrize("kind", KINDS)
def test_moments_match_exact_sums(kind, items):
    rng = np.random.default_rng(KINDS.index(kind) + 10 * len(items))
    size = np.array([6, 6, 6] if items == "short" else [17, 17, 17])
    cells = [np.array([1 + 2 * (i % 2), 1 + 2 * (i // 2 % 2), 1 + 2 * (i // 4)]) for i in range(len(COUNTS[items]))]
    flat = [int((c[0] * size[1] + c[1]) * size[2] + c[2]) for c in cells]
    # the longest items need 4M slots: the other cells hold particles of no charge
    counts = np.full(int(np.prod(size)), 0 if items == "short" else 800)
    counts[flat] = COUNTS[items]
    start = np.concatenate([[0], np.cumsum(counts)])
    p = np.zeros(start[-1], abi.PARTICLE_DTYPE)
    cell = np.repeat(np.arange(len(counts)), counts)
    at = np.stack([cell // (size[1] * size[2]), cell // size[2] % size[1], cell % size[2]], 1)
    p["position"] = ORIGIN + (at + 0.5) * WIDTH
    p["qom"] = 1.0
    for c, f, n in zip(cells, flat, COUNTS[items]):
        r, v = particles(kind, n, rng)
        mine = slice(start[f], start[f + 1])
        p["position"][mine] = ORIGIN + (c + r) * WIDTH
        p["velocity"][mine] = v
        p["q"][mine] = Q
    props = abi.Props.make(size=size, cell_width=WIDTH, origin=ORIGIN, dt=0.1)
    sim = gpu_sim(props, abi.Config.make(mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC))
    sim.upload_fields(np.zeros(abi.field_shape(props)))
    sim.upload_particles(p, counts.astype(np.uint64))
    sim.project()
    J, rho = sim.download_fields()[2:]
    sim.close()
    for c, f, n in zip(cells, flat, COUNTS[items]):
        mine = p[start[f]:start[f + 1]]
        exact = {k: [Fraction(0)] * 4 for k in product((0, 1), repeat=3)}
        top = [0.0] * 4
        for x, u in zip(mine["position"], mine["velocity"]):
            r = [(Fraction(float(x[a])) - Fraction(float(ORIGIN[a]))) / Fraction(float(WIDTH[a])) - int(c[a])
                 for a in range(3)]
            comp = [Fraction(float(t)) for t in u] + [Fraction(1)]
            for k in exact:
                w = Fraction(1)
                for a in range(3):
                    w *= r[a] if k[a] else 1 - r[a]
                exact[k] = [e + Fraction(Q) * t * w for e, t in zip(exact[k], comp)]
                top = [max(m, abs(float(t)), abs(float(t * w))) for m, t in zip(top, comp)]
        for k in exact:
            node = tuple(c + np.array(k))
            got = [float(t) for t in J[node]] + [float(rho[node])]
            terms = n if kind in ("range", "outside") else n / 4
            for e, g, m in zip(exact[k], got, top):
                tol = abs(Q) * m * n * (terms + 32) * 2.0 ** -53
                assert abs(Fraction(g) - e) <= Fraction(tol) + Fraction(2) ** -1070 * n, (kind, n, k, float(e), g, tol)
