"""J and rho of universes that are thin along an axis, at the edges of the rule
by which their finalisation goes by rows or by nodes (160,000 nodes, 16,384
rows). A particle in the middle of each cell, velocities of a few eighths: every
sum is exact, the periodic duplicates included, and one correctly rounded
quotient (or an exact product) follows, so the results are equal bit for bit
to the same sums in numpy."""
import numpy as np
import pytest

from allscale_ipic3d_gb300 import abi
from common import gpu_sim

pytestmark = pytest.mark.gpu


def expected(values, vol, div8):
    """Node sums of values / 8 per cell and corner, both faces of an axis
    added up, over vol [/ 8]."""
    s = values.shape[:3]
    raw = np.zeros(tuple(n + 1 for n in s) + values.shape[3:])
    for k in np.ndindex(2, 2, 2):
        raw[tuple(slice(a, a + n) for a, n in zip(k, s))] += values / 8
    for axis in range(3):
        first, last = [slice(None)] * 3, [slice(None)] * 3
        first[axis], last[axis] = 0, s[axis]
        both = raw[tuple(first)] + raw[tuple(last)]
        raw[tuple(first)] = raw[tuple(last)] = both
    return raw / vol / 8 if div8 else raw / vol


@pytest.mark.parametrize("prec,width,flags", [
    (abi.FP64, (0.75, 1.0, 1.25), abi.F_J_DIV8),  # quotients
    (abi.FP64, (0.5, 1.0, 2.0), 0),               # products
    (abi.FP32, (0.5, 1.0, 2.0), abi.F_J_DIV8)])
@pytest.mark.parametrize("size", [(16384, 1, 1), (16385, 1, 1), (128, 128, 3), (113, 145, 2), (1, 5000, 32),
                                  (1, 5000, 33), (2, 79999, 1), (400, 1, 401), (54, 54, 54), (55, 55, 55),
                                  (140000, 1, 1)])
def test_thin_grids(size, prec, width, flags):
    rng = np.random.default_rng(sum(size))
    props = abi.Props.make(size=size, cell_width=width, dt=0.1)
    n = props.ncells
    cell = np.stack(np.unravel_index(np.arange(n), size), 1)
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    p["position"] = (cell + 0.5) * width
    p["velocity"] = rng.integers(-64, 65, (n, 3)) / 8.0
    p["q"], p["qom"] = -0.5, -1.0
    sim = gpu_sim(props, abi.Config.make(precision=prec, mover=abi.MOVER_FIELD, projector=abi.PROJECT_CIC,
                                         flags=flags))
    sim.upload_fields(np.zeros(abi.field_shape(props)))
    sim.upload_particles(p, np.ones(n, np.uint64))
    sim.project()
    J, rho = sim.download_fields()[2:]
    sim.close()
    vol, div8 = float(np.prod(width)), bool(flags & abi.F_J_DIV8)
    np.testing.assert_array_equal(J, expected(-0.5 * p["velocity"].reshape(size + (3,)), vol, div8))
    np.testing.assert_array_equal(rho, expected(np.full(size, -0.5), vol, div8))
