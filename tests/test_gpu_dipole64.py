"""The FP64 dipole step on the integer pipe (csrc/dipole64.cuh) where its
range ends and the FP64 path takes over: coordinates that are zero, tiny or
huge, fields that vanish or need sub-cycles, q/m of zero and of extreme size,
velocities of zero and subnormal size. Histograms of the tracer against the
oracle, bit for bit."""
import numpy as np
import pytest

import allscale_ipic3d_gb300 as ipg
from allscale_ipic3d_gb300 import abi

pytestmark = pytest.mark.gpu

KINDS = ["plane", "axis", "tiny", "huge", "weak", "qom", "slow", "mixed"]


def edge_particles(kind, n, seed, L):
    """Particles of an edge kind in a box of half width L around the origin."""
    rng = np.random.default_rng(seed)
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    x = rng.uniform(-0.95, 0.95, (n, 3)) * L
    v = rng.normal(0.0, 0.3, (n, 3)) * L
    qom = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-1, 1, n)
    some = rng.random(n) < 0.5
    if kind == "plane":  # z = 0: B_x = B_y = +-0; in-plane motion keeps it
        x[:, 2] = np.where(some, 0.0, -0.0)
        v[some, 2] = 0.0
    elif kind == "axis":
        x[:, :2] = 0.0
        x[some, 0] = -0.0
    elif kind == "tiny":
        x[:, 0] *= 10.0 ** rng.uniform(-60, 0, n)
        x[:, 1] *= 10.0 ** rng.uniform(-330, 0, n)
    elif kind == "huge":
        x *= 10.0 ** rng.uniform(-2, 0, (n, 1))
    elif kind == "weak":
        qom *= 10.0 ** rng.uniform(-300, -20, n)
    elif kind == "qom":
        qom = rng.choice([0.0, -0.0, 1e-310, 1e-40, 1e40, 1e300, 30.0, -30.0], n)
    elif kind == "slow":
        v *= rng.choice([0.0, 1e-310, 1e-200, 1e-30, -1.0], (n, 3))
    p["position"], p["velocity"], p["q"], p["qom"] = x, v, 1.0, qom
    return p


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("unit", [1.0, 2.0 ** -90, 2.0 ** 95])
def test_tracer_edges_match_oracle(kind, unit):
    from test_tracer_oracle import oracle_trace
    L = 4.0 * unit
    props = abi.Props.make(size=(8, 8, 8), cell_width=(unit,) * 3, dt=0.05, planet_radius=0.5 * unit,
                           origin=(-L,) * 3, external_b=(0.0, 0.0, 2.0))
    parts = edge_particles(kind, 3000, 5, L)
    frames = ipg.trace_frames(25, 4)
    want = oracle_trace(props, parts, 25, 4, frames)
    assert want.sum() > 0
    np.testing.assert_array_equal(ipg.trace(props, parts, 25, 4, frames), want)
