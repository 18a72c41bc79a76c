"""Springs near a rest position far from zero: K (q - q0) is formed from the
difference, so the force keeps the digits that q and q0 do not share. Sliders
and pins side by side on Ground, with one spring, two of one rest position,
two of different ones, and a damper beside them; against the CPU oracle
element by element at the FP64 parity tolerance of a realize (1e-12)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from simbody_gb300 import Batch, Topology
from simbody_gb300 import _native as N

pytestmark = pytest.mark.gpu

# per mobility: (kind, coefficient, rest position); kind 0 a spring, 1 a damper
FORCES = [[(0, 1e4 / 3, 1e6 / 7)], [(0, 3.3e3, -7.1e5), (0, 5.7e3, -7.1e5)], [(0, 2.3e4, 4.1e5), (0, 10.1, 4.1e5 + 0.1), (1, 0.5, 0.0)],
          [(1, 2.0, 0.0)], []]


@pytest.fixture(scope="module")
def system():
    n = 2 * len(FORCES)
    bodies, forces = (N.BodyDesc * n)(), []
    for k, b in enumerate(bodies):
        b.parent, b.mobilizer, b.mass = 0, (N.SBG_SLIDER, N.SBG_PIN)[k // len(FORCES)], 1.5
        b.unit_inertia[0] = b.unit_inertia[1] = b.unit_inertia[2] = 0.4
        for j in (0, 4, 8):
            b.X_PF[j] = b.X_BM[j] = 1.0
        forces += [(kind, k + 1, 0, 0, coef, q0) for kind, coef, q0 in FORCES[k % len(FORCES)]]
    arr = (N.MobilityForceDesc * len(forces))(*forces)
    d = N.SystemDesc(n, len(forces), 0, 0, (C.c_double * 3)(0, 0, 0), bodies, arr, None)
    return d, (bodies, arr)


@pytest.mark.parametrize("n", [1, 33])
def test_springs_near_a_far_rest_position(engine, system, n):
    d, keep = system
    nb = d.nbodies
    rng = np.random.default_rng(n)
    rest = np.array([f[0][2] if f else 0.0 for f in FORCES] * 2)
    y = np.concatenate([rest + 1e-3 * rng.uniform(0.5, 1, size=(n, nb)), rng.uniform(0.5, 1, size=(n, nb))], axis=1)
    got, st = Batch([Topology(d, keepalive=keep)], np.zeros(n, np.int32)).realize_acceleration_from(y.ravel())
    sys_ = (N.SystemDesc * 1)(d)
    ref, _ = O.realize(sys_, 1, np.zeros(n, np.int32), np.arange(n + 1) * 2 * nb, y.ravel())
    assert (st == 0).all()
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)


def test_a_position_without_a_spring_is_not_multiplied(engine, system):
    """An infinite coordinate that no spring acts on gives the same bits alone
    and beside instances whose bodies have springs there."""
    d, keep = system
    bodies = (N.BodyDesc * d.nbodies)(*[d.bodies[k] for k in range(d.nbodies)])
    bare = N.SystemDesc(d.nbodies, 0, 0, 0, (C.c_double * 3)(0, 0, 0), bodies, None, None)
    topo = [Topology(bare, keepalive=bodies), Topology(d, keepalive=keep)]
    y = np.zeros((2, 2 * d.nbodies))
    y[0, :len(FORCES)] = np.inf  # the sliders
    alone, sa = Batch(topo[:1], np.zeros(1, np.int32)).realize_acceleration_from(y[0])
    both, sb = Batch(topo, np.arange(2, dtype=np.int32)).realize_acceleration_from(y.ravel())
    assert sa[0] == sb[0] == N.INST_NONFINITE and np.isfinite(alone).all()  # by the state, not by the forces
    np.testing.assert_array_equal(alone, both[:alone.size])
