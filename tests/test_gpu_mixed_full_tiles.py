"""FP64 work of a mixed batch on full tiles and one instance to a block.
Instances with contact spheres take the FP64 path of the mixed form always: of
a batch with contact trees, trees without, or both, in numbers at either side of
what goes one to a block, they get the bits of an FP64 batch's realize and of a
small mixed batch's steps, whichever kernel takes them."""
import time

import numpy as np
import pytest

from simbody_gb300 import Batch, Topology, Workload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trees():
    w3, w8 = Workload(3, 24), Workload(8, 24)
    topo = [Topology(w.systems[k], keepalive=w) for w in (w3, w8) for k in range(24)]
    y = [w.y0[w.instance_slice(k)] for w in (w3, w8) for k in range(24)]
    return topo, y


@pytest.mark.parametrize("n,contact", [(1, 1.0), (40, 1.0), (300, 1.0), (700, 1.0), (700, 0.02), (700, 0.1), (3100, 0.07),
                                       (3100, 1.0)])
@pytest.mark.parametrize("kinds", [24, 1])
def test_contact_instances_get_the_fp64_bits(engine, trees, n, contact, kinds):
    topo, y = trees
    rng = np.random.default_rng(n)
    touch = rng.random(n) < contact
    which = (rng.integers(0, kinds, n) + 24 * touch).astype(np.int32)
    y0 = np.concatenate([y[k] for k in which])
    bm, b64 = (Batch(topo, which, precision=p) for p in ("mixed", "fp64"))
    off = bm.y_offsets
    elems = np.repeat(touch, np.diff(off))

    def same(a, b):
        np.testing.assert_array_equal(a[elems], b[elems])
        assert np.isfinite(a).all()

    before = bm.fallback_count()
    dm, sm = bm.realize_acceleration_from(y0)
    d64, s64 = b64.realize_acceleration_from(y0)
    assert (sm == 0).all() and (s64 == 0).all()
    same(dm, d64)
    assert bm.fallback_count() - before >= touch.sum()
    # the pipelined form, where the batch has it, and the captured one
    for _ in range(2):
        same(bm.realize_acceleration_from(y0)[0], d64)
        bm.set_state(y0)
        same(bm.realize_acceleration()[0], d64)
    # steps: the bits of a batch of two (one to a block); the FP64 integration's
    # kernel is another one, which may round otherwise
    bm.set_state(y0)
    sm = bm.rk_merson_fixed(5e-4, 3)
    ym = bm.get_state()[0]
    b64.set_state(y0)
    b64.rk_merson_fixed(5e-4, 3)
    y64 = b64.get_state()[0]
    np.testing.assert_allclose(ym, y64, rtol=0, atol=1e-6 * np.abs(y64).max())
    for k in np.unique(which[touch]):
        b2 = Batch(topo, np.full(2, k, np.int32), precision="mixed")
        b2.set_state(np.tile(y[k], 2))
        s2 = b2.rk_merson_fixed(5e-4, 3)
        y2 = b2.get_state()[0][:len(y[k])]
        for i in np.nonzero(touch & (which == k))[0]:
            np.testing.assert_array_equal(ym[off[i]:off[i + 1]], y2)
            assert sm[i] == s2[0]


@pytest.mark.parametrize("n", [100, 4000])
def test_recomputing_every_instance_takes_about_an_fp64_realize(engine, trees, n):
    """Contact trees alone: the mixed realize recomputes all of them. One after
    another on few lanes they took 45 times the FP64 batch's realize; the bound
    leaves room for the mixed pass before it and for other load."""
    topo, y = trees
    which = (24 + np.arange(n) % 24).astype(np.int32)
    y0 = np.concatenate([y[k] for k in which])
    best = {}
    for p in ("mixed", "fp64"):
        b = Batch(topo, which, precision=p)
        b.set_state(y0)
        times = []
        for _ in range(6):
            t0 = time.perf_counter()
            b.realize_acceleration_async()
            b.sync()
            times.append(time.perf_counter() - t0)
        best[p] = min(times[2:])
    assert best["mixed"] <= 8 * best["fp64"], best
