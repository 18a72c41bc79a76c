"""A call that runs out of the batch's device budget leaves the batch as it was:
nothing of it stays allocated, the state is untouched, the same call fails in
the same way again, and the batch goes on working."""
import numpy as np
import pytest

from simbody_gb300 import Batch, Topology, Workload
from simbody_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trees():
    w = Workload(3, 70)
    topo = [Topology(w.systems[k], keepalive=w) for k in range(w.nsys)]
    return w, topo


def _refused(b, call):
    before = b.device_bytes, b.get_state()
    for _ in range(3):
        with pytest.raises(N.EngineError) as e:
            call()
        assert e.value.code == 4  # SBG_ERR_BUDGET
        assert b.device_bytes == before[0]
    y, t = b.get_state()
    np.testing.assert_array_equal(y, before[1][0])
    np.testing.assert_array_equal(t, before[1][1])


@pytest.mark.parametrize("precision", ["mixed", "mixed_fast", "fp64"])
def test_refused_calls_leave_nothing_behind(engine, trees, precision):
    w, topo = trees
    free = Batch(topo, w.instance_system, precision=precision)
    need = free.device_bytes
    free.set_state(w.y0)
    f = np.ones(free.u_offsets[-1])
    want_mv = free.multiply_by_m(f)[0]
    with_ops = free.device_bytes
    # nothing to spare, and room for some tables but not for the operands (at least 16 doubles a body)
    for spare in (0, 64 * free.body_offsets[-1]):
        b = Batch(topo, w.instance_system, precision=precision, device_budget_bytes=need + spare)
        assert b.device_bytes == need
        b.set_state(w.y0)
        _refused(b, lambda: b.multiply_by_m(f))
        d, st = b.realize_acceleration()
        assert (st == 0).all() and np.isfinite(d).all()
    b = Batch(topo, w.instance_system, precision=precision, device_budget_bytes=with_ops)
    b.set_state(w.y0)
    np.testing.assert_array_equal(b.multiply_by_m(f)[0], want_mv)


def test_mixed_steps_are_refused_before_the_first(engine, trees):
    w, topo = trees
    free = Batch(topo, w.instance_system, precision="mixed")
    need = free.device_bytes
    free.set_state(w.y0)
    free.rk_merson_fixed(w.h, 2)
    want = free.get_state()[0]
    steps = free.device_bytes - need
    # nothing to spare, room for the first list, for tables but not for the stage planes (40 bytes a state element)
    for spare in (0, 8 * w.ninst, 20 * free.ny_total):
        b = Batch(topo, w.instance_system, precision="mixed", device_budget_bytes=need + spare)
        b.set_state(w.y0)
        b.realize_acceleration()
        y0 = b.get_state()[0]
        for _ in range(2):
            with pytest.raises(N.EngineError) as e:
                b.rk_merson_fixed(w.h, 2)
            assert e.value.code == 4 and b.device_bytes == need
        np.testing.assert_array_equal(b.get_state()[1], np.zeros(b.ninst))
        np.testing.assert_allclose(b.get_state()[0], y0, rtol=1e-15)  # quaternions may have been normalized
    b = Batch(topo, w.instance_system, precision="mixed", device_budget_bytes=need + steps)
    b.set_state(w.y0)
    b.rk_merson_fixed(w.h, 2)
    np.testing.assert_array_equal(b.get_state()[0], want)
