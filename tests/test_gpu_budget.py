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


# Device bytes that a batch took for itself, and with operators and (mixed) steps,
# when it kept one record per body, and nothing else, per instance. None: the
# tiles fit within that, the calls' buffers beside them do not.
RECORDS_ALONE = [
    ("fp64", 1, 1024, 1786848, 2089960), ("fp64", 2, 1, 1426216, 1431864), ("fp64", 3, 33, 2998508, 3155676),
    ("fp64", 3, 300, 17880684, 19312612), ("fp64", 4, 20, 2799288, 2914656), ("fp64", 6, 512, 32889480, 35461328),
    ("fp64", 7, 512, 29326764, 31761844), ("fp64", 8, 512, 33076676, 35502908), ("fp64", 5, 100, 23415872, 24414920),
    ("mixed", 1, 1024, 2417640, None), ("mixed", 2, 1, 1815344, 2081920), ("mixed", 3, 33, 3829492, None),
    ("mixed", 3, 300, 22026356, 39026300), ("mixed", 3, 700, None, None), ("mixed", 4, 20, 3688596, None),
    ("mixed", 7, 512, 35979060, 64773884), ("mixed", 8, 512, 39707596, 68425276), ("mixed", 5, 100, 28508864, 39381344),
    ("mixed_fast", 3, 33, 1903340, 3986652), ("mixed_fast", 3, 300, 12269676, 23458276),
    ("mixed_fast", 7, 512, 20286508, 38414132),
]


@pytest.mark.parametrize("precision,config,n,alone,with_calls", RECORDS_ALONE)
def test_a_small_budget_costs_time_not_the_batch(engine, precision, config, n, alone, with_calls):
    """Where the tiles do not fit, the batch takes its instances one at a time on
    shared tables and gives the same bits. In the mixed form an instance that
    needs FP64 may come to another kernel than with room: the FP64 parity
    tolerances (1e-12, after steps 1e-10) hold there."""
    w = Workload(config, n)
    topo = [Topology(w.systems[k], keepalive=w) for k in range(w.nsys)]
    def run(budget, calls):
        b = Batch(topo, w.instance_system, precision=precision, device_budget_bytes=budget)
        f, out = np.linspace(-1, 1, b.u_offsets[-1]), {}
        b.set_state(w.y0)
        out["realize"], out["status"] = b.realize_acceleration()
        out["again"] = b.realize_acceleration_from(w.y0)[0]
        out["minv"] = b.multiply_by_minv(f)
        if calls:
            out["mv"] = b.multiply_by_m(f)[0]
            out["jtf"] = b.multiply_by_system_jacobian_transpose(np.linspace(-1, 1, 6 * b.body_offsets[-1]))[0]
            out["step status"] = b.rk_merson_fixed(w.h or 1e-3, 3)
            out["steps"] = b.get_state()[0]
            if precision == "fp64" and not any(w.systems[k].nconstraints for k in range(w.nsys)):
                b.set_state(w.y0)
                _, out["stats"] = b.rk_merson_adaptive(0.01, accuracy=1e-4)
                out["adaptive"] = b.get_state()[0]
        assert not budget or b.device_bytes <= budget
        return out, b.device_bytes

    want, _ = run(0, True)
    b = Batch(topo, w.instance_system, precision=precision)
    budgets = [(alone or int(0.75 * b.device_bytes), False)] + ([(with_calls, True)] if with_calls else [])
    del b
    for budget, calls in budgets:
        got, _ = run(budget, calls)
        for k, a in got.items():
            if precision == "mixed" and a.dtype == np.float64:
                tol = 1e-10 if k == "steps" else 1e-12
                np.testing.assert_allclose(a, want[k], rtol=0, atol=tol * np.abs(want[k]).max(), err_msg=k)
            else:
                np.testing.assert_array_equal(a, want[k], err_msg=f"{k} within {budget} bytes")


def test_a_mixed_batch_keeps_its_fp32_tiles_without_wide_fp64_ones(engine):
    """Of a mixed batch the wide FP64 tiles go first: with room for all but
    those, realize and steps stay on the FP32 tiles, operators work, and the
    results agree with those of a batch with room (FP64 work: parity tolerances)."""
    w = Workload(3, 700)
    topo = [Topology(w.systems[k], keepalive=w) for k in range(w.nsys)]
    fast = Batch(topo, w.instance_system, precision="mixed_fast")
    fast.set_state(w.y0)
    wide = -fast.device_bytes
    fast.multiply_by_m(np.ones(fast.u_offsets[-1]))
    wide += fast.device_bytes  # the wide FP64 tiles and the operators' operands
    need = Batch(topo, w.instance_system, precision="mixed").device_bytes
    out = []
    for budget in (0, need, need - wide // 2):
        b = Batch(topo, w.instance_system, precision="mixed", device_budget_bytes=budget)
        b.set_state(w.y0)
        d, st = b.realize_acceleration()
        assert b.kernel_variant == 9 and (st == 0).all()
        mv = b.multiply_by_m(np.ones(b.u_offsets[-1]))[0]
        b.rk_merson_fixed(w.h, 2)
        out.append((d, mv, b.get_state()[0]))
        assert not budget or b.device_bytes <= budget
    for o in out[1:]:
        for a, c, tol in zip(o, out[0], (1e-12, 0, 1e-10)):
            np.testing.assert_allclose(a, c, rtol=0, atol=tol * np.abs(c).max())
