"""The FP64 tile driver at the edges of its tiles: one instance, one lane short
of a warp, one over, several tiles of shared and of distinct topologies, and
every mobilizer. Against the CPU oracle at the FP64 parity tolerances (1e-12
for a realize and M^-1 f, 1e-10 after fixed steps). An instance's results do
not depend on the tile it is in."""
import numpy as np
import pytest

from oracle import oracle as O
from simbody_gb300 import Batch, Topology, Workload, engine_batch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("n", [1, 31, 33, 70])
@pytest.mark.parametrize("config", [3, 4, 6, 7, 8])
def test_distinct_topologies(engine, config, n):
    w = Workload(config, n)
    b, y0 = engine_batch(w, "fp64")
    b.set_state(y0)
    ydot, st = b.realize_acceleration()
    ref, _ = O.realize_workload(w)
    assert (st == 0).all() and _rel(ydot, ref) <= 1e-12
    f = np.random.default_rng(config).normal(size=b.u_offsets[-1])
    m = O.multiply_by_minv(w.systems, w.nsys, w.instance_system, w.y_offsets, y0, b.u_offsets, f)
    assert _rel(b.multiply_by_minv(f), m) <= 1e-12
    b.rk_merson_fixed(w.h, 3)
    yr, _, _, _ = O.rk_workload(w, w.h, 3)
    assert _rel(b.get_state()[0], yr) <= 1e-10


@pytest.mark.parametrize("n", [1, 32, 129])
def test_shared_topology_in_any_tile(engine, n):
    w = Workload(3, 8)
    topo = [Topology(w.systems[k], keepalive=w) for k in (2, 5)]
    own = [w.y0[w.instance_slice(k)] for k in (2, 5)]
    alone = []
    for t, y in zip(topo, own):
        b = Batch([t], np.zeros(1, np.int32))
        alone.append(b.realize_acceleration_from(y)[0])
    # one topology throughout, and the two mixed in one batch
    b = Batch(topo[:1], np.zeros(n, np.int32))
    got, st = b.realize_acceleration_from(np.tile(own[0], n))
    assert (st == 0).all() and np.array_equal(got, np.tile(alone[0], n))
    which = (np.arange(n) % 3 == 1).astype(np.int32)
    b = Batch(topo, which)
    got, st = b.realize_acceleration_from(np.concatenate([own[k] for k in which]))
    assert (st == 0).all() and np.array_equal(got, np.concatenate([alone[k] for k in which]))


def _with_variant(monkeypatch, w, precision, variant, run):
    monkeypatch.setenv("SBG_VARIANT", str(variant))
    b, y0 = engine_batch(w, precision)
    b.set_state(y0)
    out = run(b)
    assert b.kernel_variant == variant
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 70])
@pytest.mark.parametrize("precision", ["mixed", "mixed_fast"])
def test_fp32_tiles_match_the_one_thread_driver_bitwise(engine, monkeypatch, precision, n):
    for config in (3, 4, 6, 8):
        w = Workload(config, n)

        def run(b):
            d, st = b.realize_acceleration()
            sr = b.rk_merson_fixed(w.h, 3)
            y, t = b.get_state()
            return d, st, sr, y, t

        for a, c in zip(_with_variant(monkeypatch, w, precision, 7, run), _with_variant(monkeypatch, w, precision, 9, run)):
            np.testing.assert_array_equal(a, c)


def test_no_budget_for_the_operators_tiles_is_an_error_each_time(engine):
    # a mixed batch builds the FP64 tiles at its first tree operator; the budget is what the batch itself takes
    w = Workload(3, 33)
    topo = [Topology(w.systems[k], keepalive=w) for k in range(w.nsys)]
    need = Batch(topo, w.instance_system, precision="mixed").device_bytes
    b = Batch(topo, w.instance_system, precision="mixed", device_budget_bytes=need)
    b.set_state(w.y0)
    ydot, st = b.realize_acceleration()
    for _ in range(2):
        with pytest.raises(RuntimeError, match="budget"):
            b.multiply_by_m(np.ones(b.u_offsets[-1]))
    again, st2 = b.realize_acceleration()
    assert (st == 0).all() and np.array_equal(ydot, again) and np.array_equal(st, st2)
