"""Several tiles in one block. Tiles of fewer than four warps share a block as
soon as there are more tiles than SMs, and nothing orders one against the
other. Every tile kernel, on two and on four tiles a block, gives each instance
the bits it has with one tile a block, and a sample agrees with the CPU
oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from simbody_gb300 import Batch, Topology, Workload, engine_batch
from simbody_gb300 import _native as Nat

pytestmark = pytest.mark.gpu

N = 32 * 330 + 5  # more tiles than any GPU's SMs twice over, the last one ragged


@pytest.fixture(scope="module")
def tree():
    w = Workload(3, 8)
    y = np.tile(w.y0[w.instance_slice(5)], N).reshape(N, -1)
    y *= np.random.default_rng(5).uniform(0.5, 6, size=(N, 1))  # instances that accept and reject differently
    return w, Topology(w.systems[5], keepalive=w), y


def _run(monkeypatch, tree, precision, warps, which, run):
    w, t, y = tree
    monkeypatch.setenv("SBG_TILE", f"32,{warps}")
    monkeypatch.setenv("SBG_TILE32", str(warps))
    b = Batch([t], np.zeros(len(which), np.int32), precision=precision)
    b.set_state(y[which].ravel())
    return run(b)


def _per_instance(b, a):
    return a.reshape(b.ninst, -1)


def _passes(b):
    """Every kind of pass over the batch, each output by instance."""
    out = {}
    d, st = b.realize_acceleration()
    out["realize"], out["realize status"] = _per_instance(b, d), st
    f = np.tile(np.linspace(-1, 1, b.nu[0]), b.ninst)
    out["minv"] = _per_instance(b, b.multiply_by_minv(f))
    out["mv"] = _per_instance(b, b.multiply_by_m(f)[0])
    out["steps status"] = b.rk_merson_fixed(5e-4, 3)
    out["steps"] = _per_instance(b, b.get_state()[0])
    return out


@pytest.mark.parametrize("warps", [1, 2])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_fast"])
def test_tiles_that_share_a_block(engine, monkeypatch, tree, precision, warps):
    many = _run(monkeypatch, tree, precision, warps, np.arange(N), _passes)
    # a batch with as many tiles as SMs at most gives each its own block
    which = np.r_[0:2048, N - 37:N]
    few = _run(monkeypatch, tree, precision, warps, which, _passes)
    for k, a in few.items():
        np.testing.assert_array_equal(many[k][which], a, err_msg=k)
    assert (many["realize status"] == 0).all()


@pytest.mark.parametrize("warps", [1, 2])
def test_error_controlled_tiles_that_share_a_block(engine, monkeypatch, tree, warps):
    w, t, y = tree

    def run(b):
        st, stats = b.rk_merson_adaptive(0.01, accuracy=1e-5)
        yo, to = b.get_state()
        return st, stats, _per_instance(b, yo), to

    st, stats, yo, to = _run(monkeypatch, tree, "fp64", warps, np.arange(N), run)
    which = np.r_[0:2048, N - 37:N]
    for a, b in zip((st, stats, yo, to), _run(monkeypatch, tree, "fp64", warps, which, run)):
        np.testing.assert_array_equal(a[which], b)
    assert (st == 0).all() and len(np.unique(stats, axis=0)) > 3 and stats[:, 1].sum() > 0
    sample = np.arange(0, N, 97)
    off = np.arange(len(sample) + 1) * y.shape[1]
    ry, _, rst, rstats = O.rk_merson_adaptive(w.systems, w.nsys, np.full(len(sample), 5), off, y[sample].ravel(), 0.01,
                                              accuracy=1e-5)
    np.testing.assert_array_equal(st[sample], rst)
    np.testing.assert_array_equal(stats[sample], rstats)
    ry = ry.reshape(len(sample), -1)
    # 1e-10: the tolerance of fixed and error-controlled steps against the oracle
    assert (np.linalg.norm(yo[sample] - ry, axis=1) <= 1e-10 * np.linalg.norm(ry, axis=1)).all()


@pytest.mark.parametrize("config", [3, 6, 7, 8])
def test_steps_do_not_depend_on_the_other_instances(engine, config):
    """The error norms and projection gates are sums over an instance's bodies
    in its own order: alone, among others and with other neighbours it takes
    the same steps to the last bit."""
    w = Workload(config, 96)

    def run(idx):
        b, y0 = engine_batch(w, "fp64", instances=idx)
        b.set_state(y0)
        _, stats = b.rk_merson_adaptive(0.03, accuracy=1e-4)
        ya, ta = b.get_state()
        b.set_state(y0)
        b.rk_merson_fixed(w.h, 3)
        yf, _ = b.get_state()
        cut = [slice(b.y_offsets[k], b.y_offsets[k + 1]) for k in range(len(idx))]
        return {i: (stats[k], ta[k], ya[cut[k]], yf[cut[k]]) for k, i in enumerate(idx)}

    among = run(list(range(96)))
    for idx in [[k] for k in (0, 7, 40, 95)] + [list(range(95, -1, -5))]:
        for i, got in run(idx).items():
            for a, b in zip(got, among[i]):
                np.testing.assert_array_equal(a, b)


def _pins(angle):
    """Four pins in a row whose frames are turned by +angle on the parent's side
    and back on the child's: the rotation between them is the identity up to
    rounding."""
    c, s = np.cos(angle), np.sin(angle)
    bodies = (Nat.BodyDesc * 4)()
    for k, b in enumerate(bodies):
        b.parent, b.mobilizer, b.mass = k, Nat.SBG_PIN, 1.0
        b.com[0], b.com[1] = 0.3, 0.1
        b.unit_inertia[0], b.unit_inertia[1], b.unit_inertia[2] = 0.2, 0.3, 0.4
        for X, sg in ((b.X_PF, -1), (b.X_BM, 1)):
            X[0] = X[4] = c
            X[1], X[3] = -sg * s, sg * s
            X[8] = 1.0
        b.X_PF[9] = 0.5
    d = Nat.SystemDesc(4, 0, 0, 0, (C.c_double * 3)(0, -9.8, 0), bodies, None, None)
    return Topology(d, keepalive=bodies)


def test_frames_that_cancel_up_to_rounding(engine):
    """A body whose inboard frame is aligned with its parent's mobilizer frame
    skips that rotation, unless a neighbour in the tile needs one: the bits are
    the same."""
    angles = np.linspace(0.01, 3.1, 60)
    topo = [_pins(a) for a in angles]
    y = np.linspace(-1, 1, 8 * len(topo)).reshape(len(topo), 8)
    among, st = Batch(topo, np.arange(len(topo), dtype=np.int32)).realize_acceleration_from(y.ravel())
    assert (st == 0).all()
    for k, t in enumerate(topo):
        alone, _ = Batch([t], np.zeros(1, np.int32)).realize_acceleration_from(y[k])
        np.testing.assert_array_equal(alone, among.reshape(-1, 8)[k])
