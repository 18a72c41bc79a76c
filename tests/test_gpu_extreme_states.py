"""States that are not finite, and quaternions whose square overflows or
vanishes: the FP64 tile driver reports the instances that the CPU oracle
reports, whatever the coordinate, also those that the accelerations do not
depend on (a position on Ground). Operators too."""
import numpy as np
import pytest

from oracle import oracle as O
from simbody_gb300 import Workload, engine_batch
from simbody_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _check(w, y):
    ref, rst = O.realize(w.systems, w.nsys, w.instance_system, w.y_offsets, y)
    b, _ = engine_batch(w, "fp64")
    d, st = b.realize_acceleration_from(y)
    bad = np.array([not np.isfinite(ref[w.instance_slice(i)]).all() for i in range(w.ninst)])
    np.testing.assert_array_equal((st & N.INST_NONFINITE) != 0, bad)
    for i in np.nonzero(~bad)[0]:
        s = w.instance_slice(int(i))
        assert np.linalg.norm(d[s] - ref[s]) <= 1e-12 * np.linalg.norm(ref[s])
    return b, bad


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("config", [3, 6, 7])
def test_one_coordinate_not_finite(engine, config, value):
    w = Workload(config, 300)
    y = w.y0.copy()
    for i in range(w.ninst):  # the first coordinates (the root's), then all over
        s = w.instance_slice(i)
        y[s.start + (i % 13 if i < 150 else (7 * i) % (s.stop - s.start))] = value
    b, bad = _check(w, y)
    assert bad.mean() > 0.8
    f = np.ones(b.u_offsets[-1])
    _, st = b.multiply_by_system_jacobian(f)
    ref = O.tree_op(w.systems, w.nsys, w.instance_system, w.y_offsets, y, b.u_offsets, b.body_offsets, "jv", x=f)
    lost = np.array([not np.isfinite(ref[6 * b.body_offsets[i]:6 * b.body_offsets[i + 1]]).all() for i in range(w.ninst)])
    np.testing.assert_array_equal((st & N.INST_NONFINITE) != 0, lost)


@pytest.mark.parametrize("config", [3, 6])
def test_quaternions_out_of_range(engine, config):
    w = Workload(config, 60)
    y = w.y0.copy()
    scales = [1e100, 1e155, 1e300, 0.0, 1e-150, 1e-170]
    root_quat = np.array([w.systems[int(k)].bodies[0].mobilizer == N.SBG_FREE for k in w.instance_system])
    for i in np.nonzero(root_quat)[0]:
        y[w.instance_slice(int(i)).start:][:4] *= scales[i % len(scales)]
    _, bad = _check(w, y)
    assert bad.sum() > 0
