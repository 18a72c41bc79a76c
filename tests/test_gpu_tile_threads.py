"""Batches on different host threads: handles are independent, so two batches
whose FP32 tiles take blocks of different sizes launch the same kernels side by
side."""
import threading

import numpy as np
import pytest

from simbody_gb300 import Batch, Topology, Workload

pytestmark = pytest.mark.gpu


def test_fp32_tiles_of_different_widths_on_two_threads(engine, monkeypatch):
    w = Workload(3, 8)
    topo = [Topology(w.systems[k], keepalive=w) for k in range(8)]
    which = np.arange(256, dtype=np.int32) % 8
    y = np.concatenate([w.y0[w.instance_slice(int(k))] for k in which])
    batches = []
    for warps in ("8", "1", "4", "2"):
        monkeypatch.setenv("SBG_TILE32", warps)
        b = Batch(topo, which, precision="mixed")
        b.set_state(y)
        b.rk_merson_fixed(5e-4, 1)
        assert b.kernel_variant == 9
        batches.append(b)
    out, errors = [None] * len(batches), []
    start = threading.Barrier(len(batches))

    def work(k):
        try:
            start.wait()
            for _ in range(20):
                batches[k].set_state(y)
                batches[k].rk_merson_fixed(1e-5, 48)  # a launch a step
            out[k] = batches[k].get_state()[0]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(batches))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for o in out[1:]:
        np.testing.assert_array_equal(o, out[0])
