"""The host side of the C ABI over a stand-in for the CUDA runtime
(fake_cuda_runtime.cpp), on the CPU: any runtime call or launch fails in turn,
with pageable host memory copied in place and by way of the staging buffer.

  - A call that returns an error has no copy from or to the caller's memory
    under way, and the same call succeeds afterwards.
  - Batches without instances, or whose bodies have no coordinates, take the
    calls that copy states in both modes.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from simbody_gb300 import _native as N
from simbody_gb300 import build as B

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake") / "libhost.so"
    include = Path(B._nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{include}", "-o", str(out),
                    str(B.CSRC / "capi.cpp"), str(HERE / "fake_cuda_runtime.cpp"), "-lpthread"], check=True,
                   capture_output=True)
    lib = C.CDLL(str(out))
    for name, (res, args) in N.ENGINE_API.items():
        if hasattr(lib, name):
            fn = getattr(lib, name)
            fn.restype, fn.argtypes = res, args
    lib.fake_fail_at.restype = lib.fake_calls.restype = C.c_long
    lib.fake_fail_at.argtypes = [C.c_long]
    yield lib
    lib.fake_pageable(1)
    lib.fake_fail_at(0)


def _topology(lib, mobilizers):
    n = len(mobilizers)
    bodies = (N.BodyDesc * n)()
    for k, b in enumerate(bodies):
        b.parent, b.mobilizer, b.mass = k, mobilizers[k], 1.0
        b.unit_inertia[0] = b.unit_inertia[1] = b.unit_inertia[2] = 1.0
        for j in (0, 4, 8):
            b.X_PF[j] = b.X_BM[j] = 1.0
        b.X_PF[10] = 1.0
    d = N.SystemDesc(n, 0, 0, 0, (C.c_double * 3)(0, -9.8, 0), bodies, None, None)
    t = C.c_void_p()
    assert lib.sbg_topology_create(C.byref(d), C.byref(t)) == 0
    return t


def _batch(lib, topo, n, precision):
    b = C.c_void_p()
    cfg = N.BatchConfig(precision, 0, 0)
    which = np.zeros(n, np.int32)
    rc = lib.sbg_batch_create((C.c_void_p * 1)(topo), 1, which.ctypes.data_as(C.POINTER(C.c_int32)), n, C.byref(cfg),
                              C.byref(b))
    assert rc == 0, lib.sbg_last_error()
    return b


def _d(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _i(a):
    return a.ctypes.data_as(C.POINTER(C.c_int32))


def _calls(lib, b, n, nq, nu, nb):
    """name -> call over the caller's arrays, which outlive it."""
    y, u, body, st, t = (np.ones(n * (nq + nu)), np.ones(n * nu), np.ones(6 * n * nb), np.zeros(n, np.int32), np.zeros(n))
    o, ou, oq, ob = np.zeros_like(y), np.zeros_like(u), np.zeros(n * nq), np.zeros(10 * n * nb)
    return {
        "set_state": lambda: lib.sbg_batch_set_state(b, _d(t), _d(y)),
        "get_state": lambda: lib.sbg_batch_get_state(b, _d(t), _d(o)),
        "realize": lambda: lib.sbg_realize_acceleration(b, _d(o), _i(st)),
        "get_ydot": lambda: lib.sbg_batch_get_ydot(b, _d(o), _i(st)),
        "realize from host": lambda: lib.sbg_realize_acceleration_host(b, _d(y), _d(o), _i(st)),
        "qdotdot": lambda: lib.sbg_batch_get_qdotdot(b, _d(oq)),
        "minv": lambda: lib.sbg_multiply_by_minv(b, _d(u), _d(ou)),
        "m": lambda: lib.sbg_multiply_by_m(b, _d(u), _d(ou), _i(st)),
        "residual": lambda: lib.sbg_calc_residual_force(b, _d(u), _d(body), _d(u), _d(ou), _i(st)),
        "steps": lambda: lib.sbg_rk_merson_fixed(b, 1e-3, 2, None, _i(st)),
        "step to": lambda: lib.sbg_rk_merson_step_to(b, 1e-3, 2e-3, None, _i(st)),
        "composite": lambda: lib.sbg_calc_composite_body_inertias(b, _d(ob), _i(st)),
    }


@pytest.mark.parametrize("pageable", [1, 0])
@pytest.mark.parametrize("precision,n", [(N.PRECISION_FP64, 3), (N.PRECISION_MIXED, 200), (N.PRECISION_FP64, 1500)])
def test_no_copy_is_under_way_after_an_error(host, precision, n, pageable):
    host.fake_pageable(pageable)
    topo = _topology(host, [N.SBG_PIN, N.SBG_BALL, N.SBG_SLIDER])
    nq, nu, nb = 6, 5, 3
    b = _batch(host, topo, n, precision)
    calls = _calls(host, b, n, nq, nu, nb)
    for name in ("set_state", "realize from host", "realize", "qdotdot"):  # plans and buffers of the first calls
        assert calls[name]() == 0
    failed = 0
    for name, call in calls.items():
        if name == "qdotdot":
            assert calls["realize"]() == 0
        for k in range(1, 400):
            host.fake_fail_at(k)
            rc = call()
            reached = host.fake_calls() >= k
            under_way = host.fake_copies_under_way()
            host.fake_fail_at(0)
            if not reached:
                assert rc == 0, (name, host.sbg_last_error())
                break
            assert under_way == 0, (name, k, host.sbg_last_error())
            failed += rc != 0
            if name == "qdotdot":
                assert calls["realize"]() == 0
            assert call() == 0, (name, k, host.sbg_last_error())
        else:
            pytest.fail(f"{name}: more runtime calls than expected")
    assert failed > 20
    host.sbg_batch_destroy(b)
    host.sbg_topology_destroy(topo)
    host.fake_pageable(1)


@pytest.mark.parametrize("pageable", [1, 0])
@pytest.mark.parametrize("precision", [N.PRECISION_FP64, N.PRECISION_MIXED, N.PRECISION_MIXED_FAST])
@pytest.mark.parametrize("n,mobilizers", [(0, [N.SBG_PIN]), (3, [N.SBG_WELD, N.SBG_WELD])])
def test_batches_without_coordinates(host, precision, pageable, n, mobilizers):
    host.fake_pageable(pageable)
    topo = _topology(host, mobilizers)
    b = _batch(host, topo, n, precision)
    nu = 0 if n else 1
    for name, call in _calls(host, b, n, nu, nu, len(mobilizers)).items():
        assert call() == 0, (name, host.sbg_last_error())
    host.sbg_batch_destroy(b)
    host.sbg_topology_destroy(topo)
    host.fake_pageable(1)
