"""Tiles of exactly the size asked for (Device.set_fusion(exact_tiles=True)): with the
default, 12, states of at most 20 qubits run smaller ones.  The pass count tells
which tiles ran: it is the planner's for that tile size."""
import ctypes as C
import json

import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200 import workloads as W
from quantumsimevo_b200.circuit import Device, StateVector

pytestmark = pytest.mark.gpu
TOL = 1e-12


def planned_passes(n, ops, k, cap):
    need = C.c_size_t()
    args = (n, L.dptr(ops), len(ops), None, 0, k, cap)
    L.check(L.lib.qse_plan_describe(*args, None, 0, C.byref(need)))
    buf = C.create_string_buffer(need.value)
    L.check(L.lib.qse_plan_describe(*args, buf, need.value, C.byref(need)))
    return len(json.loads(buf.value)["passes"])


def execute(dev, n, ops):
    st = StateVector(n, dev)
    stats = L.QseExecStats()
    L.check(L.lib.qse_execute(st.handle, L.dptr(ops), len(ops), None, 0, None, None, 0, C.byref(stats)))
    return st.download(), stats.passes


@pytest.mark.parametrize("n,cap", [(12, 0), (13, 0), (14, 0), (18, 0), (20, 0), (21, 0), (15, 1)])
def test_twelve_qubit_tiles(n, cap):
    dev = Device(0)
    ops = W.random_circuit(n, 25 * n if cap == 0 else 90, 3100 + n)
    want = O.run(n, ops)
    dev.set_fusion(True, 12, cap, exact_tiles=True)
    got, passes = execute(dev, n, ops)
    assert np.max(np.abs(got - want)) <= TOL
    assert passes == planned_passes(n, ops, 12, cap or 256)
    dev.set_fusion(True, 12, cap)   # back to the engine's choice
    got, passes = execute(dev, n, ops)
    assert np.max(np.abs(got - want)) <= TOL
    assert passes == planned_passes(n, ops, 11 if n <= 18 else 10 if n <= 20 else 12, cap or 256)
