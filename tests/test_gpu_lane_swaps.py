"""Passes that read or write memory with the lowest qubits in registers swap them
with lane bits by shuffles on the memory side (jit.cpp to_memory_layout, laneSwap),
on states of 20 qubits and more.  Circuits that do so where they read, where they
write, at both ends and at neither, on one and on two states, in tiles from 16
threads (too few: no swaps) up, against the oracle.  QSE_JIT_DUMP's sources tell
that the swaps are where the case says."""
import re

import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.circuit import Device, StateVector

pytestmark = pytest.mark.gpu
LOW, HIGH = (0, 1, 2), (3, 4, 5, 6)   # all in the tile of a single pass


def circuit(where, params=False):
    """Rotations on HIGH, with rotations on LOW ahead of them, after them or both
    (CNOTs in between keep the order)."""
    rows = []

    def rot(qubits):
        for q in qubits:
            for t in (L.RX, L.RY):
                rows.append((t, q, 0))

    def link(a, b):
        rows.extend((L.CNOT, t, a[i % len(a)]) for i, t in enumerate(b))

    if where in ("load", "both"):
        rot(LOW)
        link(LOW, HIGH)
    rot(HIGH)
    if where in ("store", "both"):
        link(HIGH, LOW)
        rot(LOW)
    ops = np.zeros(len(rows), dtype=L.OP_DTYPE)
    ops["type"], ops["target"], ops["control"] = np.array(rows).T
    rotation = (ops["type"] == L.RX) | (ops["type"] == L.RY)
    ops["param"], ops["coeff"] = -1, 1.0
    angles = np.random.default_rng(len(rows)).uniform(-3, 3, int(rotation.sum()))
    if params:
        ops["param"][rotation] = np.arange(rotation.sum())
    else:
        ops["theta"][rotation] = angles
    return ops, angles


def swaps(text):
    """Lane swaps ahead of a kernel's first gate and after its last."""
    body = text.split('extern "C"')[1]
    gates = [m.start() for m in re.finditer(r"op(H|X|Y|RX|RY)[cs]?<|xb\[s", body)]
    at = [m.start() for m in re.finditer(r"laneSwap<", body)]
    return sum(p < gates[0] for p in at), sum(p > gates[-1] for p in at)


def expect(where, threads, states, got):
    """Two or three of LOW's qubits move at the end that the case names (per state);
    one may be left in the registers at the other end, where there are rotations."""
    for end, n in zip(("load", "store"), got):
        if threads < 32 or where == "neither":
            assert n == 0
        elif where in (end, "both"):
            assert n in (2 * states, 3 * states)
        else:
            assert n <= states


@pytest.mark.parametrize("where", ["load", "store", "both", "neither"])
@pytest.mark.parametrize("n,k", [(20, 8), (20, 9), (20, 10), (20, 12), (21, 11), (22, 12), (23, 12)])
def test_one_state(n, k, where, tmp_path, monkeypatch):
    monkeypatch.setenv("QSE_JIT_DUMP", str(tmp_path))
    dev = Device(0)
    dev.set_fusion(True, k, 0, exact_tiles=True)
    ops, _ = circuit(where)
    rng = np.random.default_rng(n * k)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    st = StateVector(n, dev)
    st.upload(psi)
    L.check(L.lib.qse_execute(st.handle, L.dptr(ops), len(ops), None, 0, None, None, 0, None))
    assert np.max(np.abs(st.download() - O.run_on(psi, n, ops))) <= 1e-12
    (source,) = tmp_path.iterdir()
    expect(where, 1 << (k - 4), 1, swaps(source.read_text()))


@pytest.mark.parametrize("where", ["load", "store", "both", "neither"])
@pytest.mark.parametrize("n", [20, 22, 23])
def test_two_states(n, where, tmp_path, monkeypatch):
    """The reverse sweep undoes the circuit from its end, on |psi> and |lambda>."""
    monkeypatch.setenv("QSE_JIT_DUMP", str(tmp_path))
    ops, params = circuit(where, params=True)
    z, w = [1, 2, 4 | 8, 1 << 6, 1 << (n - 1)], [0.5, -1.0, 0.25, 1.0, 0.75]
    v, g = ParametrizedCircuit(n, ops, z, w, 0.125, device=Device(0)).value_and_grad(params)
    obs, keep = L.observable(z, w, 0.125)
    vw, gw = O.adjoint(n, ops, params, obs)
    assert abs(v - vw) <= 1e-10
    assert np.max(np.abs(g - gw)) <= 1e-10
    (reverse,) = [f for f in tmp_path.iterdir() if f.name.startswith("qse_pass_adjoint")]
    expect({"load": "store", "store": "load"}.get(where, where), 256 if n < 22 else 128, 2, swaps(reverse.read_text()))
