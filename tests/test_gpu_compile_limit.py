"""A deep circuit on a small state runs on the interpreter instead of waiting for
the compiler (engine.cu plan_for): more than 32 new kernels, counted in 12-qubit
tiles, whose plans small states otherwise take apart into more and shorter ones.
QSE_JIT_DUMP gets one file per kernel compiled, so the number of files tells the
two apart; the results are the oracle's either way."""

import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200 import workloads as W
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.circuit import Device, StateVector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gates,interpreted", [
    (16, 4000, True),    # 45 passes in 12-qubit tiles, 54 in the state's 11-qubit ones
    (14, 6000, True),    # 57 and 72
    (20, 3000, True),    # 43 and 62
    (14, 2400, False),   # fewer than 32 either way
    (12, 6000, False),   # 13 passes in one 12-qubit tile, 47 in 11-qubit ones
])
def test_deep_circuits(n, gates, interpreted, tmp_path, monkeypatch):
    monkeypatch.setenv("QSE_JIT_DUMP", str(tmp_path))
    ops = W.random_circuit(n, gates, 900 + n)
    st = StateVector(n, Device(0))
    L.check(L.lib.qse_execute(st.handle, L.dptr(ops), len(ops), None, 0, None, None, 0, None))
    compiled = len(list(tmp_path.iterdir()))
    assert compiled == 0 if interpreted else compiled > 0
    # 1e-12 for some hundred gates elsewhere; roundings add up at most linearly
    assert np.max(np.abs(st.download() - O.run(n, ops))) <= 1e-11


def test_deep_gradient_of_one_tile(tmp_path, monkeypatch):
    """40 reverse passes of at most 256 gates: interpreted as in a state of more
    qubits (its tile has no larger one to be counted in)."""
    monkeypatch.setenv("QSE_JIT_DUMP", str(tmp_path))
    n, gates, npar = 6, 256 * 40, 8
    rng = np.random.default_rng(1)
    ops = np.zeros(gates, dtype=L.OP_DTYPE)
    ops["type"] = rng.choice([L.RX, L.RY, L.H], gates)
    ops["target"] = rng.integers(0, n, gates)
    ops["param"] = np.where(ops["type"] == L.H, -1, rng.integers(0, npar, gates))
    ops["coeff"] = 1.0
    params = rng.uniform(-3, 3, npar)
    z, w = [1 << q for q in range(n)], list(np.linspace(-1, 1, n))
    dev = Device(0)
    L.check(L.lib.qse_ctx_set_jit(dev.handle, 0))
    v0, g0 = ParametrizedCircuit(n, ops, z, w, 0.25, device=dev).value_and_grad(params)
    L.check(L.lib.qse_ctx_set_jit(dev.handle, 1))
    v, g = ParametrizedCircuit(n, ops, z, w, 0.25, device=dev).value_and_grad(params)
    assert len(list(tmp_path.iterdir())) == 0
    obs, keep = L.observable(z, w, 0.25)
    vw, gw = O.adjoint(n, ops, params, obs)
    # 10240 gates, some 850 occurrences a parameter: 1e-10 for a hundred of them elsewhere
    for value, grad in ((v0, g0), (v, g)):
        assert abs(value - vw) <= 1e-10
        assert np.max(np.abs(grad - gw)) <= 1e-9
