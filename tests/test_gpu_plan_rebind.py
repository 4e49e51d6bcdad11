"""Plans reused with other numbers: the same gates with new angles and 2x2
matrices give, bit for bit, what a new context (nothing cached) gives: forward
executes on small states (specialised kernels and the interpreter), through the
compact prefix, with angles that make constants exactly 1, and gradients."""
import numpy as np
import pytest

from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200 import workloads as W
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.circuit import Device, StateVector

pytestmark = pytest.mark.gpu


def _state(n, dev, ops):
    st = StateVector(n, dev)
    L.check(L.lib.qse_execute(st.handle, L.dptr(ops), len(ops), None, 0, None, None, 0, None))
    return st.download()


def _variants(ops, seed):
    """ops, then the same gates with other angles and matrices, then all angles 0, then pi."""
    rng = W.SplitMix64(seed)
    yield ops
    for kind in range(3):
        v = ops.copy()
        for i in range(len(v)):
            if v[i]["theta"] != 0.0:
                v[i]["theta"] = (rng.uniform() * 7.0 - 3.5, 0.0, np.pi)[kind]
            if v[i]["type"] == L.GATE2X2:
                v[i]["m"] = W.gate2x2_unitary(rng)
        yield v


@pytest.mark.parametrize("n,jit", [(3, 1), (4, 1), (9, 1), (13, 1), (13, 0), (16, 1), (24, 1)])
def test_new_numbers_match_a_new_context(n, jit):
    # the compact prefix (24 qubits) starts with gates on few qubits
    ops = W.random_circuit(n, 25 * n, 40 + n) if n < 24 else np.concatenate(
        [W.random_circuit(10, 100, 1), W.random_circuit(20, 150, 2), W.random_circuit(24, 80, 3)])
    dev = Device(0)
    L.check(L.lib.qse_ctx_set_jit(dev.handle, jit))
    for v in list(_variants(ops, n)) + [ops]:
        cold = Device(0)
        L.check(L.lib.qse_ctx_set_jit(cold.handle, jit))
        assert np.array_equal(_state(n, dev, v), _state(n, cold, v))
        del cold


@pytest.mark.parametrize("n", [3, 8, 14, 22])
def test_new_parameters_gradient_matches_a_new_context(n):
    rng = np.random.default_rng(n)
    circuits = [W.hea_batch(1, n, n, 3, 3, seed=n)[0]]
    if n >= 4 and n % 2 == 0:
        ops, p, _, obs = W.qaoa_maxcut(n, 2, seed=n)
        circuits.append((n, ops, p, obs))
    for _, ops, p, obs in circuits:
        warm = ParametrizedCircuit(n, ops, *obs, device=Device(0))
        for params in (p, p + 0.25, np.zeros_like(p), np.full_like(p, np.pi), rng.uniform(-4, 4, p.size), p):
            v, g = warm.value_and_grad(params)
            cv, cg = ParametrizedCircuit(n, ops, *obs, device=Device(0)).value_and_grad(params)
            assert v == cv and np.array_equal(g, cg)
