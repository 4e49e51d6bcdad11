"""A pass of SWAPs only relabels the qubits: nothing is launched for it, unless it
makes its input from a recorded basis state or writes the probabilities of a
sampled state."""
import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200 import workloads as W
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.circuit import Device, StateVector

pytestmark = pytest.mark.gpu


def swaps(n):
    pairs = [(0, n - 1), (1, 2), (n - 2, 0)]
    return W.to_array([(L.SWAP, a, b, -1, 0, 0.0, 1.0, (0.0,) * 8) for a, b in pairs])


def execute(st, ops):
    L.check(L.lib.qse_execute(st.handle, L.dptr(ops), len(ops), None, 0, None, None, 0, None))


@pytest.mark.parametrize("jit", [1, 0])
@pytest.mark.parametrize("n", [4, 12, 20, 22])
def test_swaps_launch_nothing(n, jit):
    dev = Device(0)
    L.check(L.lib.qse_ctx_set_jit(dev.handle, jit))
    ops = W.random_circuit(n, 4 * n, 60 + n)
    st = StateVector(n, dev)
    execute(st, ops)
    before = dev.kernel_launches
    execute(st, swaps(n))
    assert dev.kernel_launches == before
    want = O.run(n, np.concatenate([ops, swaps(n)]))
    assert np.max(np.abs(st.download() - want)) <= 1e-12
    # gates after the relabelling, and from a recorded basis state
    more = W.random_circuit(n, 2 * n, 70 + n)
    execute(st, more)
    assert np.max(np.abs(st.download() - O.run_on(want, n, more))) <= 1e-12
    st.reset()
    execute(st, swaps(n))
    execute(st, more)
    assert np.max(np.abs(st.download() - O.run(n, np.concatenate([swaps(n), more])))) <= 1e-12


@pytest.mark.parametrize("n", [13, 22])
def test_sampled_state_is_relabelled(n):
    """Shots after swaps of a state that is sampled again and again."""
    dev = Device(0)
    ops = W.random_circuit(n, 4 * n, 80 + n)
    u = np.random.default_rng(n).random(500)
    st = StateVector(n, dev)
    execute(st, ops)
    want = O.run(n, ops)
    for _ in range(3):
        out = np.empty(u.size, dtype=np.uint64)
        L.check(L.lib.qse_sample(st.handle, u.ctypes.data_as(L._pd), u.size, 0, out.ctypes.data_as(L._pu64)))
        assert np.array_equal(out, O.sample(st.download(), n, u))
        execute(st, swaps(n))
        want = O.run_on(want, n, swaps(n))
        assert np.max(np.abs(st.download() - want)) <= 1e-12


@pytest.mark.parametrize("n", [6, 20])
def test_gradient_through_swaps(n):
    """SWAPs at both ends and between blocks of gates that fill passes of their own."""
    rows = []
    for block in range(3):
        rows += [(L.SWAP, a, b, -1, 1.0) for a, b in ((0, n - 1), (1, n - 2))]
        rows += [(L.RX, q, 0, block, 1.0) for q in range(n)] + [(L.CNOT, (q + 1) % n, q, -1, 1.0) for q in range(n)]
    rows += [(L.SWAP, 0, 2, -1, 1.0)]
    ops = np.zeros(len(rows), dtype=L.OP_DTYPE)
    for i, (t, a, b, p, c) in enumerate(rows):
        ops[i]["type"], ops[i]["target"], ops[i]["control"], ops[i]["param"], ops[i]["coeff"] = t, a, b, p, c
    params = np.array([0.3, -0.7, 1.1])
    z, w = [1, 3, 1 << (n - 1)], [1.0, 0.5, -0.25]
    v, g = ParametrizedCircuit(n, ops, z, w, 0.125, device=Device(0)).value_and_grad(params)
    obs, keep = L.observable(z, w, 0.125)
    vw, gw = O.adjoint(n, ops, params, obs)
    assert abs(v - vw) <= 1e-10
    assert np.max(np.abs(g - gw)) <= 1e-10
