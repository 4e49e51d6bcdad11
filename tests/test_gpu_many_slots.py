"""Batched circuits at the limits of a CTA (as many threads as the widest tile
uses), and reverse passes with many gradient slots: the interpreter keeps 8 or 1
partial sums per warp and slot, 8 where they fit in shared memory.  Values and
gradients against the FP64 oracle's adjoint (1e-10, as the other gradient
tests), at slot counts on both sides of the change, up to counts that only fit
with one partial per warp."""
import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.batch import Batch, BatchConfig
from quantumsimevo_b200.circuit import Device

pytestmark = pytest.mark.gpu
TOL = 1e-10


def circuit(n, gates, seed, phases):
    """`gates` parametrised gates with a slot each: rotations on every qubit in
    turn, or, with phases, a rotation layer every 500 phase gates and at the end."""
    ops = np.zeros(gates, dtype=L.OP_DTYPE)
    for i in range(gates):
        q = i % n
        rotation = not phases or i % 500 < n or i >= gates - n
        kind = (L.RX, L.RY)[(i // n) % 2] if rotation else (L.RZ, L.PHASE, L.CPHASE)[i % 3]
        ops[i]["type"], ops[i]["target"], ops[i]["param"], ops[i]["coeff"] = kind, q, i, 1.0
        if kind == L.CPHASE:
            ops[i]["control"] = (q + 1) % n
    params = np.random.default_rng(seed).uniform(-3, 3, gates)
    obs = ([1 << q for q in range(n)] + [3], list(np.linspace(-1, 1, n + 1)), 0.25)
    return ops, params, obs


def expected(n, ops, params, obs):
    o, keep = L.observable(*obs)
    return O.adjoint(n, ops, params, o)


# default shape (128 threads): 8 partials at 60 slots, 1 beyond some 200
@pytest.mark.parametrize("cfg", [None, BatchConfig(threads=32, reg_bits=2), BatchConfig(threads=512, reg_bits=3)])
@pytest.mark.parametrize("gates", [60, 300, 700, 1500])
def test_batched_circuits(cfg, gates):
    n = 6
    ops, params, obs = circuit(n, gates, gates, phases=False)
    b = Batch([(n, ops, len(params), obs)], Device(0))
    if cfg is not None:
        b.config = cfg
    v, g = b.run(params)
    vw, gw = expected(n, ops, params, obs)
    assert abs(v[0] - vw) <= TOL
    assert np.max(np.abs(g - gw)) <= TOL


# CTAs have no more threads than the widest tile: from the narrowest circuits, over
# each CTA size, up to the configured one
@pytest.mark.parametrize("cfg", [None, BatchConfig(threads=512, reg_bits=3), BatchConfig(threads=256, reg_bits=2)])
@pytest.mark.parametrize("widths", [(4,), (5, 6), (4, 8, 9), (6, 10), (11, 4), (12, 4)])
def test_batches_of_narrow_circuits(cfg, widths):
    circs, params, vw, gw = [], [], [], []
    for i, n in enumerate(widths):
        ops, p, obs = circuit(n, 12 * n, 7 * i + n, phases=False)
        circs.append((n, ops, len(p), obs))
        params.append(p)
        v, g = expected(n, ops, p, obs)
        vw.append(v)
        gw.append(g)
    b = Batch(circs, Device(0))
    if cfg is not None:
        b.config = cfg
    v, g = b.run(np.concatenate(params))
    assert np.max(np.abs(v - np.array(vw))) <= TOL
    assert np.max(np.abs(g - np.concatenate(gw))) <= TOL


@pytest.mark.parametrize("n,gates", [(5, 90), (10, 300), (11, 500), (12, 1000)])
def test_gradient_without_specialised_kernels(n, gates):
    ops, params, obs = circuit(n, gates, gates, phases=True)
    dev = Device(0)
    L.check(L.lib.qse_ctx_set_jit(dev.handle, 0))
    v, g = ParametrizedCircuit(n, ops, *obs, device=dev).value_and_grad(params)
    vw, gw = expected(n, ops, params, obs)
    assert abs(v - vw) <= TOL
    assert np.max(np.abs(g - gw)) <= TOL
