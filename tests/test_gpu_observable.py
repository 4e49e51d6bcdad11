"""<O> of sums of Z-strings whose masks cover every split of the kernel's index
bits (thread bits, register bits, chunk bits), at sizes around its 4096-amplitude
chunk, against a plain double-precision sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 11, 12, 13, 15, 20])
@pytest.mark.parametrize("nterms", [0, 1, 40])
def test_expectation_matches_plain_sum(n, nterms):
    from quantumsimevo_b200.circuit import Circuit

    rng = np.random.default_rng(1000 * n + nterms)
    c = Circuit(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    c.state.upload(psi)
    z = rng.integers(0, 1 << n, nterms, dtype=np.uint64)
    w = rng.standard_normal(nterms)
    i = np.arange(1 << n, dtype=np.uint64)
    o = np.full(1 << n, 0.25)
    for m, x in zip(z, w):
        par = np.zeros(1 << n, dtype=np.uint64)
        for b in range(n):
            if (int(m) >> b) & 1:
                par ^= (i >> np.uint64(b)) & np.uint64(1)
        o += x * (1.0 - 2.0 * par.astype(np.float64))
    want = float(np.sum(o * (psi.real ** 2 + psi.imag ** 2)))
    # |O| <= 0.25 + sum |w|: a few hundred roundings of 2^-53 of that, with the norm 1
    assert abs(c.expectation(z, w, 0.25) - want) <= 1e-13 * (0.25 + float(np.abs(w).sum()))


def _plain(psi, z, w, c):
    """sum_x (c + sum_t w_t (-1)^popcount(x & z_t)) |psi_x|^2 in doubles."""
    i = np.arange(psi.size, dtype=np.uint64)
    o = np.full(psi.size, c)
    for m, x in zip(z, w):
        o += np.where(np.bitwise_count(i & m) & 1, -x, x)
    return float(np.sum(o * (psi.real ** 2 + psi.imag ** 2)))


# the terms sit in shared memory, 16 B each: a launch gets 48 KiB unasked, some of it
# taken by the kernel's static arrays
@pytest.mark.parametrize("nterms", [3007, 3008, 3009, 3068, 3069, 3072, 3073, 4096])
def test_as_many_terms_as_are_accepted(nterms):
    from quantumsimevo_b200.circuit import Circuit

    n = 13
    rng = np.random.default_rng(nterms)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    c = Circuit(n)
    c.state.upload(psi)
    z = rng.integers(0, 1 << n, nterms, dtype=np.uint64)
    w = rng.standard_normal(nterms)
    # up to 4096 terms added one by one: as many roundings of 2^-53 of sum |w|, with the norm 1
    assert abs(c.expectation(z, w, 0.25) - _plain(psi, z, w, 0.25)) <= 1e-12 * (0.25 + float(np.abs(w).sum()))


def test_too_many_terms_is_a_size_error():
    from quantumsimevo_b200 import _lib as L
    from quantumsimevo_b200.circuit import Circuit

    c = Circuit(5)
    with pytest.raises(L.QseError) as e:
        c.expectation(np.ones(4097, dtype=np.uint64), np.ones(4097), 0.0)
    assert e.value.status == 5   # QSE_ERR_SIZE
    assert abs(c.expectation([1], [1.0], 0.0) - 1.0) <= 1e-15


def test_gradient_with_as_many_terms_as_are_accepted():
    import oracle_ffi as O
    from quantumsimevo_b200 import _lib as L
    from quantumsimevo_b200 import workloads as W
    from quantumsimevo_b200.autograd import ParametrizedCircuit

    n = 10
    ops, params, _, _ = W.qaoa_maxcut(n, 2, seed=5)
    rng = np.random.default_rng(6)
    z = [int(x) for x in rng.integers(1, 1 << n, 4096)]
    w = [float(x) / 64.0 for x in rng.standard_normal(4096)]
    v, g = ParametrizedCircuit(n, ops, z, w, 0.5).value_and_grad(params)
    obs, keep = L.observable(z, w, 0.5)
    vw, gw = O.adjoint(n, ops, params, obs)
    assert abs(v - vw) <= 1e-10
    assert np.max(np.abs(g - gw)) <= 1e-10


# one amplitude per thread up to 17 qubits, 16 above, and at 17 qubits from 65 terms on
@pytest.mark.parametrize("n,nterms", [(4, 100), (16, 64), (16, 65), (17, 0), (17, 64), (17, 65), (17, 300), (18, 5)])
def test_either_side_of_the_kernels(n, nterms):
    from quantumsimevo_b200.circuit import Circuit

    rng = np.random.default_rng(100 * n + nterms)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    c = Circuit(n)
    c.state.upload(psi)
    z = rng.integers(0, 1 << n, nterms, dtype=np.uint64)
    w = rng.standard_normal(nterms)
    # some hundred terms added one by one: as many roundings of 2^-53 of sum |w|, with the norm 1
    assert abs(c.expectation(z, w, 0.25) - _plain(psi, z, w, 0.25)) <= 1e-13 * (0.25 + float(np.abs(w).sum()))


@pytest.mark.parametrize("n", [16, 17, 18])
def test_gradient_on_either_side(n):
    import oracle_ffi as O
    from quantumsimevo_b200 import _lib as L
    from quantumsimevo_b200.autograd import ParametrizedCircuit

    ops = np.zeros(2 * n, dtype=L.OP_DTYPE)
    ops["type"], ops["target"], ops["param"], ops["coeff"] = [L.RY, L.RX] * n, np.arange(2 * n) // 2, np.arange(2 * n), 1.0
    params = np.random.default_rng(n).uniform(-3, 3, 2 * n)
    z, w = [(1 << q) | 1 for q in range(1, n)] + [1 << (n - 1)], list(np.linspace(-1, 1, n))
    v, g = ParametrizedCircuit(n, ops, z, w, 0.5).value_and_grad(params)
    obs, keep = L.observable(z, w, 0.5)
    vw, gw = O.adjoint(n, ops, params, obs)
    assert abs(v - vw) <= 1e-10
    assert np.max(np.abs(g - gw)) <= 1e-10
