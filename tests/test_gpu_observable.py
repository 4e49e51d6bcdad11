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
