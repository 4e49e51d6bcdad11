"""qse_state_canonicalize: the amplitudes move to logical order in place, for
maps made of swaps (one pass), of longer cycles (two passes) and at sizes
around the tile (2^11 amplitudes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(n, kind):
    rng = np.random.default_rng(n)
    if kind == "reversed":
        return list(range(n))[::-1]
    if kind == "high pair":
        return list(range(n - 2)) + [n - 1, n - 2]
    if kind == "high swaps":   # the low bits stay
        p = list(range(n))
        for a, b in ((n - 1, n - 4), (n - 2, n - 3)):
            p[a], p[b] = p[b], p[a]
        return p
    if kind == "cycle":
        return list(range(1, n)) + [0]
    return list(rng.permutation(n))


@pytest.mark.parametrize("kind", ["reversed", "high pair", "high swaps", "cycle", "random"])
@pytest.mark.parametrize("n", [4, 5, 8, 9, 10, 11, 12, 13, 16, 21])
def test_canonicalize_moves_amplitudes_to_logical_order(n, kind):
    from quantumsimevo_b200 import _lib as L
    from quantumsimevo_b200.circuit import StateVector

    st = StateVector(n)
    rng = np.random.default_rng(100 + n)
    phys = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    st.upload(phys)
    want = _map(n, kind)   # logical qubit -> physical bit, reached by relabelling swaps
    for q in range(n):
        cur = st.qubit_map()
        L.check(L.lib.qse_apply_swap(st.handle, q, cur.index(want[q])))
    assert st.qubit_map() == want
    L.check(L.lib.qse_state_canonicalize(st.handle))
    assert st.qubit_map() == list(range(n))
    i = np.arange(1 << n, dtype=np.int64)
    p = np.zeros_like(i)
    for q in range(n):
        p |= ((i >> q) & 1) << want[q]
    assert np.array_equal(st.download(), phys[p])
