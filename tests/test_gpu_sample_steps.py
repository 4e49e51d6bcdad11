"""Exact sampling of states whose running sum changes binade inside a block in
every way the block routine treats apart: zero prefixes that end off its run
length, many binades in one block, ties before and after the crossing,
subnormal sums, and a crossing on a block's first or last element."""
import numpy as np
import pytest

import oracle_ffi as O
from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200.circuit import StateVector

pytestmark = pytest.mark.gpu


def _amplitudes(kind, size, rng):
    if kind == "zero prefix":          # 0, then values; the first nonzero at an odd place
        m = rng.random(size)
        m[: rng.integers(1, 4000)] = 0.0
    elif kind == "growing":            # the sum doubles every few dozen elements
        m = np.exp2(np.arange(size) % 4096 / 40.0 - 60.0) * (1.0 + rng.random(size))
    elif kind == "ties":               # squares of dyadic values: exact halves of the grid
        m = np.exp2(-rng.integers(0, 27, size).astype(np.float64))
    elif kind == "ties then jump":
        m = np.exp2(-27.0 + 0.0 * np.arange(size))
        m[0] = 1.0
        m[4095] = 2.0
        m[min(4096, size - 1)] = 4.0
        m[5000:5010] = 1.5   # (empty at 12 qubits)
    elif kind == "subnormal":          # squares below 2^-1022, then normal ones
        m = np.exp2(-rng.integers(505, 530, size).astype(np.float64))
        m[size // 2 + 17:] = np.exp2(-20.0)
    elif kind == "uniform":
        m = np.full(size, 1.0 / np.sqrt(size))
    else:                              # "random": Gaussian amplitudes
        return (rng.standard_normal(size) + 1j * rng.standard_normal(size)) / np.sqrt(2.0 * size)
    return m.astype(np.complex128)


@pytest.mark.parametrize("kind", ["zero prefix", "growing", "ties", "ties then jump", "subnormal", "uniform", "random"])
@pytest.mark.parametrize("n", [12, 13, 15, 17])
@pytest.mark.parametrize("few", [True, False])
def test_sample_bit_exact_across_binades(n, kind, few):
    size = 1 << n
    rng = np.random.default_rng(7 * n + len(kind))
    amp = _amplitudes(kind, size, rng)
    cum = O.cdf(amp, n)
    cum = np.asarray(cum)
    at = np.concatenate([rng.integers(0, size, 40), np.arange(0, size, max(1, size // 64)), [0, 63, 64, 65, 4095]])
    u = cum[at] / cum[-1]
    u = np.concatenate([u, np.nextafter(u, 0.0), np.nextafter(u, 1.0), rng.random(200), [0.0]])
    u = np.clip(u, 0.0, np.nextafter(1.0, 0.0))
    if few:   # the route of a few shots: one thread block per shot
        u = u[rng.permutation(len(u))[:60]]
    st = StateVector(n)
    st.upload(amp)
    out = np.empty(len(u), dtype=np.uint64)
    u = np.ascontiguousarray(u)
    L.check(L.lib.qse_sample(st.handle, u.ctypes.data_as(L._pd), len(u), 0, out.ctypes.data_as(L._pu64)))
    assert np.array_equal(out, O.sample(amp, n, u))


# 24 shots per 4096-amplitude block and more are bucketed by block, fewer answered a warp each
@pytest.mark.parametrize("kind", ["zero prefix", "growing", "ties", "ties then jump", "subnormal", "uniform", "random"])
@pytest.mark.parametrize("n", [14, 15, 17, 21])   # 21: more blocks than thread blocks rebuild at a time
def test_few_and_many_shots_per_block(n, kind):
    size = 1 << n
    rng = np.random.default_rng(11 * n + len(kind))
    amp = _amplitudes(kind, size, rng)
    cum = np.asarray(O.cdf(amp, n))
    limit = 24 * (size // 4096)
    at = rng.integers(0, size, limit)
    u = cum[at] / cum[-1]
    u[::3] = np.nextafter(u[::3], 0.0)
    u[1::3] = rng.random(len(u[1::3]))
    u = np.clip(u, 0.0, np.nextafter(1.0, 0.0))
    st = StateVector(n)
    st.upload(amp)
    want = O.sample(amp, n, u)
    for shots in (limit - 1, limit):
        out = np.empty(shots, dtype=np.uint64)
        L.check(L.lib.qse_sample(st.handle, u.ctypes.data_as(L._pd), shots, 0, out.ctypes.data_as(L._pu64)))
        assert np.array_equal(out, want[:shots])
    drawn = np.empty((2, limit), dtype=np.uint64)   # the device's own draws: the same on either route
    L.check(L.lib.qse_sample(st.handle, None, limit - 1, 5, drawn[0].ctypes.data_as(L._pu64)))
    L.check(L.lib.qse_sample(st.handle, None, limit, 5, drawn[1].ctypes.data_as(L._pu64)))
    assert np.array_equal(drawn[0, : limit - 1], drawn[1, : limit - 1])
