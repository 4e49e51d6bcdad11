"""qse_plan_compile generates and compiles what an execute runs: the same layouts,
register shapes and lane swaps by qubit count (NVRTC needs no GPU).  The sources
are read back from QSE_JIT_DUMP."""
import ctypes as C
import re

import numpy as np
import pytest

from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200 import workloads as W


def kernels(tmp_path, monkeypatch, n, ops, nstates, tile=0, params=None):
    """{file name: text after the device templates} of every kernel compiled."""
    monkeypatch.setenv("QSE_JIT_DUMP", str(tmp_path))
    p = None if params is None else np.ascontiguousarray(params)
    size = C.c_size_t()
    rc = L.lib.qse_plan_compile(n, L.dptr(ops), len(ops), None if p is None else p.ctypes.data_as(L._pd),
                                0 if p is None else p.size, tile, nstates, C.byref(size))
    if rc == 6:
        pytest.skip("NVRTC not available: " + L.lib.qse_last_error().decode())
    L.check(rc)
    assert size.value > 0
    return {f.name: f.read_text().split('extern "C"')[1] for f in tmp_path.iterdir()}


def amplitudes(text):
    return int(re.search(r"double2 a0\[(\d+)\]", text).group(1))


# (qubits, tile asked for, amplitudes per thread, lane swaps possible)
@pytest.mark.parametrize("n,tile,amps,swaps", [
    (3, 0, 8, False), (4, 0, 8, False), (14, 0, 8, False), (19, 0, 8, False), (20, 0, 8, True), (21, 0, 16, True),
    (14, 12, 16, False), (20, 12, 16, True), (20, 10, 16, True), (22, 0, 16, True),
])
def test_forward_passes(tmp_path, monkeypatch, n, tile, amps, swaps):
    k = kernels(tmp_path, monkeypatch, n, W.random_circuit(n, 6 * n, 40 + n), 1, tile)
    assert {amplitudes(t) for t in k.values()} == {amps}
    assert any("laneSwap<" in t for t in k.values()) == swaps


def test_first_pass_from_a_compact_state(tmp_path, monkeypatch):
    """32 amplitudes per thread where the first pass of a large state makes its input
    from a compact one, 16 in the others."""
    k = kernels(tmp_path, monkeypatch, 24, W.hrz_qft(24, seed=2), 1)
    assert {amplitudes(t) for f, t in k.items() if f.startswith("qse_pass_compact_in")} == {32}
    assert {amplitudes(t) for f, t in k.items() if not f.startswith("qse_pass_compact_in")} == {16}


@pytest.mark.parametrize("n,amps,swaps", [(10, 8, False), (11, 8, False), (19, 8, False), (20, 8, True), (22, 16, True), (24, 16, True)])
def test_reverse_passes(tmp_path, monkeypatch, n, amps, swaps):
    ops, params, _, _ = W.qaoa_maxcut(n if n % 2 == 0 else n + 1, 1, seed=3)
    ops = ops[(ops["target"] < n) & (ops["control"] < n)]
    k = kernels(tmp_path, monkeypatch, n, ops, 2, 0, params)
    assert {amplitudes(t) for t in k.values()} == {amps}
    assert any("laneSwap<" in t and "(a1)" in t for t in k.values()) == swaps


def test_streamed_passes_swap_no_lanes(tmp_path, monkeypatch):
    k = kernels(tmp_path, monkeypatch, 26, W.random_circuit(26, 120, 9), 3)
    streamed = [t for t in k.values() if "nfill" in t]
    assert streamed and not any("laneSwap<" in t for t in streamed)
