"""The autotuner's cache file: an entry that an earlier revision of the batched
kernels wrote (its key had no revision) stands for kernels that no longer exist
and is measured again; the entry written then is used."""
import json

import numpy as np
import pytest

from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200.batch import Batch
from quantumsimevo_b200.circuit import Device

pytestmark = pytest.mark.gpu


def unrevised_key(circs):
    """FNV-1a over the batch's structure, as 8-byte little-endian words."""
    import torch

    h = 1469598103934665603

    def mix(v):
        nonlocal h
        for b in int(v).to_bytes(8, "little"):
            h = ((h ^ b) * 1099511628211) & (2 ** 64 - 1)

    mix(len(circs))
    for n, ops, _, obs in circs:
        mix(n)
        mix(len(ops))
        for op in ops:
            mix(int(op["type"]) | int(op["target"]) << 32)
            mix(int(op["control"]) | int(op["param"] >= 0) << 32)
            mix(op["controls"])
        mix(len(obs[0]))
    return f"{torch.cuda.get_device_name(0)}/{h:016x}"


def test_entries_of_earlier_kernels_are_measured_again(tmp_path):
    ops = np.zeros(12, dtype=L.OP_DTYPE)
    ops["type"], ops["target"], ops["param"], ops["coeff"] = L.RY, np.arange(12) % 6, np.arange(12), 1.0
    circs = [(6, ops, 12, ([1, 2], [1.0, 0.5], 0.0))]
    path = tmp_path / "tune.json"
    marked = dict(threads=64, reg_bits=2, max_gates=0, chain_tiles=77, ctas_per_sm=0, grad_slots=0, wide_regs=0)
    path.write_text("{\n  " + json.dumps(unrevised_key(circs)) + ": " + json.dumps(marked, separators=(",", ":")) + "\n}\n")
    cfg = Batch(circs, Device(0)).autotune(str(path))
    assert cfg.chain_tiles != 77
    entries = json.loads(path.read_text())
    assert len(entries) == 2
    # the entry just written is used: marked in the file, it comes back marked
    new = next(k for k in entries if k != unrevised_key(circs))
    entries[new]["chain_tiles"] = 78
    lines = [f"  {json.dumps(k)}: {json.dumps(v, separators=(',', ':'))}" for k, v in entries.items()]
    path.write_text("{\n" + ",\n".join(lines) + "\n}\n")
    assert Batch(circs, Device(0)).autotune(str(path)).chain_tiles == 78
