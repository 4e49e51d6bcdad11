"""The work that programs built on this framework give it, as timed cases.

Every case goes through a public entry point (Circuit, ParametrizedCircuit and
its autograd function, Batch, or the C ABI's per-gate calls that the C++
adapter makes) at the sizes of the repository's own configurations, tests and
benchmark, and at odd sizes between them:

  train     gradient-descent steps on a parameterised circuit through torch
            autograd (forward and adjoint); every step has new angles, as an
            optimiser gives them
  energy    <O> of one circuit at several angle vectors (a scan of a QAOA
            landscape): forward passes and the expectation, no gradient
  circuit   one execute from |0..0>; small states come back to the host with a
            few shots, large ones stay on the device as a torch tensor
  noisy     one execute with Pauli noise from given draws
  gates     the per-gate interface: one kernel per gate, as
            CircuitUnitaryOperationB200 drives it
  sample    exact sampling of a state that has just changed
  batch     values and gradients of many small circuits in one call
"""
import math
import random

import numpy as np
import torch

from quantumsimevo_b200 import _lib as L
from quantumsimevo_b200.autograd import ParametrizedCircuit
from quantumsimevo_b200.batch import Batch, BatchConfig
from quantumsimevo_b200.circuit import Circuit, StateVector

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a variational circuit of a few qubits in an optimiser loop: the
        # smallest calls, all latency and launches
        dict(name="train_hea_8q", kind="train", family="hea", qubits=8, layers=3, steps=8, structure=1),
        # the same at an odd size where the state is a few MiB
        dict(name="train_hea_17q", kind="train", family="hea", qubits=17, layers=6, steps=3, structure=2),
        # QAOA Max-Cut training at the repository's 24-qubit, p = 8 configuration
        dict(name="train_qaoa_24q_p8", kind="train", family="qaoa", qubits=24, layers=8, steps=3, structure=4),
        # QAOA landscape scan, the cost layer written with CNOT RZ CNOT as the
        # playground's Max-Cut writes it
        dict(name="energy_qaoa_28q_p2", kind="energy", family="qaoa_cx", qubits=28, layers=2, steps=4, structure=5),
        # the 16-qubit, 1260-gate layered-rotation configuration, state and shots to the host
        dict(name="layered_16q", kind="circuit", family="layered", qubits=16, layers=20, shots=4096, structure=0),
        # the headline circuit, H + RZ + QFT on 30 qubits (540 gates), state kept on the device
        dict(name="hrz_qft_30q", kind="circuit", family="hrz_qft", qubits=30, layers=1, shots=0, structure=0),
        # the noisy random-layer configuration at an odd size
        dict(name="noisy_random_27q", kind="noisy", family="random", qubits=27, layers=6, structure=3),
        # the drop-in route: one call and one kernel per gate
        dict(name="gates_26q", kind="gates", family="gates", qubits=26, layers=1, structure=6),
        # shots from a small state, and a million shots from the largest one
        dict(name="sample_17q", kind="sample", qubits=17, shots=5000),
        dict(name="sample_30q", kind="sample", qubits=30, shots=1000000),
        # many small variational circuits at once: widths that fit one tile, and
        # the benchmark's widths (10 to 22) at a quarter of its circuit count
        dict(name="batch_48_narrow", kind="batch", count=48, wmin=6, wmax=13, dmin=2, dmax=6, structure=7),
        dict(name="batch_128", kind="batch", count=128, wmin=10, wmax=22, dmin=4, dmax=12, structure=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "energy", "circuit", "circuit", "noisy", "gates", "sample", "sample", "batch"])
    s = rng.randrange(1 << 20)
    if kind == "train":
        fam = rng.choice(["hea", "qaoa"])
        n = rng.randint(6, 22)
        return dict(kind=kind, family=fam, qubits=n, layers=rng.randint(2, 6), steps=rng.randint(2, 4), structure=s)
    if kind == "energy":
        return dict(kind=kind, family=rng.choice(["qaoa", "qaoa_cx"]), qubits=rng.randint(12, 28),
                    layers=rng.randint(1, 3), steps=rng.randint(2, 4), structure=s)
    if kind == "circuit":
        fam = rng.choice(["layered", "hrz_qft", "random"])
        n = rng.randint(10, 28)
        return dict(kind=kind, family=fam, qubits=n, layers=rng.randint(1, 6) if n > 16 else rng.randint(4, 20),
                    shots=rng.choice([0, 100, 4096]) if n <= 18 else 0, structure=s)
    if kind == "noisy":
        return dict(kind=kind, family="random", qubits=rng.randint(12, 27), layers=rng.randint(2, 8), structure=s)
    if kind == "gates":
        return dict(kind=kind, family="gates", qubits=rng.randint(10, 28), layers=1, structure=s)
    if kind == "sample":
        return dict(kind=kind, qubits=rng.randint(12, 29), shots=_log(rng, 1, 1000000))
    lo = rng.randint(6, 12)
    return dict(kind=kind, count=_log(rng, 8, 96), wmin=lo, wmax=lo + rng.randint(0, 8), dmin=2, dmax=rng.randint(3, 8),
                structure=s)


# ---- circuits, as plain tuples (type, target, other, theta, controls, param, coeff, matrix) ----
NONE8 = (0.0,) * 8


def _g(t, q, other=0, theta=0.0, controls=0, param=-1, coeff=1.0, m=NONE8):
    return (t, q, other, theta, controls, param, coeff, m)


def _edges(n, seed):
    """About 3n/2 distinct edges: a ring and random chords."""
    rng = random.Random(seed)
    e = {(min(i, (i + 1) % n), max(i, (i + 1) % n)) for i in range(n)}
    while len(e) < min((3 * n) // 2, n * (n - 1) // 2):
        u, v = rng.sample(range(n), 2)
        e.add((min(u, v), max(u, v)))
    return sorted(e)


def _gates(case):
    """(gates, parameter count, angle slots).  The structure comes from the case;
    gates with theta None take the next of the `angle slots` angles drawn from
    the inputs' seed."""
    fam, n, layers = case["family"], case["qubits"], case["layers"]
    rng = random.Random(case["structure"])
    g, npar = [], 0
    if fam == "hea":   # RY RZ on every qubit, then a ring of CNOTs
        for _ in range(layers):
            for q in range(n):
                g += [_g(L.RY, q, param=npar), _g(L.RZ, q, param=npar + 1)]
                npar += 2
            g += [_g(L.CNOT, (q + 1) % n, q) for q in range(n)]
    elif fam in ("qaoa", "qaoa_cx"):
        npar = 2 * layers
        g = [_g(L.H, q) for q in range(n)]
        for l in range(layers):
            for u, v in _edges(n, case["structure"]):
                if fam == "qaoa":
                    g += [_g(L.RZ, u, param=l, coeff=2.0), _g(L.RZ, v, param=l, coeff=2.0),
                          _g(L.CPHASE, v, u, param=l, coeff=-4.0)]
                else:
                    g += [_g(L.CNOT, v, u), _g(L.RZ, v, param=l, coeff=4.0), _g(L.CNOT, v, u)]
            g += [_g(L.RX, q, param=layers + l, coeff=2.0) for q in range(n)]
    elif fam == "layered":
        for _ in range(layers):
            for q in range(n):
                g += [_g(L.RX, q, theta=None), _g(L.RY, q, theta=None), _g(L.RZ, q, theta=None)]
            g += [_g(L.CNOT, q + 1, q) for q in list(range(0, n - 1, 2)) + list(range(1, n - 1, 2))]
    elif fam == "hrz_qft":
        g = [_g(L.H, q) for q in range(n)] + [_g(L.RZ, q, theta=None) for q in range(n)]
        for i in range(n):
            g.append(_g(L.H, i))
            g += [_g(L.CPHASE, i, j, math.pi / 2.0 ** (j - i)) for j in range(i + 1, n)]
        g += [_g(L.SWAP, i, n - 1 - i) for i in range(n // 2)]
    elif fam == "random":   # one 1-qubit gate per qubit, disjoint 2-qubit gates, one MCPHASE per layer
        for _ in range(layers):
            for q in range(n):
                t = rng.choice([L.H, L.X, L.Y, L.Z, L.RX, L.RY, L.RZ, L.PHASE])
                g.append(_g(t, q, theta=None if t in (L.RX, L.RY, L.RZ, L.PHASE) else 0.0))
            perm = rng.sample(range(n), n)
            for k in range(n // 2):
                a, b = perm[2 * k], perm[2 * k + 1]
                t = rng.choice([L.CNOT, L.CPHASE, L.SWAP])
                g.append(_g(t, b, a, theta=None if t == L.CPHASE else 0.0))
            pick = rng.sample(range(n), 4)
            g.append(_g(L.MCPHASE, pick[3], theta=None, controls=sum(1 << p for p in pick[:3])))
    else:   # "gates": H on every qubit, then every gate type at low, middle and high positions
        g = [_g(L.H, q) for q in range(n)]
        c, s = math.cos(0.3), math.sin(0.3)
        for q in (0, 1 + rng.randrange(3), n // 2, n - 2 - rng.randrange(2), n - 1):
            o = rng.choice([x for x in range(n) if x != q])
            g += [_g(t, q, theta=None) for t in (L.RX, L.RY, L.RZ, L.PHASE)] + [_g(t, q) for t in (L.X, L.Y, L.Z)]
            g += [_g(L.CNOT, q, o), _g(L.CPHASE, q, o, theta=None),
                  _g(L.MCPHASE, q, theta=None, controls=sum(1 << x for x in rng.sample([x for x in range(n) if x != q], 3))),
                  _g(L.GATE2X2, q, m=(c, 0.0, 0.0, -s, 0.0, -s, c, 0.0))]
    return g, npar, sum(1 for x in g if x[3] is None)


def _with_angles(gates, seed):
    rng = random.Random(seed)
    return [x if x[3] is not None else x[:3] + (rng.uniform(0.0, TWO_PI),) + x[4:] for x in gates]


def _ops(gates):
    a = np.zeros(len(gates), dtype=L.OP_DTYPE)
    for i, (t, q, o, th, ctl, par, co, m) in enumerate(gates):
        a[i] = (t, q, o, par, ctl, th, co, m)
    return a


def _observable(case):
    n = case["qubits"]
    if case["family"] == "hea":
        return [1 << q for q in range(n)], [1.0] * n, 0.0
    e = _edges(n, case["structure"])
    return [(1 << u) | (1 << v) for u, v in e], [-0.5] * len(e), 0.5 * len(e)


def _params(case, npar, seed):
    rng = np.random.default_rng(seed)
    hi = TWO_PI if case["kind"] == "batch" or case["family"] == "hea" else math.pi
    return rng.uniform(0.0, hi, npar)


RATE = 0.05   # learning rate of the training loops

# gate types of the noise model's rate map (each takes two uniforms)
NOISY = (L.X, L.Y, L.Z, L.H, L.CNOT, L.PHASE, L.RX, L.RY, L.RZ)


def _batch_circuits(case, seed):
    """(qubits, gates, params, observable) of every circuit of a batch."""
    rng = random.Random(case["structure"])
    out = []
    for i in range(case["count"]):
        w, d = rng.randint(case["wmin"], case["wmax"]), rng.randint(case["dmin"], case["dmax"])
        c = dict(kind="batch", family="hea", qubits=w, layers=d, structure=0)
        g, npar, _ = _gates(c)
        out.append((w, g, _params(c, npar, seed * 1000 + i), _observable(c)))
    return out


class _DeviceView:
    """A state's device buffer (2^n complex128) for torch.  It holds the state: the
    tensor keeps this object, so the buffer lives as long as any view of it."""

    def __init__(self, ptr, state):
        self.state = state
        self.__cuda_array_interface__ = {"shape": (1 << state.num_qubits, 2), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3}


def _amplitudes(state):
    """The state's amplitudes in logical order, as a torch view of its own buffer."""
    L.check(L.lib.qse_state_canonicalize(state.handle))
    p = L.C.c_void_p()
    L.check(L.lib.qse_state_device_ptr(state.handle, L.C.byref(p)))
    return torch.view_as_complex(torch.as_tensor(_DeviceView(p.value, state), device="cuda"))


def _random_state(n, seed, out):
    """Gaussian amplitudes of norm 1 (a random circuit's output statistics)."""
    v = torch.view_as_real(out)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    v.normal_(generator=gen)
    v.mul_(1.0 / math.sqrt(float((v * v).sum() if n < 26 else sum(float((x * x).sum()) for x in v.split(1 << 24)))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("train", "energy"):
        gates, npar, _ = _gates(case)
        s["circuit"] = ParametrizedCircuit(case["qubits"], _ops(gates), *_observable(case))
        if kind == "train":
            s["params"] = torch.tensor(_params(case, npar, seed), dtype=torch.float64, device="cuda")
        else:
            s["params"] = [_params(case, npar, seed * 100 + k) for k in range(case["steps"])]
    elif kind == "batch":
        circs = _batch_circuits(case, seed)
        s["batch"] = Batch([(w, _ops(g), len(p), obs) for w, g, p, obs in circs])
        # the configuration that the autotuner picks for batches of such circuits
        s["batch"].config = BatchConfig(threads=256, reg_bits=3, max_gates=48, chain_tiles=16)
        s["params"] = np.concatenate([p for _, _, p, _ in circs])
    elif kind == "sample":
        n = case["qubits"]
        s["circuit"] = Circuit(n, seed=1)
        _random_state(n, seed, _amplitudes(s["circuit"].state))
        torch.cuda.synchronize()
        s["uniforms"] = np.random.default_rng(seed).random(case["shots"])
        s["controls"] = (L.C.c_uint32 * (n - 1))(*range(n - 1))
    elif kind == "gates":
        gates, _, _ = _gates(case)
        s["state"] = StateVector(case["qubits"])
        s["gates"] = _with_angles(gates, seed)
    else:
        gates, _, _ = _gates(case)
        gates = _with_angles(gates, seed)
        s["circuit"] = Circuit(case["qubits"], kind == "noisy", noise_rng=L.RNG_INJECTED, seed=1)
        s["circuit"].add_ops(_ops(gates))
        if kind == "noisy":
            s["uniforms"] = np.random.default_rng(seed).random(2 * sum(1 for x in gates if x[0] in NOISY))
        else:
            s["uniforms"] = np.random.default_rng(seed).random(case["shots"])
    return s


def _apply(h, x):
    """One per-gate call of the C ABI."""
    t, q, o, th, ctl, _, _, m = x
    lib = L.lib
    if t in _PLAIN:
        st = _PLAIN[t](h, q)
    elif t in _ANGLE:
        st = _ANGLE[t](h, q, th)
    elif t == L.CNOT:
        st = lib.qse_apply_cnot(h, o, q)
    elif t == L.CPHASE:
        st = lib.qse_apply_cphase(h, o, q, th)
    elif t == L.MCPHASE:
        c = [b for b in range(64) if (ctl >> b) & 1]
        st = lib.qse_apply_mcphase(h, (L.C.c_uint32 * len(c))(*c), len(c), q, th)
    else:
        st = lib.qse_apply_gate2x2(h, (L.C.c_double * 8)(*m), q)
    L.check(st)


_PLAIN = {L.H: L.lib.qse_apply_h, L.X: L.lib.qse_apply_x, L.Y: L.lib.qse_apply_y, L.Z: L.lib.qse_apply_z}
_ANGLE = {L.RX: L.lib.qse_apply_rx, L.RY: L.lib.qse_apply_ry, L.RZ: L.lib.qse_apply_rz, L.PHASE: L.lib.qse_apply_phase}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "train":
        p, values = s["params"], []
        for _ in range(case["steps"]):
            p = p.detach().requires_grad_(True)
            e = s["circuit"].expectation(p)
            (g,) = torch.autograd.grad(e, p)
            p = p - RATE * g
            values.append(e.detach())
        return [torch.stack(values), p.detach(), g]
    if kind == "energy":
        return np.array([s["circuit"].value(p) for p in s["params"]])
    if kind == "batch":
        return list(s["batch"].run(s["params"]))
    if kind == "sample":
        c = s["circuit"]
        # a phase flip of the all-ones basis state (a Grover oracle), then the shots
        L.check(L.lib.qse_apply_mcphase(c.state.handle, s["controls"], case["qubits"] - 1, case["qubits"] - 1, math.pi))
        return c.sample(case["shots"], uniforms=s["uniforms"])
    if kind == "gates":
        s["state"].reset()
        for x in s["gates"]:
            _apply(s["state"].handle, x)
        return _amplitudes(s["state"])
    c = s["circuit"]
    c.state.reset()
    if kind == "noisy":
        c.noise.reset_stats()
        c.execute(noise_uniforms=s["uniforms"])
        bits, phases = c.noise.counts()
        return [_amplitudes(c.state), np.array(bits), np.array(phases)]
    c.execute()
    if case["qubits"] <= 18:
        out = [c.get_state_vector()]
        return out + [c.sample(case["shots"], uniforms=s["uniforms"])] if case["shots"] else out
    return _amplitudes(c.state)


def _count(gates, n):
    """Floating-point operations of a gate list on 2^n amplitudes: 4 per amplitude
    for a rotation (one real FMA per component, its cosine or sine taken out as a
    factor of the state), 2 for an H (likewise), 12 for a general 2x2, and 6 for
    each run of phase gates between two of those (a run merges into one factor)."""
    f, run = 0.0, False
    for x in gates:
        f += {L.RX: 4.0, L.RY: 4.0, L.H: 2.0, L.GATE2X2: 12.0}.get(x[0], 0.0) * (1 << n)
        if x[0] in (L.Z, L.PHASE, L.RZ, L.CPHASE, L.MCPHASE):
            run = True
        elif run:
            f, run = f + 6.0 * (1 << n), False
    return f


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # forward on one state, reverse on two, each circuit's state resident on the chip
        b = f = 0.0
        for w, g, p, _ in _batch_circuits(case, 0):
            b += 16.0 * len(p)
            f += 3.0 * _count(g, w)
        return {"bytes": b, "flops": f}
    n = case["qubits"]
    if kind == "sample":
        return {"bytes": 16.0 * (1 << n) + 16.0 * case["shots"], "flops": 4.0 * (1 << n)}
    gates, npar, _ = _gates(case)
    if kind == "train":
        # the state written once, and both states read and written once by the sweep back
        return {"bytes": case["steps"] * 80.0 * (1 << n), "flops": case["steps"] * 3.0 * _count(gates, n)}
    if kind == "energy":
        return {"bytes": case["steps"] * 32.0 * (1 << n), "flops": case["steps"] * _count(gates, n)}
    return {"bytes": 16.0 * (1 << n), "flops": _count(gates, n)}


# ---- the same results in plain torch, 64 bits ----
def _matrix(t, th, m):
    c, s = math.cos(th / 2), math.sin(th / 2)
    r = math.sqrt(0.5)
    return {L.H: (r, r, r, -r), L.X: (0, 1, 1, 0), L.Y: (0, -1j, 1j, 0), L.RX: (c, -1j * s, -1j * s, c),
            L.RY: (c, -s, s, c), L.GATE2X2: (complex(m[0], m[1]), complex(m[2], m[3]), complex(m[4], m[5]),
                                             complex(m[6], m[7]))}[t]


def _sub(psi, fixed):
    """View of the amplitudes whose qubits in `fixed` ({qubit: bit}) have those bits."""
    v, at, top = psi.reshape(-1), 0, int(math.log2(psi.numel()))
    shape, idx = [], []
    for q in sorted(fixed, reverse=True):
        shape += [1 << (top - q - 1), 2]
        idx += [slice(None), fixed[q]]
        top = q
    return v.view(shape + [1 << top])[tuple(idx)]


def _exact_gate(psi, x, angle, dagger=False):
    """Applies gate x (or its inverse) to psi in place."""
    t, q, o, _, ctl, _, _, m = x
    th = -angle if dagger else angle
    if t in (L.Z, L.PHASE):
        _sub(psi, {q: 1}).mul_(-1.0 if t == L.Z else complex(math.cos(th), math.sin(th)))
    elif t == L.RZ:
        _sub(psi, {q: 0}).mul_(complex(math.cos(th / 2), -math.sin(th / 2)))
        _sub(psi, {q: 1}).mul_(complex(math.cos(th / 2), math.sin(th / 2)))
    elif t in (L.CPHASE, L.MCPHASE):
        bits = {q: 1, o: 1} if t == L.CPHASE else {**{b: 1 for b in range(64) if (ctl >> b) & 1}, q: 1}
        _sub(psi, bits).mul_(complex(math.cos(th), math.sin(th)))
    elif t in (L.CNOT, L.SWAP, L.X):
        a, b = {L.CNOT: ({o: 1, q: 0}, {o: 1, q: 1}), L.SWAP: ({o: 0, q: 1}, {o: 1, q: 0}), L.X: ({q: 0}, {q: 1})}[t]
        u, v = _sub(psi, a), _sub(psi, b)
        w = u.clone()
        u.copy_(v)
        v.copy_(w)
    else:
        a, b, c, d = _matrix(t, th, m)
        u, v = _sub(psi, {q: 0}), _sub(psi, {q: 1})
        w = c * u
        u.mul_(a).add_(v, alpha=b)
        v.mul_(d).add_(w)


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda" if torch.cuda.is_available() else "cpu")
    psi[0] = 1.0
    return psi


def _diagonal(n, obs, device):
    i = torch.arange(1 << n, device=device)
    d = torch.full((1 << n,), float(obs[2]), dtype=torch.float64, device=device)
    for z, w in zip(obs[0], obs[1]):
        par = torch.zeros(1 << n, dtype=torch.int64, device=device)
        for b in range(n):
            if (z >> b) & 1:
                par ^= (i >> b) & 1
        d += w * (1 - 2 * par).to(torch.float64)
    return d


def _angles(gates, p):
    return [x[3] if x[5] < 0 else (x[3] or 0.0) + x[6] * float(p[x[5]]) for x in gates]


def _exact_grad(n, gates, p, obs):
    """<O> and its gradient by the textbook adjoint sweep."""
    th = _angles(gates, p)
    psi = _zero(n)
    for x, a in zip(gates, th):
        _exact_gate(psi, x, a)
    d = _diagonal(n, obs, psi.device)
    lam = psi * d
    value = torch.vdot(psi, lam).real
    slots = [[] for _ in p]
    for x, a in zip(reversed(gates), reversed(th)):
        if x[5] >= 0:
            # d<O>/dtheta = 2 Re <lam| dU/dtheta U^-1 |psi>, with psi still after the gate
            t, q, o = x[0], x[1], x[2]
            if t in (L.RX, L.RY):
                w = psi.clone()
                _exact_gate(w, _g(L.X if t == L.RX else L.Y, q), 0.0)
                v = torch.vdot(lam.view(-1), w).imag
            elif t == L.RZ:
                v = (torch.sum(_sub(lam, {q: 0}).conj() * _sub(psi, {q: 0})) -
                     torch.sum(_sub(lam, {q: 1}).conj() * _sub(psi, {q: 1}))).imag
            else:
                b = {q: 1, o: 1}
                v = -2.0 * torch.sum(_sub(lam, b).conj() * _sub(psi, b)).imag
            slots[x[5]].append(x[6] * v)
        _exact_gate(psi, x, a, dagger=True)
        _exact_gate(lam, x, a, dagger=True)
    return float(value), np.array([float(sum(v)) for v in slots])


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None   # whole numbers
    if kind == "batch":
        circs = _batch_circuits(case, seed)
        if sum(len(g) for _, g, _, _ in circs) > 20000 or max(w for w, _, _, _ in circs) > 18:
            return None   # minutes of small torch calls
        r = [_exact_grad(w, g, p, obs) for w, g, p, obs in circs]
        return [np.array([v for v, _ in r]), np.concatenate([g for _, g in r])]
    gates, npar, _ = _gates(case)
    n = case["qubits"]
    if kind == "train":
        p, values = _params(case, npar, seed), []
        for _ in range(case["steps"]):
            v, g = _exact_grad(n, gates, p, _observable(case))
            p = p - RATE * g
            values.append(v)
        return [np.array(values), p, g]
    if kind == "energy":
        d, out = None, []
        for k in range(case["steps"]):
            psi = _zero(n)
            for x, a in zip(gates, _angles(gates, _params(case, npar, seed * 100 + k))):
                _exact_gate(psi, x, a)
            d = _diagonal(n, _observable(case), psi.device) if d is None else d
            out.append(float(torch.sum(d * (psi.real ** 2 + psi.imag ** 2))))
        return np.array(out)
    gates = _with_angles(gates, seed)
    psi = _zero(n)
    for x in gates:
        _exact_gate(psi, x, x[3])
    if kind == "noisy":
        bits, phases = _noise_counts(gates, n, np.random.default_rng(seed).random(2 * sum(1 for x in gates if x[0] in NOISY)))
        for q in range(n):
            if bits[q] % 2:
                _exact_gate(psi, _g(L.X, q), 0.0)
        for q in range(n):
            if phases[q] % 2:
                _exact_gate(psi, _g(L.Z, q), 0.0)
        return [psi, None, None]
    if kind == "gates" or n > 18:
        return psi
    out = [psi.cpu().numpy()]
    return out + [None] if case["shots"] else out


# the noise model's default rates: 1e-3 for X, Y, Z, PHASE, RX, RY, RZ, 2e-3 for H, 5e-3 for CNOT
RATES = {**{t: 1e-3 for t in NOISY}, L.H: 2e-3, L.CNOT: 5e-3}


def _noise_counts(gates, n, u):
    bits, phases, k = [0] * n, [0] * n, 0
    for x in gates:
        if x[0] in RATES:
            bits[x[1]] += u[k] < RATES[x[0]]
            phases[x[1]] += u[k + 1] < RATES[x[0]]
            k += 2
    return bits, phases
