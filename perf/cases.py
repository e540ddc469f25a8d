"""The work that users of quantr_gb300 have it do, as timed cases.

Every case is one call sequence of the public interface on inputs drawn from a seed: a `Circuit`
simulated, read and sampled; a gate program applied to a register that the program keeps (in the
fast and the exact mode, complex128 and complex64); energies; energy + adjoint gradient; batches of
independent circuits; Custom gates. Sizes follow the repository's own configurations (12-, 14-, 20-,
24- and 30-qubit circuits, 31 to 33 qubits of complex64, batches of 10 to 24 qubits) and lie between
them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import quantr_gb300 as q
from quantr_gb300 import _native as nat
from quantr_gb300 import batch, gradients
from quantr_gb300.program import ProgramBuilder

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a small circuit written against the quantr API: simulate, read the state, 1000 shots
        {"name": "circuit_12q", "kind": "circuit", "n": 12, "columns": 40, "shots": 1000},
        # a parity run: every gate in the reference's own arithmetic and order
        {"name": "exact_14q", "kind": "apply", "family": "brickwork_qft", "mode": "exact",
         "precision": "c128", "n": 14, "layers": 20},
        # a mid-size register kept by the program: random columns, an odd qubit count
        {"name": "columns_17q", "kind": "apply", "family": "columns", "mode": "fast",
         "precision": "c128", "n": 17, "layers": 40},
        # the headline family where the register just leaves one SM's and fills the L2 cache
        {"name": "brickwork_21q", "kind": "apply", "family": "brickwork_qft", "mode": "fast",
         "precision": "c128", "n": 21, "layers": 20},
        # the headline circuit: 30 qubits of complex128, norm and a few shots
        {"name": "brickwork_30q", "kind": "sample", "family": "brickwork_qft", "precision": "c128",
         "n": 30, "layers": 20, "shots": 256},
        # the reduced-precision family on a large complex64 register: norm and energy
        {"name": "brickwork_c64_30q", "kind": "energy", "family": "brickwork", "precision": "c64",
         "n": 30, "layers": 4},
        # one objective evaluation of a variational loop
        {"name": "energy_24q", "kind": "energy", "family": "ansatz", "precision": "c128", "n": 24,
         "layers": 4},
        # the differentiation configuration: 400 angles
        {"name": "gradient_20q", "kind": "gradient", "precision": "c128", "n": 20, "layers": 10},
        # a gradient whose vectors no longer fit the L2 cache, odd size
        {"name": "gradient_23q", "kind": "gradient", "precision": "c128", "n": 23, "layers": 4},
        # the same in complex64
        {"name": "gradient_c64_24q", "kind": "gradient", "precision": "c64", "n": 24, "layers": 4},
        # a batch of uneven circuits in complex128
        {"name": "batch_10_20q", "kind": "batch", "precision": "c128", "count": 96, "n_min": 10,
         "n_max": 20, "layers": 4},
        # Custom gates (an oracle with None columns, a damped map) on a register that is sampled
        # and read as a sparse map
        {"name": "custom_18q", "kind": "custom", "n": 18, "layers": 6, "shots": 20000},
    ]


def draw(rng):
    """One more case of the listed kinds; sizes over their whole range, odd ones among them."""
    kind = rng.choice(["circuit", "exact", "columns", "brickwork", "sample", "energy", "gradient",
                       "batch", "custom"])
    if kind == "circuit":
        return {"kind": "circuit", "n": rng.randint(4, 14), "columns": rng.randint(8, 60),
                "shots": int(10 ** rng.uniform(1, 4.5))}
    if kind == "exact":
        return {"kind": "apply", "family": rng.choice(["brickwork_qft", "columns"]),
                "mode": "exact", "precision": "c128", "n": rng.randint(9, 18),
                "layers": rng.randint(4, 24)}
    if kind == "columns":
        return {"kind": "apply", "family": "columns", "mode": "fast",
                "precision": rng.choice(["c128", "c64"]), "n": rng.randint(9, 22),
                "layers": rng.randint(8, 48)}
    if kind == "brickwork":
        return {"kind": "apply", "family": rng.choice(["brickwork_qft", "brickwork", "qft"]),
                "mode": "fast", "precision": rng.choice(["c128", "c64"]), "n": rng.randint(10, 22),
                "layers": rng.randint(2, 20)}
    if kind == "sample":
        return {"kind": "sample", "family": rng.choice(["brickwork_qft", "qft", "columns"]),
                "precision": "c128", "n": rng.randint(20, 28), "layers": rng.randint(4, 20),
                "shots": rng.randint(50, 1000)}
    if kind == "energy":
        precision = rng.choice(["c128", "c64"])
        return {"kind": "energy", "family": rng.choice(["ansatz", "brickwork"]),
                "precision": precision, "n": rng.randint(13, 27 if precision == "c128" else 31),
                "layers": rng.randint(2, 6)}
    if kind == "gradient":
        return {"kind": "gradient", "precision": rng.choice(["c128", "c64"]),
                "n": rng.randint(13, 25), "layers": rng.randint(2, 10)}
    if kind == "batch":
        n_min = rng.randint(4, 14)
        return {"kind": "batch", "precision": rng.choice(["c128", "c64"]),
                "count": int(2 ** rng.uniform(4, 9)), "n_min": n_min,
                "n_max": rng.randint(n_min, 20), "layers": rng.randint(2, 5)}
    return {"kind": "custom", "n": rng.randint(8, 22), "layers": rng.randint(2, 8),
            "shots": int(10 ** rng.uniform(2, 4.5))}


# ---- circuits: gates as (name, target, controls, param, k) -------------------------------------
_ONE_WIRE = ("H", "X", "Y", "Z", "S", "T", "Rx", "Ry", "Rz", "Phase")


def _columns(r, n, layers):
    out = []
    for col in range(layers):
        for w in range(n):
            name = _ONE_WIRE[r.integers(len(_ONE_WIRE))]
            out.append((name, w, (), r.uniform(0.0, TWO_PI) if name in ("Rx", "Ry", "Rz", "Phase")
                        else 0.0, 0))
        c, t = r.permutation(n)[:2]
        out.append(("CNot", int(t), (int(c),), 0.0, 0))
        if col % 5 == 4 and n >= 3:
            c1, c2, t = r.permutation(n)[:3]
            out.append(("Toffoli", int(t), (int(c1), int(c2)), 0.0, 0))
    return out


def _brickwork(r, n, layers):
    out = []
    for layer in range(layers):
        for name in ("Rz", "Ry", "Rz"):
            out += [(name, w, (), r.uniform(0.0, TWO_PI), 0) for w in range(n)]
        out += [("CNot", i + 1, (i,), 0.0, 0) for i in range(layer % 2, n - 1, 2)]
    return out


def _qft(n):
    out = []
    for i in range(n):
        out.append(("H", i, (), 0.0, 0))
        out += [("CRk", i, (i + k - 1,), 0.0, k) for k in range(2, n - i + 1)]
    return out + [("Swap", i, (n - 1 - i,), 0.0, 0) for i in range(n // 2)]


def _ansatz(r, n, layers):
    out = []
    for _ in range(layers):
        out += [("Ry", w, (), r.uniform(-math.pi, math.pi), 0) for w in range(n)]
        out += [("Rz", w, (), r.uniform(-math.pi, math.pi), 0) for w in range(n)]
        out += [("CNot", (w + 1) % n, (w,), 0.0, 0) for w in range(n)]
    return out


def _gates(case, r):
    n, family = case["n"], case.get("family", "ansatz")
    if family == "columns":
        return _columns(r, n, case["layers"])
    if family == "ansatz":
        return _ansatz(r, n, case["layers"])
    if family == "qft":  # of a product state, so that the transform has something to act on
        return [("Ry", w, (), r.uniform(0.0, math.pi), 0) for w in range(n)] + _qft(n)
    return _brickwork(r, n, case["layers"]) + (_qft(n) if family == "brickwork_qft" else [])


def _rng(case, seed):
    return np.random.default_rng([seed, case.get("n", case.get("n_max", 0))])


def _program(gates, n):
    b = ProgramBuilder(n)
    for name, t, ctl, param, k in gates:
        if name == "Custom":
            b.add_custom(t, ctl, param[0], param[1])
        else:
            b.add(name, t, ctl, param, k)
    return b.build()


def _observable(r, n):
    return r.standard_normal(n), r.standard_normal(n)


def _circuit(case, seed):
    """The random-column circuit through the builder, one call a column as a user writes it."""
    r, n = _rng(case, seed), case["n"]
    gates, c = _columns(r, n, case["columns"]), q.Circuit(n)
    at = 0
    while at < len(gates):
        if gates[at][0] in ("CNot", "Toffoli"):
            name, t, ctl, _, _ = gates[at]
            c.add_gate(getattr(q.Gate, name)(*ctl), t)
            at += 1
        else:
            c.add_gates([getattr(q.Gate, g[0])(g[3]) if g[0] in ("Rx", "Ry", "Rz", "Phase")
                         else getattr(q.Gate, g[0]) for g in gates[at:at + n]])
            at += n
    return gates, c


def _custom_gates(case, seed):
    """Layers of rotations, a 3-wire phase oracle that returns None where it does nothing, and a
    damped 2-wire map (not unitary), on random wires."""
    r, n = _rng(case, seed), case["n"]
    gates = [("H", w, (), 0.0, 0) for w in range(0, n, 2)]
    for _ in range(case["layers"]):
        gates += [("Ry", w, (), r.uniform(0.0, 0.2), 0) for w in range(n)]
        w = [int(x) for x in r.permutation(n)[:5]]
        flip = np.zeros((8, 8), np.complex128)
        flip[7, 7] = -1.0
        none = np.ones(8, np.uint8)
        none[7] = 0
        gates.append(("Custom", w[2], (w[0], w[1]), (flip, none), 0))
        g = math.sqrt(r.uniform(0.85, 1.0))
        damp = np.diag(np.array([1.0, 1.0, 1.0, g], np.complex128))
        gates.append(("Custom", w[4], (w[3],), (damp, np.zeros(4, np.uint8)), 0))
        gates += [("CNot", int(b), (int(a),), 0.0, 0) for a, b in r.permutation(n)[:2 * (n // 4)].reshape(-1, 2)]
    return gates


def _batch_items(case, seed):
    # the sizes belong to the case (uniform over its range), the angles and observables to the seed
    sizes = np.random.default_rng(5).integers(case["n_min"], case["n_max"] + 1, case["count"])
    r, out = _rng(case, seed), []
    for n in sizes.tolist():
        gates = _ansatz(r, n, case["layers"])
        a, b = _observable(r, n)
        out.append((n, gates, a, b))
    return out


def _native(case):
    return nat.QGPU_C64 if case["precision"] == "c64" else nat.QGPU_C128


_MODES = {"fast": nat.QGPU_MODE_FAST, "exact": nat.QGPU_MODE_EXACT}


def prepare(case, seed):
    kind, state = case["kind"], {"case": case}
    if kind == "circuit":
        state["circuit"] = _circuit(case, seed)[1]
        state["seed"] = seed
        return state
    if kind == "batch":
        state["circuits"] = [batch.BatchCircuit(_program(g, n), a, b)
                             for n, g, a, b in _batch_items(case, seed)]
        return state
    r = _rng(case, seed)
    if kind == "custom":
        state["program"] = _program(_custom_gates(case, seed), case["n"])
        state["handle"] = nat.Handle(case["n"])
        state["seed"] = seed
        return state
    state["program"] = _program(_gates(case, r), case["n"])
    state["observable"] = _observable(r, case["n"])
    state["seed"] = seed
    state["handle"] = nat.Handle(case["n"], _native(case), _MODES[case.get("mode", "fast")])
    return state


def _padded(a, length, dtype):
    """`a` at the front of a buffer of a size that the inputs do not change."""
    out = np.zeros(length, dtype)
    out[:a.size] = a
    return out


def _histogram(idx, cnt, shots):
    return _padded(idx, shots, np.int64), _padded(cnt, shots, np.int64)


def _survivors(n):
    """At most this many of a normalised register's probabilities reach 1e-6."""
    return min(1 << n, 1100000)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "circuit":
        q.seed(state["seed"])
        sim = state["circuit"].clone_and_simulate()
        amps = sim.get_state().take().get_amplitudes()
        shots = sim.measure_all(case["shots"]).take()
        return (amps, *_histogram(shots.indices, shots.counts, case["shots"]))
    if kind == "batch":
        energies, grads, _ = batch.run_batch(state["circuits"], _native(case))
        flat = np.concatenate(grads)
        return (energies, flat) if case["precision"] == "c128" else \
            (energies.astype(np.float32), flat.astype(np.float32))
    h, p = state["handle"], state["program"]
    if kind == "gradient":
        e, g = gradients.energy_and_gradient(h, p, *state["observable"])
        # results of a complex64 register are kept in its own precision
        return (e, g) if case["precision"] == "c128" else (np.float32(e), g.astype(np.float32))
    if kind == "energy":
        e = gradients.energy(h, p, *state["observable"])
        out = np.array([e, h.norm()])
        return out if case["precision"] == "c128" else out.astype(np.float32)
    h.set_zero()
    h.apply(p.ops, p.mats, p.none)
    if kind == "apply":
        amps = h.download()
        return amps if case["precision"] == "c128" else amps.astype(np.complex64)
    if kind == "sample":
        idx, cnt, _ = h.measure(case["shots"], state["seed"])
        return (h.norm(), *_histogram(idx, cnt, case["shots"]))
    idx, cnt, _ = h.measure(case["shots"], state["seed"])
    keys, amps = h.extract_nonzero()
    size = _survivors(case["n"])
    return (*_histogram(idx, cnt, case["shots"]), _padded(keys, size, np.int64),
            _padded(amps, size, np.complex128))


# ---- what a pass cannot do without ---------------------------------------------------------------
def _gate_flops(name, n):
    """Floating operations of one gate on 2^n amplitudes: 14 per amplitude of a full 2x2 complex
    map, 7 of a real one, 6 of a phase, none where amplitudes only move."""
    dim = float(1 << n)
    return {"Rx": 14, "Ry": 7, "H": 7, "Rz": 6, "Phase": 6, "T": 3, "CRk": 1.5,
            "Custom": 6}.get(name, 0) * dim


def work(case):
    """The register written once and read once by what follows (a gradient: both of its vectors),
    and the gates' arithmetic."""
    if case["kind"] == "batch":
        nbytes = flops = 0.0
        for n, gates, _, _ in _batch_items(case, 0):
            flops += 3.0 * sum(_gate_flops(g[0], n) for g in gates) + 8.0 * n * (1 << n)
            nbytes += 80.0 * len(gates) + 16.0 * n + 8.0 * (len(gates) + 1)
        return {"bytes": nbytes, "flops": flops}
    n, dim = case["n"], float(1 << case["n"])
    amp = 8.0 if case.get("precision") == "c64" else 16.0
    if case["kind"] == "circuit":
        gates = _columns(_rng(case, 0), n, case["columns"])
    elif case["kind"] == "custom":
        gates = _custom_gates(case, 0)
    else:
        gates = _gates(case, _rng(case, 0))
    flops = sum(_gate_flops(g[0], n) for g in gates)
    if case["kind"] == "gradient":
        return {"bytes": 4.0 * amp * dim, "flops": 3.0 * flops + 8.0 * n * dim}
    if case["kind"] == "energy":
        flops += 8.0 * n * dim
    return {"bytes": 2.0 * amp * dim, "flops": flops}


# ---- the same in 64 bits with torch ----------------------------------------------------------------
_R = math.sqrt(0.5)
_FIXED = {"H": (_R, _R, _R, -_R), "X": (0, 1, 1, 0), "Y": (0, -1j, 1j, 0), "Z": (1, 0, 0, -1),
          "S": (1, 0, 0, 1j), "T": (1, 0, 0, complex(_R, _R))}


def _matrix(name, p):
    c, s = math.cos(0.5 * p), math.sin(0.5 * p)
    return {"Rx": (c, -1j * s, -1j * s, c), "Ry": (c, -s, s, c),
            "Rz": (complex(c, -s), 0, 0, complex(c, s)),
            "Phase": (complex(c, s), 0, 0, complex(c, s))}.get(name) or _FIXED[name]


def _apply_exact(psi, n, gate, inverse=False):
    """psi with the gate applied, as a tensor with one axis of two per wire (wire 0 first)."""
    name, t, ctl, p, k = gate
    v = psi.view((2,) * n).clone()
    if name == "Custom":
        wires = list(ctl) + [t]
        block = torch.from_numpy(np.ascontiguousarray(p[0])).to(psi.device)  # [input, output]
        live = torch.from_numpy(1 - p[1].astype(np.int64)).to(psi.device).bool()
        rest = [w for w in range(n) if w not in wires]
        m = v.permute(wires + rest).reshape(1 << len(wires), -1)
        new = torch.where(live[:, None], (block.T * live[None, :]) @ m, m)
        back = [0] * n
        for i, w in enumerate(wires + rest):
            back[w] = i
        return new.view((2,) * n).permute(back).reshape(-1)
    if name == "Swap":
        return v.transpose(t, ctl[0]).reshape(-1)
    sel = [slice(None)] * n
    for c in ctl:
        sel[c] = 1
    s0, s1 = list(sel), list(sel)
    s0[t], s1[t] = 0, 1
    s0, s1 = tuple(s0), tuple(s1)
    if name in ("CNot", "Toffoli"):
        a = v[s0].clone()
        v[s0] = v[s1]
        v[s1] = a
        return v.view(-1)
    if name == "CRk":
        ph = TWO_PI / 2.0 ** k
        v[s1] *= complex(math.cos(ph), math.sin(ph))
        return v.view(-1)
    m = _matrix(name, p)
    if inverse:
        m = tuple(complex(x).conjugate() for x in (m[0], m[2], m[1], m[3]))
    a, b = v[s0].clone(), v[s1].clone()
    v[s0] = m[0] * a + m[1] * b
    v[s1] = m[2] * a + m[3] * b
    return v.view(-1)


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128,
                      device="cuda" if torch.cuda.is_available() else "cpu")
    psi[0] = 1.0
    return psi


def _state(gates, n):
    psi = _zero(n)
    for g in gates:
        psi = _apply_exact(psi, n, g)
    return psi


def _hamiltonian(psi, n, a, b):
    """(sum_i a_i Z_i Z_{i+1} + b_i X_i) psi over the wires, periodic."""
    x = torch.arange(1 << n, device=psi.device)
    out = torch.zeros_like(psi)
    for i in range(n):
        bits = (x >> (n - 1 - i)) ^ (x >> (n - 1 - (i + 1) % n))
        out += float(a[i]) * (1 - 2 * (bits & 1)).double() * psi
        out += float(b[i]) * psi.view((2,) * n).flip(i).reshape(-1)
    return out


_PAULI = {"Rx": ("X", 1.0), "Ry": ("Y", 1.0), "Rz": ("Z", 1.0), "Phase": (None, -1.0)}


def _gradient_exact(gates, n, a, b):
    phi = _state(gates, n)
    lam = _hamiltonian(phi, n, a, b)
    e = torch.vdot(phi, lam).real.item()
    grad = np.zeros(len(gates))
    for i in range(len(gates) - 1, -1, -1):
        name, t = gates[i][0], gates[i][1]
        if name in _PAULI:
            pauli, sign = _PAULI[name]
            w = _apply_exact(phi, n, (pauli, t, (), 0.0, 0)) if pauli else phi
            grad[i] = sign * torch.vdot(lam, w).imag.item()
        phi = _apply_exact(phi, n, gates[i], True)
        lam = _apply_exact(lam, n, gates[i], True)
    return e, grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        return _state(_circuit(case, seed)[0], case["n"]).cpu().numpy(), None, None
    if kind == "batch":
        items = _batch_items(case, seed)
        if sum(len(g) for _, g, _, _ in items) > 25000:
            return None
        both = [_gradient_exact(g, n, a, b) for n, g, a, b in items]
        return np.array([e for e, _ in both]), np.concatenate([g for _, g in both])
    if kind == "custom":
        psi = _state(_custom_gates(case, seed), case["n"])
        p = psi.real ** 2 + psi.imag ** 2
        return None, None, None, _padded(psi[p >= 1e-6].cpu().numpy(), _survivors(case["n"]),
                                         np.complex128)
    n, r = case["n"], _rng(case, seed)
    if n > 26:
        return None
    gates = _gates(case, r)
    a, b = _observable(r, n)
    if kind == "gradient":
        return _gradient_exact(gates, n, a, b)
    psi = _state(gates, n)
    if kind == "apply":
        return psi.cpu().numpy()
    norm = torch.linalg.vector_norm(psi).item() ** 2
    if kind == "sample":
        return norm, None, None
    return np.array([torch.vdot(psi, _hamiltonian(psi, n, a, b)).real.item(), norm])
