"""The work that programs built on this package have it do, as cases to measure.

A case is a dict of plain values; ``kind`` names the entry points it goes through:

* ``run``       -- ``StateVectorSimulator.run``: a whole small circuit from the IR to amplitudes, probabilities,
                   entanglement entropy and measured counts (what a script or a notebook calls);
* ``circuit``   -- the same results of a larger circuit through the C-ABI binding, with a handle of its own (what the
                   reference's state-vector backend does with the library);
* ``gates``     -- the C-ABI binding: a kept handle, one call per gate with host matrices, then <Z_q> (the drop-in path);
* ``program``   -- a recorded circuit replayed on a kept state vector (the planned path, up to the 16 GiB state);
* ``density``   -- ``DensityMatrixSimulator.run`` of a noisy circuit;
* ``channel``   -- a recorded noisy circuit replayed on a kept density matrix, then trace, purity and diagonal;
* ``train``     -- one training step of a variational circuit: energy forward, adjoint gradient backward through autograd;
* ``gradient``  -- one adjoint gradient of a large circuit, complex128 states;
* ``gradient64``-- the same with complex64 states (results to single precision, which is what the states hold);
* ``batch``     -- gradients of many circuits of uneven size and several parameter sets in one call;
* ``readout``   -- measurements of a state in hand: Hamiltonian expectation, <Z_q>, sampled counts.

Circuits are U3 + CX brick-walls and RY/RZ + CZ-ring ansatzes with angles uniform on [0, 2 pi) and the transverse-field
Ising Hamiltonian, as in the package's benchmark and tests; ``prepare`` draws the angles from its seed.
"""
import math
import random

import numpy as np
import torch

from invariantq_b200.binding import NativeDensityMatrix, NativeStateVector
from invariantq_b200.channels import build_kraus_channel
from invariantq_b200.circuits import brickwall, noisy_brickwall, tfim_terms
from invariantq_b200.gradients import (Ansatz, PauliHamiltonian, adjoint_gradient, adjoint_gradient_batch,
                                       adjoint_gradient_c64, expectation)
from invariantq_b200.ir import op_kind
from invariantq_b200.simulator import DensityMatrixSimulator, StateVectorSimulator

DEPOLARIZING = 1e-3   # after every one-qubit gate of the noisy circuits


def listed():
    return [
        # the smallest whole call: a notebook-size circuit, where handle set-up, launches and host work are everything
        {"name": "run_5q", "kind": "run", "qubits": 5, "depth": 4, "shots": 1024},
        # gate-by-gate use of the binding on a mid-size state: one call per gate, a handful of tile passes
        {"name": "gates_17q", "kind": "gates", "qubits": 17, "depth": 20},
        # the headline state: 30 qubits (16 GiB), a planned brick-wall replayed
        {"name": "program_30q", "kind": "program", "qubits": 30, "depth": 20},
        # a small noisy circuit through the density-matrix driver
        {"name": "density_5q", "kind": "density", "qubits": 5, "depth": 4, "shots": 1024},
        # a large density matrix (1 GiB) under gates and channels; an odd qubit count
        {"name": "channel_13q", "kind": "channel", "qubits": 13, "depth": 6},
        # one step of a small variational loop: latency of a gradient
        {"name": "train_8q", "kind": "train", "qubits": 8, "layers": 4},
        # one step of an ordinary variational loop
        {"name": "train_20q", "kind": "train", "qubits": 20, "layers": 8},
        # a gradient whose two state-sized buffers (8 GiB) are far beyond the caches
        {"name": "gradient_28q", "kind": "gradient", "qubits": 28, "layers": 6},
        # the half-memory variant, odd qubit count
        {"name": "gradient64_25q", "kind": "gradient64", "qubits": 25, "layers": 6},
        # many circuits of uneven size (8 to 18 qubits) with 16 parameter sets each: the batched workload
        {"name": "batch_24", "kind": "batch", "circuits": 24, "least": 8, "most": 18, "sets": 16, "shape": 5},
        # measuring a state of 1 GiB: TFIM energy (51 Pauli strings), <Z_q> for every qubit, shots
        {"name": "readout_26q", "kind": "readout", "qubits": 26, "shots": 4096},
        # the benchmark's ordinary circuit: 20 qubits, depth 20, amplitudes, probabilities, <Z_q>, half-cut entropy, 8192 shots
        {"name": "circuit_20q", "kind": "circuit", "qubits": 20, "depth": 20, "shots": 8192},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["run", "circuit", "gates", "program", "density", "channel", "train", "gradient", "gradient64", "batch", "readout"])
    if kind == "run":
        return {"kind": kind, "qubits": rng.randint(2, 14), "depth": _log(rng, 1, 24), "shots": _log(rng, 100, 20000)}
    if kind == "circuit":
        return {"kind": kind, "qubits": rng.randint(8, 23), "depth": _log(rng, 1, 24), "shots": _log(rng, 100, 20000)}
    if kind == "gates":
        n = rng.randint(4, 25)
        return {"kind": kind, "qubits": n, "depth": _log(rng, 1, 24 if n < 24 else 12)}
    if kind == "program":
        n = rng.randint(12, 30)
        return {"kind": kind, "qubits": n, "depth": _log(rng, 2, 24 if n < 29 else 12)}
    if kind == "density":
        return {"kind": kind, "qubits": rng.randint(2, 7), "depth": _log(rng, 1, 10), "shots": _log(rng, 100, 20000)}
    if kind == "channel":
        n = rng.randint(6, 13)
        return {"kind": kind, "qubits": n, "depth": _log(rng, 1, 12 if n < 13 else 5)}
    if kind == "train":
        return {"kind": kind, "qubits": rng.randint(3, 22), "layers": _log(rng, 1, 10)}
    if kind in ("gradient", "gradient64"):
        n = rng.randint(13, 28)
        return {"kind": kind, "qubits": n, "layers": _log(rng, 1, 8 if n < 27 else 5)}
    if kind == "batch":
        lo = rng.randint(4, 12)
        return {"kind": kind, "circuits": _log(rng, 4, 24), "least": lo, "most": lo + rng.randint(0, 7),
                "sets": _log(rng, 1, 16), "shape": rng.randint(0, 999)}
    return {"kind": kind, "qubits": rng.randint(12, 28), "shots": _log(rng, 100, 100000)}


# ------------------------------------------------------------------ the framework's side

class _Array:
    def __init__(self, handle, count):
        self.handle = handle   # the tensor holds this object, and so the handle that owns its memory
        self.__cuda_array_interface__ = {"data": (handle.device_ptr(), False), "shape": (count,), "typestr": "<c16",
                                         "version": 3}


def _device_view(handle, count):
    """The handle's amplitudes as a torch tensor (no copy)."""
    return torch.as_tensor(_Array(handle, count), device="cuda")


def _angles(count, seed):
    return np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi, count)


def _noise():
    return {"u3": build_kraus_channel("depolarizing", [DEPOLARIZING])}


def _issue(dm, circuit, noise):
    """The driver's calls for a noisy circuit, on a handle the program keeps."""
    for op in circuit.ops:
        q = [circuit.get_qubit_index(w) for w in op.qubits]
        if op_kind(op) == "NoiseOp":
            kraus = build_kraus_channel(op.channel_name, op.params)
            for w in q:
                dm.apply_1q_kraus(w, kraus)
        elif len(q) == 1:
            dm.apply_1q_unitary(q[0], op.matrix)
            if op.name in noise:
                dm.apply_1q_kraus(q[0], noise[op.name])
        else:
            dm.apply_2q_unitary(q[0], q[1], op.matrix)


def _batch_circuits(case):
    r = random.Random(1000 + case["shape"])
    return [(r.randint(case["least"], case["most"]), r.randint(2, 6)) for _ in range(case["circuits"])]


def prepare(case, seed):
    kind, n = case["kind"], case.get("qubits")
    s = {"kind": kind, "case": case}
    if kind == "run":
        s["circuit"] = brickwall(n, case["depth"], seed)
        s["sim"] = StateVectorSimulator()
    elif kind in ("gates", "circuit"):
        c = brickwall(n, case["depth"], seed)
        s["gates"] = [([c.get_qubit_index(q) for q in op.qubits], op.matrix) for op in c.ops]
        if kind == "gates":
            s["sv"] = NativeStateVector(n)
    elif kind == "program":
        c = brickwall(n, case["depth"], seed)
        sv = s["sv"] = NativeStateVector(n)
        with sv.record() as rec:
            for op in c.ops:
                q = [c.get_qubit_index(w) for w in op.qubits]
                (sv.apply_1q(q[0], op.matrix) if len(q) == 1 else sv.apply_2q(q[0], q[1], op.matrix))
        s["program"] = rec.program
    elif kind == "density":
        s["circuit"] = noisy_brickwall(n, case["depth"], seed)
        s["sim"] = DensityMatrixSimulator(noise_model=_noise())
    elif kind == "channel":
        c = noisy_brickwall(n, case["depth"], seed)
        dm = s["dm"] = NativeDensityMatrix(n)
        with dm.record() as rec:
            _issue(dm, c, _noise())
        s["program"] = rec.program
    elif kind == "batch":
        r = np.random.default_rng(seed)
        s["jobs"] = []
        for q, layers in _batch_circuits(case):
            a = Ansatz.hardware_efficient(q, layers)
            s["jobs"].append((a, PauliHamiltonian.tfim(q, 1.0), r.uniform(0.0, 2.0 * math.pi, (case["sets"], a.num_params))))
    elif kind == "readout":
        sv = s["sv"] = NativeStateVector(n)
        sv.sync()   # the handle's own stream is done with the array before torch writes to it
        v = _device_view(sv, 1 << n)
        g = torch.Generator(device="cuda").manual_seed(seed)
        v.copy_(torch.randn(1 << n, dtype=torch.complex128, device="cuda", generator=g))
        v /= torch.linalg.vector_norm(v)
        torch.cuda.synchronize()
        s["terms"] = tfim_terms(n, 1.0)
    else:
        s["ansatz"] = Ansatz.hardware_efficient(n, case["layers"])
        s["ham"] = PauliHamiltonian.tfim(n, 1.0 if kind == "train" else 0.7)
        s["params"] = _angles(s["ansatz"].num_params, seed)
        if kind == "train":
            s["params"] = torch.tensor(s["params"], device="cuda", requires_grad=True)
    return s


def _issue_gates(sv, gates):
    for q, m in gates:
        if len(q) == 1:
            sv.apply_1q(q[0], m)
        else:
            sv.apply_2q(q[0], q[1], m)


def _tally(counts, shots):
    """Outcomes and counts of a counts dictionary, as two arrays of one length for every run."""
    out = np.full((2, shots), -1, np.int64)
    out[0, :len(counts)] = [int(k, 2) for k in counts]
    out[1, :len(counts)] = list(counts.values())
    return out


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "run":
        r = s["sim"].run(s["circuit"], shots=case["shots"], seed=7)
        return {"statevector": r.statevector, "entropy": float(r.entanglement_entropy), "counts": _tally(r.counts, case["shots"])}
    if kind == "circuit":
        sv, n = NativeStateVector(case["qubits"]), case["qubits"]
        _issue_gates(sv, s["gates"])
        out = {"state": sv.get_amplitudes(), "probabilities": sv.get_probabilities(), "z": sv.expval_z_all(),
               "entropy": float(sv.von_neumann_entropy(list(range(n // 2)))),
               "shots": sv.sample(case["shots"], 7).astype(np.int64)}
        sv.close()
        return out
    if kind == "gates":
        sv = s["sv"]
        sv.reset()
        _issue_gates(sv, s["gates"])
        return {"z": sv.expval_z_all(), "state": _device_view(sv, sv.dim)}
    if kind == "program":
        sv = s["sv"]
        sv.reset()
        s["program"].run(sv)
        return {"z": sv.expval_z_all(), "state": _device_view(sv, sv.dim)}
    if kind == "density":
        r = s["sim"].run(s["circuit"], shots=case["shots"], seed=7)
        return {"matrix": r.density_matrix, "entropy": float(r.entanglement_entropy), "trace": float(r.metadata["trace"]),
                "purity": float(r.metadata["purity"]), "counts": _tally(r.counts, case["shots"])}
    if kind == "channel":
        dm = s["dm"]
        dm.reset()
        s["program"].run(dm)
        return {"trace": dm.trace(), "purity": dm.purity(), "diagonal": dm.get_diagonal(),
                "matrix": _device_view(dm, dm.dim * dm.dim)}
    if kind == "train":
        p = s["params"]
        p.grad = None
        e = expectation(p, s["ansatz"], s["ham"])
        e.backward()
        return {"energy": e.detach(), "grad": p.grad}
    if kind == "gradient":
        e, g = adjoint_gradient(s["ansatz"], s["ham"], s["params"])
        return {"energy": e, "grad": g}
    if kind == "gradient64":
        e, g = adjoint_gradient_c64(s["ansatz"], s["ham"], s["params"])
        return {"energy": np.float32(e), "grad": g.astype(np.float32)}
    if kind == "batch":
        out = adjoint_gradient_batch(s["jobs"])
        return {"energies": np.concatenate([e for e, _ in out]), "grads": np.concatenate([g.reshape(-1) for _, g in out])}
    sv, (coeffs, paulis) = s["sv"], s["terms"]
    vals, cnts = sv.sample_counts(case["shots"], 7)
    tally = np.full((2, case["shots"]), -1, np.int64)
    tally[0, :len(vals)], tally[1, :len(vals)] = vals, cnts
    return {"energy": sv.expval_pauli_sum(coeffs, paulis).real, "z": sv.expval_z_all(), "counts": tally}


def work(case):
    """Inputs and outputs once; arithmetic: 14 per amplitude for a dense one-qubit gate, 6 for a rotation or a phase, 6
    per entry of a density matrix and channel, 4 for one gradient term or Hamiltonian string."""
    kind, n = case["kind"], case.get("qubits", 0)
    dim = float(1 << n)
    if kind in ("run", "circuit", "gates", "program"):
        out = (24.0 if kind in ("run", "circuit") else 16.0) * dim
        return {"bytes": out + 64.0 * n * case["depth"], "flops": 14.0 * dim * n * case["depth"]}
    if kind in ("density", "channel"):
        d = case["depth"]
        return {"bytes": 16.0 * dim * dim, "flops": dim * dim * d * (n * (28.0 + 2 * 6.0) + (n // 2) * 4 * 6.0)}
    if kind == "readout":
        return {"bytes": 16.0 * dim, "flops": dim * (4.0 * (2 * n - 1) + n)}

    def one(q, layers):
        return (1 << q) * (2.0 * q * layers * (6 + 12 + 4) + 4.0 * (2 * q - 1))
    if kind == "batch":
        cs = _batch_circuits(case)
        return {"bytes": 16.0 * case["sets"] * sum(2 * q * k + 1 for q, k in cs),
                "flops": case["sets"] * sum(one(q, k) for q, k in cs)}
    return {"bytes": 16.0 * (2 * n * case["layers"] + 1), "flops": one(n, case["layers"])}


# ------------------------------------------------------------------ the same in plain torch, 64 bits

def _u3(th, ph, lam):
    c, s = math.cos(th / 2), math.sin(th / 2)
    e = lambda x: complex(math.cos(x), math.sin(x))   # noqa: E731
    return [[c, -e(lam) * s], [e(ph) * s, e(ph + lam) * c]]


def _apply1(v, q, m):
    """2x2 m on index bit q of the flat vector v."""
    x = v.view(-1, 2, 1 << q)
    a, b = x[:, 0], x[:, 1]
    return torch.stack((m[0][0] * a + m[0][1] * b, m[1][0] * a + m[1][1] * b), 1).view(-1)


def _cx(v, c, t):
    """Control bit c, target bit t."""
    hi, lo = max(c, t), min(c, t)
    x = v.clone().view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    if c == hi:
        x[:, 1] = x[:, 1].flip(2)
    else:
        x[:, :, :, 1] = x[:, :, :, 1].flip(1)
    return x.view(-1)


def _cz_(v, a, b):
    hi, lo = max(a, b), min(a, b)
    v.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)[:, 1, :, 1] *= -1
    return v


def _zero(n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    v[0] = 1.0
    return v


def _brickwall_state(n, depth, seed):
    ang = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, size=(depth, n, 3))
    v = _zero(n)
    for layer in range(depth):
        for q in range(n):
            v = _apply1(v, q, _u3(*(float(a) for a in ang[layer, q])))
        for q in range(layer % 2, n - 1, 2):
            v = _cx(v, q, q + 1)
    return v


def _z_all(v, n):
    p = v.real.square() + v.imag.square()
    return torch.stack([(p.view(-1, 2, 1 << q)[:, 0].sum() - p.view(-1, 2, 1 << q)[:, 1].sum()) for q in range(n)])


def _entropy_of(p):
    p = p[p > 1e-14]
    return float(-(p * torch.log2(p)).sum())


def _tfim(v, n, h):
    """H v for H = -sum Z_i Z_{i+1} - h sum X_i, for every row of v."""
    idx = torch.arange(1 << n, device="cuda")
    diag = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for i in range(n - 1):
        diag -= 1.0 - 2.0 * (((idx >> i) ^ (idx >> (i + 1))) & 1)
    out = diag * v
    for q in range(n):
        out -= h * v.view(-1, 2, 1 << q).flip(1).reshape(v.shape)
    return out


def _energies_and_gradients(n, layers, params, h):
    """Adjoint gradients of the RY/RZ + CZ-ring ansatz: one row of params, one state."""
    ring = [(q, (q + 1) % n) for q in range(n if n > 2 else 1)]
    p = torch.as_tensor(np.asarray(params), device="cuda").view(-1, layers, 2, n)
    sets = p.shape[0]
    c, s = torch.cos(p / 2)[..., None, None], torch.sin(p / 2)[..., None, None]

    def ry(v, k, q, sign=1.0):
        x = v.view(sets, -1, 2, 1 << q)
        a, b, cq, sq = x[:, :, 0], x[:, :, 1], c[:, k, 0, q], sign * s[:, k, 0, q]
        return torch.stack((cq * a - sq * b, sq * a + cq * b), 2).view(sets, -1)

    def rz(v, k, q, sign=1.0):
        x, ph = v.view(sets, -1, 2, 1 << q), torch.complex(c[:, k, 1, q], sign * s[:, k, 1, q])
        return torch.stack((ph.conj() * x[:, :, 0], ph * x[:, :, 1]), 2).view(sets, -1)

    v = torch.zeros(sets, 1 << n, dtype=torch.complex128, device="cuda")
    v[:, 0] = 1.0
    for k in range(layers):
        for q in range(n):
            v = ry(v, k, q)
        for q in range(n):
            v = rz(v, k, q)
        for a, b in ring:
            v = _cz_(v, a, b)
    lam = _tfim(v, n, h)
    energies = torch.sum(lam.conj() * v, 1).real
    g = torch.zeros(sets, layers, 2, n, dtype=torch.float64, device="cuda")
    for k in reversed(range(layers)):
        for a, b in ring:
            v, lam = _cz_(v, a, b), _cz_(lam, a, b)
        for q in reversed(range(n)):
            x, y = v.view(sets, -1, 2, 1 << q), lam.view(sets, -1, 2, 1 << q)
            z = y.conj() * x
            g[:, k, 1, q] = (z[:, :, 0].sum((1, 2)) - z[:, :, 1].sum((1, 2))).imag
            v, lam = rz(v, k, q, -1.0), rz(lam, k, q, -1.0)
        for q in reversed(range(n)):
            x, y = v.view(sets, -1, 2, 1 << q), lam.view(sets, -1, 2, 1 << q)
            g[:, k, 0, q] = ((y[:, :, 1].conj() * x[:, :, 0]).sum((1, 2)) - (y[:, :, 0].conj() * x[:, :, 1]).sum((1, 2))).real
            v, lam = ry(v, k, q, -1.0), ry(lam, k, q, -1.0)
    return energies, g.view(sets, -1)


def _noisy_matrix(n, depth, seed):
    """rho of the noisy brick-wall, row-major: row bit of qubit q is n + q, column bit q."""
    ang = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, size=(depth, n, 3))
    r = torch.zeros(1 << (2 * n), dtype=torch.complex128, device="cuda")
    r[0] = 1.0
    conj = lambda m: [[complex(x).conjugate() for x in row] for row in m]   # noqa: E731

    def unitary(r, q, m):
        return _apply1(_apply1(r, n + q, m), q, conj(m))

    def channel(r, q, kraus):
        return sum(unitary(r, q, k) for k in kraus)
    d = DEPOLARIZING
    a, b = math.sqrt(1 - 0.75 * d), math.sqrt(d / 4)
    depol = [[[a, 0], [0, a]], [[0, b], [b, 0]], [[0, -1j * b], [1j * b, 0]], [[b, 0], [0, -b]]]
    amp = lambda g: [[[1, 0], [0, math.sqrt(1 - g)]], [[0, math.sqrt(g)], [0, 0]]]     # noqa: E731
    phase = lambda g: [[[1, 0], [0, math.sqrt(1 - g)]], [[0, 0], [0, math.sqrt(g)]]]   # noqa: E731
    t1, t2, tg = 100e-6, 80e-6, 50e-9
    gamma, lam = 1 - math.exp(-tg / t1), 1 - math.exp(-tg * (1 / t2 - 1 / (2 * t1)))
    for layer in range(depth):
        for q in range(n):
            r = channel(unitary(r, q, _u3(*(float(x) for x in ang[layer, q]))), q, depol)
        for q in range(layer % 2, n - 1, 2):
            r = _cx(_cx(r, n + q, n + q + 1), q, q + 1)
            for w in (q, q + 1):
                r = channel(r, w, amp(2e-3))
            for w in (q, q + 1):
                r = channel(r, w, phase(1e-3))
        for q in range(n):
            r = channel(channel(r, q, amp(gamma)), q, phase(lam))
    return r


def exact(case, seed):
    kind, n = case["kind"], case.get("qubits")
    if kind in ("run", "circuit", "gates", "program"):
        if n > 26:
            return None
        v = _brickwall_state(n, case["depth"], seed)
        if kind in ("gates", "program"):
            return {"z": _z_all(v, n), "state": v}
        entropy = _entropy_of(torch.linalg.svdvals(v.view(1 << (n - n // 2), 1 << (n // 2))).square())
        if kind == "run":
            return {"statevector": v.cpu().numpy(), "entropy": entropy, "counts": None}
        return {"state": v.cpu().numpy(), "probabilities": v.real.square() + v.imag.square(), "z": _z_all(v, n),
                "entropy": entropy, "shots": None}
    if kind in ("density", "channel"):
        m = _noisy_matrix(n, case["depth"], seed).view(1 << n, 1 << n)
        diag = torch.diagonal(m).real.clone()
        out = {"matrix": m if kind == "density" else m.reshape(-1), "trace": float(diag.sum()),
               "purity": float((m.real.square() + m.imag.square()).sum())}
        if kind == "channel":
            return {**out, "diagonal": diag}
        # above 6 qubits the driver reports the entropy of the diagonal, as the reference does
        w = torch.linalg.eigvalsh(m) if n <= 6 else diag.clamp(min=0.0)
        return {**out, "entropy": _entropy_of(w), "counts": None}
    if kind == "batch":
        r, es, gs = np.random.default_rng(seed), [], []
        for q, layers in _batch_circuits(case):
            e, g = _energies_and_gradients(q, layers, r.uniform(0.0, 2.0 * math.pi, (case["sets"], 2 * q * layers)), 1.0)
            es.append(e)
            gs.append(g.view(-1))
        return {"energies": torch.cat(es), "grads": torch.cat(gs)}
    if kind == "readout":
        g = torch.Generator(device="cuda").manual_seed(seed)
        v = torch.randn(1 << n, dtype=torch.complex128, device="cuda", generator=g)
        v /= torch.linalg.vector_norm(v)
        return {"energy": float(torch.vdot(v, _tfim(v, n, 1.0)).real), "z": _z_all(v, n), "counts": None}
    if n > 25:
        return None
    e, g = _energies_and_gradients(n, case["layers"], _angles(2 * n * case["layers"], seed)[None], 1.0 if kind == "train" else 0.7)
    return {"energy": e[0], "grad": g[0]}
