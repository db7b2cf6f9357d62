"""The staged executor of small circuits (iq_resident.cu) against the tile passes: every qubit count on both sides of
its two stage widths, every gate kind, circuits longer than the planner's window, parameters used by several gates (one
stage holds each parameter once), fixed gates only, and sets of parameters that share one launch.

Tolerance: a gate adds at most 4 eps of the state's norm to psi and lambda, forward and back, and a parameter's
gradient sums one term bounded by 2 sum|c| per use, so both paths stay within 16 eps * gates * uses * sum|c| of the
exact value, and within twice that of each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ONE = ["rx", "ry", "rz", "p", "h", "x", "sx", "u3"]


def _circuit(rng, n, ngates, shared):
    gates, free = [], 0
    for i in range(ngates):
        k = rng.choice(ONE + (["cx", "cz"] * 4 if n > 1 else []))
        if k in ("cx", "cz"):
            a, b = rng.choice(n, 2, replace=False)
            gates.append((k, (int(a), int(b)), -1))
            continue
        width = {"u3": 3}.get(k, 0 if k in ("h", "x", "sx") else 1)
        p = -1
        if width:
            p = free
            if shared and free >= 6 and rng.random() < 0.5:
                p = int(rng.integers(0, free - width + 1))
            else:
                free += width
        gates.append((k, (int(rng.integers(n)),), p))
    return gates


@pytest.mark.parametrize("n", [1, 2, 3, 5, 7, 8, 10, 11, 12])
@pytest.mark.parametrize("ngates,shared", [(12, False), (90, True), (700, False)])
def test_stages_match_tile_passes(monkeypatch, n, ngates, shared):
    from invariantq_b200 import gradients as G
    rng = np.random.default_rng(1000 * n + ngates)
    gates = _circuit(rng, n, ngates, shared)
    gates.append(("ry", (n - 1,), 0))
    a = G.Ansatz(n, gates)
    paulis = ["".join(rng.choice(list("IXYZ"), n)) for _ in range(6)] + ["Z" * n]
    coeffs = rng.normal(size=len(paulis))
    th = rng.uniform(-7, 7, (3, a.num_params))
    jobs = [(a, G.PauliHamiltonian(n, coeffs, paulis), th)]
    (e, g), = G.adjoint_gradient_batch(jobs)
    assert G.adjoint_stats()["resident_sets"] == 3
    monkeypatch.setenv("IQ_RESIDENT_MAX_QUBITS", "0")
    (e0, g0), = G.adjoint_gradient_batch(jobs)
    assert G.adjoint_stats()["resident_sets"] == 0
    uses = np.zeros(a.num_params)
    for k, _, p in gates:
        if p >= 0:
            uses[p:p + (3 if k == "u3" else 1)] += 1
    tol = 32 * np.finfo(float).eps * (3 * ngates + 1) * np.abs(coeffs).sum()   # a U3 is three rotations
    assert np.max(np.abs(e - e0)) < tol
    assert np.all(np.abs(g - g0) < tol * np.maximum(uses, 1))


def test_fixed_gates_only():
    from invariantq_b200 import gradients as G
    a = G.Ansatz(3, [("h", (0,), -1), ("cx", (0, 1), -1), ("cx", (1, 2), -1), ("ry", (0,), 0)])
    h = G.PauliHamiltonian(3, [1.0, 0.5], ["ZZI", "XXX"])
    e, g = G.adjoint_gradient(a, h, np.zeros(1))
    assert abs(e - 1.5) < 1e-12 and abs(g[0]) < 1e-12
