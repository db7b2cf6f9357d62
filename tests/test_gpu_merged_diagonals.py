"""Stages whose diagonals are merged (merge_stage_diagonals): circuits full of phases, CZ signs, permutations with phases
and lone diagonals, through the specialised kernels and the interpreting kernel on the same plan, against a dense numpy
simulation; gradients of ansatzes with several Z rotations per qubit against the parameter shift."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _gates(n, count, rng):
    s, t = np.diag([1, 1j]), np.diag([1, np.exp(0.25j * np.pi)])
    h = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
    x = np.array([[0, 1], [1, 0]], complex)
    cz = np.diag([1, 1, 1, -1]).astype(complex)
    cx = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], complex)
    swap = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], complex)
    iswap = np.array([[1, 0, 0, 0], [0, 0, 1j, 0], [0, 1j, 0, 0], [0, 0, 0, 1]], complex)
    for _ in range(count):
        a, b = (int(q) for q in rng.choice(n, 2, replace=False))
        if rng.random() < 0.6:
            th = rng.uniform(0, 2 * np.pi, 3)
            u3 = np.array([[np.cos(th[0] / 2), -np.exp(1j * th[2]) * np.sin(th[0] / 2)],
                           [np.exp(1j * th[1]) * np.sin(th[0] / 2), np.exp(1j * (th[1] + th[2])) * np.cos(th[0] / 2)]])
            yield (a,), [s, t, h, x, np.diag([1, np.exp(1j * th[0])]), u3, u3][rng.integers(7)]
        else:
            yield (a, b), [cz, cz, cx, swap, iswap, np.diag(np.exp(1j * rng.uniform(0, 6, 4)))][rng.integers(6)]


def _apply(v, n, qs, m):
    """first listed qubit = most significant bit of the local index"""
    ax = [n - 1 - q for q in qs]
    k = len(qs)
    w = np.tensordot(np.asarray(m, complex).reshape((2,) * 2 * k), v.reshape((2,) * n), axes=(range(k, 2 * k), ax))
    return np.moveaxis(w, range(k), ax).reshape(-1)


@pytest.mark.parametrize("n,slots", [(7, 4), (8, 3), (11, 4), (12, 3), (13, 4), (15, 4)])
def test_states(n, slots):
    from invariantq_b200.binding import NativeStateVector
    rng = np.random.default_rng(n * 10 + slots)
    gates = list(_gates(n, 160, rng))
    want = np.zeros(1 << n, complex)
    want[0] = 1
    for qs, m in gates:
        want = _apply(want, n, qs, m)
    got = []
    for jit in (2, 0):
        sv = NativeStateVector(n)
        sv.set_option("reg_slots", slots)
        sv.set_option("plan_style", 2)
        sv.set_option("tile_bits", 12)
        sv.set_option("chunk_bits", 4)
        sv.set_option("nbuf", 1)
        sv.set_option("jit", jit)
        for qs, m in gates:
            sv.apply_1q(qs[0], m) if len(qs) == 1 else sv.apply_2q(qs[0], qs[1], m)
        got.append(sv.get_amplitudes())
    assert np.abs(got[0] - want).max() <= TOL
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("n,sets", [(13, 1), (13, 3), (14, 2)])
def test_gradients(n, sets):
    from invariantq_b200.gradients import Ansatz, PauliHamiltonian, adjoint_gradient_batch, ansatz_energies
    rng = np.random.default_rng(n + sets)
    ops, p = [], 0
    for layer in range(2):
        for q in range(n):
            for g in ("rz", "rz", "ry", "p", "rx")[: 5 if q % 2 else 3]:
                ops.append((g, (q,), p))
                p += 1
        for q in range(n):
            ops.append((("cz", "cx")[layer], (q, (q + 1) % n), -1))
    for q in range(0, n, 3):
        ops += [("h", (q,), -1), ("rz", (q,), p), ("rz", (q,), p + 1)]
        p += 2
    a, h = Ansatz(n, ops), PauliHamiltonian.tfim(n, 0.8)
    params = rng.uniform(0, 2 * np.pi, (sets, p))
    (e, g), = adjoint_gradient_batch([(a, h, params)])
    for s in range(sets):
        picks = rng.choice(p, 6, replace=False)
        rows = [params[s]] + [params[s] + d * np.eye(p)[j] * np.pi / 2 for j in picks for d in (1, -1)]
        es = ansatz_energies(a, h, np.array(rows))
        assert abs(e[s] - es[0]) <= TOL * n
        assert np.abs(g[s, picks] - 0.5 * (es[1::2] - es[2::2])).max() <= TOL * n
