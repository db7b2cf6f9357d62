"""Pauli sums and lambda = H psi in both forms (tiles in shared memory; one amplitude per thread) at the sizes where they
differ: arrays smaller than a tile or a block, groups at the two ways to sum strings, more strings than are staged at once."""
import numpy as np
import pytest

from tests.test_gpu_hamiltonian import _apply

pytestmark = pytest.mark.gpu


def _strings(n, count, parts, rng):
    xs = rng.integers(0, 2, (parts, n))
    xs[0] = 0
    return ["".join("IZXY"[2 * x + z] for x, z in zip(xs[k % parts], rng.integers(0, 2, n))) for k in range(count)]


@pytest.mark.parametrize("gather", ["0", "1"])
@pytest.mark.parametrize("n,count,parts", [(1, 4, 2), (2, 9, 3), (5, 40, 7), (8, 45, 3), (11, 64, 64), (12, 48, 3), (12, 51, 3),
                                           (13, 15, 1), (13, 513, 30), (14, 300, 60), (15, 2048, 20), (15, 2049, 3),
                                           (16, 4500, 2), (19, 90, 30)])
def test_pauli_sum(monkeypatch, gather, n, count, parts):
    from invariantq_b200.binding import NativeStateVector
    monkeypatch.setenv("IQ_HAM_GATHER", gather)
    rng = np.random.default_rng(1000 * n + count)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a /= np.linalg.norm(a)
    strings = _strings(n, count, parts, rng)
    c = rng.normal(size=count)
    want = sum(ck * np.vdot(a, _apply(a, s)) for ck, s in zip(c, strings))
    sv = NativeStateVector(n)
    sv.set_amplitudes(a)
    # a sum of `count` coefficients per amplitude, one after the other: at most count * eps / 2 of their sum
    assert abs(sv.expval_pauli_sum(c, strings) - want) <= (64 + count) * 2.0**-52 * np.abs(c).sum()


@pytest.mark.parametrize("n,count,parts,sets", [(13, 60, 20, 1), (13, 60, 20, 3), (14, 700, 9, 1), (14, 2100, 40, 2), (19, 40, 12, 1)])
def test_gradients(monkeypatch, n, count, parts, sets):
    """Framed and unframed gradients, one and several sets: the forms against each other."""
    from invariantq_b200.gradients import Ansatz, PauliHamiltonian, adjoint_gradient_batch, adjoint_gradient_c64
    rng = np.random.default_rng(n + count)
    strings = _strings(n, count, parts, rng)
    c = rng.normal(size=count)
    a, h = Ansatz.hardware_efficient(n, 2), PauliHamiltonian(n, c, strings)
    p = rng.uniform(0, 2 * np.pi, (sets, a.num_params))
    out, out64 = [], []
    for gather in ("0", "1"):
        monkeypatch.setenv("IQ_HAM_GATHER", gather)
        out.append(adjoint_gradient_batch([(a, h, p)])[0])
        out64.append(adjoint_gradient_c64(a, h, p[0]))
    tol = (64 + count) * 2.0**-52 * np.abs(c).sum()
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= 4 * tol
    # lambda is rounded to float2 from sums that differ by `tol`: an ulp apart at most, and an ulp more at each of the
    # two dozen stage boundaries behind it
    for x, y in zip(*out64):
        assert np.abs(np.asarray(x) - np.asarray(y)).max() <= 4 * tol + 32 * 2.0**-23 * np.abs(c).sum()
