"""Pauli sums through the Hamiltonian sweeps (iq_ham.cu) against dense numpy sums: arrays below, at and above one tile
of 2^12 amplitudes, strings inside one sweep's bits, across sweeps and wider than a tile, more distinct X parts than
one call of the kernel takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _apply(amps, s):
    n = len(s)
    idx = np.arange(1 << n)
    xm = sum(1 << q for q, c in enumerate(s) if c in "XY")
    out = amps[idx ^ xm].astype(np.complex128)
    for q, c in enumerate(s):
        bit = (idx >> q) & 1
        if c == "Z":
            out = out * (1 - 2 * bit)
        elif c == "Y":     # <bit|Y|1 - bit> = -i for bit 0, i for bit 1
            out = out * np.where(bit == 1, 1j, -1j)
    return out


def _strings(n, rng):
    out = ["".join("Z" if q in (i, i + 1) else "I" for q in range(n)) for i in range(n - 1)]
    out += ["".join("X" if q == i else "I" for q in range(n)) for i in range(n)]
    out += ["".join("Y" if q in (i, (i + 5) % n) else "I" for q in range(n)) for i in range(0, n, 3)]
    out += ["I" * n, "X" * n, "Y" * n]
    out += ["".join(rng.choice(list("IXYZ"), n)) for _ in range(80 if n == 14 else 6)]
    return out


@pytest.mark.parametrize("n", [1, 3, 8, 11, 12, 13, 14, 18, 21])
def test_pauli_sum(n):
    from invariantq_b200.binding import NativeStateVector
    rng = np.random.default_rng(n)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a /= np.linalg.norm(a)
    strings = _strings(n, rng)
    c = rng.normal(size=len(strings))
    want = sum(ck * np.vdot(a, _apply(a, s)) for ck, s in zip(c, strings))
    sv = NativeStateVector(n)
    sv.set_amplitudes(a)
    got = sv.expval_pauli_sum(c, strings)
    # each <P> is a sum of 2^n products of total magnitude <= 1, summed in a tree: well under 64 eps each
    assert abs(got - want) <= 64 * 2.0**-52 * np.abs(c).sum()


@pytest.mark.parametrize("n", [3, 11, 13, 14, 17, 21])
def test_lambda_through_gradients(n):
    """lambda = H psi feeds every gradient: adjoint gradients of a random Hamiltonian against the parameter shift."""
    from invariantq_b200.gradients import Ansatz, PauliHamiltonian, adjoint_gradient, adjoint_gradient_c64, ansatz_energies
    rng = np.random.default_rng(100 + n)
    strings = [s for s in _strings(n, rng)][:50]
    c = rng.normal(size=len(strings))
    a = Ansatz.hardware_efficient(n, 2)
    h = PauliHamiltonian(n, c, strings)
    p = rng.uniform(0, 2 * np.pi, a.num_params)
    e, g = adjoint_gradient(a, h, p)
    picks = rng.choice(a.num_params, 3, replace=False)
    rows = [p] + [p + d * np.eye(a.num_params)[j] * np.pi / 2 for j in picks for d in (1, -1)]
    es = ansatz_energies(a, h, np.array(rows))
    tol = 1e-12 * np.abs(c).sum()
    assert abs(e - es[0]) <= tol
    assert np.abs(g[picks] - 0.5 * (es[1::2] - es[2::2])).max() <= tol
    if n >= 7:   # complex64 states round to 6e-8 a few times per pass
        e64, g64 = adjoint_gradient_c64(a, h, p)
        assert abs(e64 - e) <= 2e-5 * np.abs(c).sum() and np.abs(g64 - g).max() <= 2e-5 * np.abs(c).sum()
