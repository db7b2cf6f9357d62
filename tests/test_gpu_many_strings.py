"""Hamiltonian sweeps around 512 strings, the most whose tables a sweep keeps in shared memory: below and above one tile,
real and imaginary strings, and in a Pauli frame."""
import numpy as np
import pytest

from tests.test_gpu_hamiltonian import _apply

pytestmark = pytest.mark.gpu


def _strings(n, count, parts, rng):
    """`count` different strings over `parts` X parts within the lowest bits (one sweep)."""
    xs = rng.choice(1 << min(n, 8), parts, replace=False)
    seen = set()
    while len(seen) < count:
        x, z = int(xs[len(seen) % parts]), int(rng.integers(1 << n))
        seen.add("".join("IZXY"[(z >> q & 1) | (x >> q & 1) << 1] for q in range(n)))
    return sorted(seen)


@pytest.mark.parametrize("n,count,parts", [(10, 512, 3), (10, 513, 3), (10, 2000, 9), (12, 513, 1), (14, 511, 5), (14, 513, 5),
                                           (14, 3000, 7), (17, 700, 40)])
def test_pauli_sum(n, count, parts):
    from invariantq_b200.binding import NativeStateVector
    rng = np.random.default_rng(count + n)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a /= np.linalg.norm(a)
    strings = _strings(n, count, parts, rng)
    c = rng.normal(size=count)
    want = sum(ck * np.vdot(a, _apply(a, s)) for ck, s in zip(c, strings))
    sv = NativeStateVector(n)
    sv.set_amplitudes(a)
    # a sum of `count` coefficients per amplitude, one after the other: at most count * eps / 2 of their sum
    assert abs(sv.expval_pauli_sum(c, strings) - want) <= (64 + count) * 2.0**-52 * np.abs(c).sum()


@pytest.mark.parametrize("n,count", [(13, 513), (14, 900)])
def test_gradient_in_a_frame(n, count):
    """The gradient is linear in H: 513 and more strings at once against the sum over parts of at most 300."""
    from invariantq_b200.gradients import Ansatz, PauliHamiltonian, adjoint_gradient
    rng = np.random.default_rng(n)
    strings = _strings(n, count, 6, rng)
    c = rng.normal(size=count)
    a = Ansatz.hardware_efficient(n, 3)
    p = rng.uniform(0, 2 * np.pi, a.num_params)
    e, g = adjoint_gradient(a, PauliHamiltonian(n, c, strings), p)
    es, gs = 0.0, np.zeros_like(g)
    for k in range(0, count, 300):
        ek, gk = adjoint_gradient(a, PauliHamiltonian(n, c[k:k + 300], strings[k:k + 300]), p)
        es, gs = es + ek, gs + gk
    tol = (64 + count) * 2.0**-52 * np.abs(c).sum()
    assert abs(e - es) <= tol and np.abs(g - gs).max() <= 4 * tol
