"""Reduced-state spectra of every size of the fused tridiagonalisation (rows in shared memory up to 1024, in global
memory above): random states, states whose reduced matrix is diagonal or rank one (nothing to reflect in some columns)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _entropy(a, n, k):
    p = np.linalg.svd(a.reshape(1 << (n - k), 1 << k), compute_uv=False) ** 2
    p = p[p > 1e-14]
    return -(p * np.log2(p)).sum()


def _state(kind, n, rng):
    dim = 1 << n
    if kind == "random":
        a = rng.normal(size=dim) + 1j * rng.normal(size=dim)
    elif kind == "product":
        a = np.ones(1)
        for _ in range(n):
            a = np.kron(rng.normal(size=2) + 1j * rng.normal(size=2), a)
    elif kind == "ghz":
        a = np.zeros(dim, complex)
        a[0], a[-1] = 1, 1j
    else:   # a few basis states: a sparse reduced matrix
        a = np.zeros(dim, complex)
        a[rng.choice(dim, 40, replace=False)] = rng.normal(size=40) + 1j * rng.normal(size=40)
    return a / np.linalg.norm(a)


@pytest.mark.parametrize("kind", ["random", "product", "ghz", "sparse"])
@pytest.mark.parametrize("n,k", [(14, 7), (17, 8), (18, 9), (20, 10), (22, 11)])
def test_spectrum(kind, n, k):
    from invariantq_b200.binding import NativeStateVector
    if n == 22 and kind == "product":
        pytest.skip("the large size is covered by the other states")
    a = _state(kind, n, np.random.default_rng(n * 10 + k))
    sv = NativeStateVector(n)
    sv.set_amplitudes(a)
    want = _entropy(a, n, k)
    # eigenvalues to a few ulps of the largest, times -log2 p up to 47 for each of 2^k
    assert abs(sv.von_neumann_entropy(list(range(k))) - want) <= 1e-9
