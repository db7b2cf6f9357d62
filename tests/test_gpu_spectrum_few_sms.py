"""The fused tridiagonalisation with fewer SMs than its shared-memory rows need (a MIG slice): rows in global memory."""
import pytest

from tests.test_gpu_spectrum import _entropy, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "ghz", "sparse"])
@pytest.mark.parametrize("n,k,sms", [(14, 7, 15), (14, 7, 1), (17, 8, 31), (17, 8, 5), (18, 9, 63), (20, 10, 127)])
def test_spectrum(kind, n, k, sms, monkeypatch):
    import numpy as np

    from invariantq_b200.binding import NativeStateVector
    monkeypatch.setenv("IQ_ENTROPY_SMS", str(sms))
    a = _state(kind, n, np.random.default_rng(n * 10 + k))
    sv = NativeStateVector(n)
    sv.set_amplitudes(a)
    # eigenvalues to a few ulps of the largest, times -log2 p up to 47 for each of 2^k
    assert abs(sv.von_neumann_entropy(list(range(k))) - _entropy(a, n, k)) <= 1e-9
