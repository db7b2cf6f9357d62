"""Handles leave their streams and buffers to later handles (iq_runtime.cu): results after reuse, several threads, sizes
around the kept small state (2^16 amplitudes) and around one and several readback chunks, and the release call."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(n, seed):
    from invariantq_b200.binding import NativeStateVector
    rng = np.random.default_rng(seed)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a /= np.linalg.norm(a)
    sv = NativeStateVector(n)
    assert sv.get_amplitudes()[0] == 1.0 and abs(sv.norm_squared() - 1.0) == 0.0   # a fresh state, whatever came before
    sv.set_amplitudes(a)
    assert np.array_equal(sv.get_amplitudes(), a)
    # |a|^2 with and without a fused multiply-add differ by an ulp
    assert np.abs(sv.get_probabilities() - np.abs(a) ** 2).max() <= 4 * 2.0**-52 * np.abs(a).max() ** 2
    sv.apply_1q(n - 1, np.array([[0, 1], [1, 0]]))
    assert np.array_equal(sv.get_amplitudes(), np.roll(a, 1 << (n - 1)))
    shots = sv.sample(500, 3)
    assert shots.max() < 1 << n
    v, c = sv.sample_counts(500, 3)
    assert np.array_equal(np.repeat(v, c.astype(int)), np.sort(shots))
    sv.close()


@pytest.mark.parametrize("n", [1, 5, 16, 17, 18, 19, 21])
def test_reuse(n):
    from invariantq_b200 import _lib
    for k in range(3):
        _check(n, 10 * n + k)
    _lib.load().iq_adjoint_release()
    _check(n, n)


def test_threads():
    errs = []

    def work(t):
        try:
            for k in range(6):
                _check(3 + (5 * t + k) % 15, 100 * t + k)
        except BaseException as e:   # noqa: B902
            errs.append(e)
    ts = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs
