"""Counts of sampled shots (count_outcomes) against the shots themselves: one launch up to 8192 shots, tiles and merges
above; few distinct outcomes (long runs) and nearly all distinct; the largest index value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shots", [1, 2, 3, 31, 1023, 1024, 1025, 8191, 8192, 8193, 16384, 16385, 100001])
@pytest.mark.parametrize("n", [1, 5, 18])
def test_counts(n, shots):
    from invariantq_b200.binding import NativeStateVector
    sv = NativeStateVector(n)
    for q in range(n):
        t = 0.4 + 0.13 * q
        sv.apply_1q(q, np.array([[np.cos(t), -np.sin(t)], [np.sin(t), np.cos(t)]]))
    s = sv.sample(shots, 11)
    v, c = sv.sample_counts(shots, 11)
    wv, wc = np.unique(s, return_counts=True)
    assert np.array_equal(v, wv) and np.array_equal(c, wc.astype(np.uint64))
