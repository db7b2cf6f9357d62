"""Which passes run in the pair pipeline: not the light ones whose tiles move in 64 copies."""
import ctypes

import numpy as np
import pytest

from tests.test_steady_phases import shipped  # noqa: F401  (fixture)

CX = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], complex)


def random_pairs(n, layers, seed, dense=False):
    """Layers of one-qubit gates and CX (dense: two-qubit unitaries) on pairs of a random permutation."""
    rng = np.random.default_rng(seed)

    def unitary(d):
        q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
        return q * (np.diag(r) / np.abs(np.diag(r)))

    ops = []
    for _ in range(layers):
        if not dense:
            ops += [([q], unitary(2)) for q in range(n)]
        p = [int(x) for x in rng.permutation(n)]
        ops += [([p[2 * i], p[2 * i + 1]], unitary(4) if dense else CX) for i in range(n // 2)]
    return ops


def forms(lib, n, ops):
    ks = np.array([len(q) for q, _ in ops], np.int32)
    qs, offs, flat = np.full((len(ops), 5), -1, np.int32), np.zeros(len(ops), np.int64), []
    for i, (q, u) in enumerate(ops):
        qs[i, :len(q)] = q[::-1]
        offs[i] = sum(x.size for x in flat)
        flat.append(np.asarray(u, complex).reshape(-1))
    pool, boxes, pair = np.concatenate(flat), np.zeros(512, np.int32), np.zeros(512, np.int32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)   # noqa: E731
    k = lib.shipped_forms(n, len(ops), p(ks), p(qs), p(pool), p(offs), p(boxes), p(pair), 512)
    assert k > 0
    return boxes[:k], pair[:k]


@pytest.mark.parametrize("n", [24, 28])
def test_light_passes_of_many_copies(shipped, n):  # noqa: F811
    boxes, pair = forms(shipped, n, random_pairs(n, 8, n))
    assert (boxes == 6).any() and (boxes < 6).any()
    assert pair[boxes < 6].all() and not pair[boxes == 6].all()


def test_heavy_passes_stay_in_pairs(shipped):  # noqa: F811
    boxes, pair = forms(shipped, 28, random_pairs(28, 6, 3, dense=True))
    heavy = boxes[1:-1] == 6
    assert heavy.any() and pair[1:-1][heavy].any()
