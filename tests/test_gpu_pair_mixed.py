"""Programs whose passes run partly in the pair pipeline, partly in three one-tile CTAs (tests/test_pair_rule.py)."""
import numpy as np
import pytest

from tests.test_gpu_pair import TOL
from tests.test_pair_rule import random_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers,dense", [(20, 8, False), (21, 5, False), (20, 4, True)])
def test_mixed_forms(n, layers, dense):
    from invariantq_b200.binding import NativeStateVector
    got = []
    for threads in (0, 128):
        sv = NativeStateVector(n)
        sv.set_option("jit", 2)
        if threads:
            sv.set_option("jit_threads", threads)
        with sv.record() as rec:
            for q, u in random_pairs(n, layers, n, dense):
                sv.apply_1q(q[0], u) if len(q) == 1 else sv.apply_2q(q[0], q[1], u)
        for _ in range(2):
            sv.reset()
            rec.program.run(sv)
        assert sv.stats()["jit_passes"] > 0
        got.append(sv.get_amplitudes())
        sv.close()
    assert abs(np.vdot(got[0], got[0]).real - 1) <= TOL
    assert np.abs(got[0] - got[1]).max() <= TOL
