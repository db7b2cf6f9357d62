"""The pair pipeline (two groups of a CTA computing tiles in turn over three buffers) against the one-tile-per-CTA
kernels of the same plans: fewer tiles than SMs, one group idle, uneven shares per CTA, buffers used many times; states
and density matrices; a state that is replayed.  Both apply the same products in the same order of gates; a gate adds at
most 4 eps of the norm, so 1e-12 holds for a thousand of them."""
import numpy as np
import pytest

from tests.test_gpu_merged_diagonals import _gates

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("n", [12, 13, 14, 19, 20, 21, 23])
def test_states(n):
    from invariantq_b200.binding import NativeStateVector
    rng = np.random.default_rng(n)
    gates = list(_gates(n, 120, rng))
    got = []
    for threads in (0, 128):   # 0: the library's choice
        sv = NativeStateVector(n)
        sv.set_option("jit", 2)
        if threads:
            sv.set_option("jit_threads", threads)
        with sv.record() as rec:
            for qs, m in gates:
                sv.apply_1q(qs[0], m) if len(qs) == 1 else sv.apply_2q(qs[0], qs[1], m)
        for _ in range(3):
            sv.reset()
            rec.program.run(sv)
        assert sv.stats()["jit_passes"] > 0
        got.append(sv.get_amplitudes())
        sv.close()
    assert abs(np.vdot(got[0], got[0]).real - 1) <= TOL
    assert np.abs(got[0] - got[1]).max() <= TOL


@pytest.mark.parametrize("n", [6, 7, 10])
def test_density_matrices(n):
    from invariantq_b200.binding import NativeDensityMatrix
    from invariantq_b200.channels import build_kraus_channel
    rng = np.random.default_rng(100 + n)
    kraus = build_kraus_channel("depolarizing", [0.02])
    gates = list(_gates(n, 40, rng))
    got = []
    for threads in (0, 128):
        dm = NativeDensityMatrix(n)
        dm.set_option("jit", 2)
        if threads:
            dm.set_option("jit_threads", threads)
        for qs, m in gates:
            if len(qs) == 1:
                dm.apply_1q_unitary(qs[0], m)
                dm.apply_1q_kraus(qs[0], kraus)
            else:
                dm.apply_2q_unitary(qs[0], qs[1], m)
        got.append(dm.get_matrix())
        assert dm.stats()["jit_passes"] > 0
        dm.close()
    assert abs(np.trace(got[0]) - 1) <= TOL
    assert np.abs(got[0] - got[1]).max() <= TOL


def test_explicit_default_shape_is_the_default():
    """The autotuner sets every option: the default number of CTAs, set explicitly, runs the default kernels."""
    from invariantq_b200.binding import NativeStateVector
    gates = list(_gates(20, 60, np.random.default_rng(5)))
    got = []
    for ctas in (None, 3, 4):
        sv = NativeStateVector(20)
        sv.set_option("jit", 2)
        if ctas:
            sv.set_option("ctas_per_sm", ctas)
        for qs, m in gates:
            sv.apply_1q(qs[0], m) if len(qs) == 1 else sv.apply_2q(qs[0], qs[1], m)
        got.append(sv.get_amplitudes())
        sv.close()
    assert np.array_equal(got[0], got[1])
    assert np.abs(got[0] - got[2]).max() <= TOL
