"""Memory that earlier calls left for later ones (adjoint workspaces, freed handles' buffers) is given back when an
allocation would fail without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GIB = 1 << 30


@pytest.fixture
def ballast():
    """Fill the device up to `left` free bytes; freed after the test."""
    held = []

    def fill(left):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        assert free > left
        held.append(torch.empty(free - left, dtype=torch.uint8, device="cuda"))
        assert abs(torch.cuda.mem_get_info()[0] - left) < (64 << 20)
    from invariantq_b200 import gradients
    gradients.adjoint_release()
    torch.cuda.empty_cache()
    yield fill
    held.clear()
    torch.cuda.empty_cache()
    gradients.adjoint_release()


def _gradient(n, nsets=1, streams=1):
    from invariantq_b200.gradients import Ansatz, PauliHamiltonian, adjoint_gradient_batch
    a = Ansatz.hardware_efficient(n, 1)
    p = np.random.default_rng(n).uniform(0, 2 * np.pi, (nsets, a.num_params))
    return adjoint_gradient_batch([(a, PauliHamiltonian.tfim(n, 1.0), p)] * streams, num_streams=streams)


def test_state_takes_a_kept_workspace(ballast):
    from invariantq_b200.binding import NativeStateVector
    _gradient(27)                      # leaves a workspace of 4 GiB
    ballast(GIB)
    sv = NativeStateVector(27)         # 2 GiB
    assert abs(sv.norm_squared() - 1.0) == 0.0
    sv.close()


def test_gradient_takes_another_kept_workspace(ballast):
    want = _gradient(27)
    from invariantq_b200 import gradients
    gradients.adjoint_release()
    _gradient(26, streams=2)           # leaves two of 2 GiB
    ballast(GIB)
    got = _gradient(27)                # 4 GiB: its own workspace's 2, 1 free and the other's 2
    assert np.array_equal(got[0][0], want[0][0]) and np.array_equal(got[0][1], want[0][1])


def test_scratch_takes_a_kept_workspace(ballast):
    from invariantq_b200.binding import NativeStateVector
    sv = NativeStateVector(12)
    values, counts = sv.sample_counts(1 << 25, 3)
    _gradient(26)                      # leaves 2 GiB
    ballast(GIB // 4)
    v, c = sv.sample_counts(1 << 25, 3)   # scratch of more than 1 GiB
    assert np.array_equal(v, values) and np.array_equal(c, counts)
    sv.close()
