"""A handle's memory and the streams of others: a state whose address was given out stays as it is until the work that
reads it is done, although the handle is gone and new handles of its size are made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


class _Array:
    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": "<c16", "version": 3}


def _handles(kind):
    from invariantq_b200.binding import NativeDensityMatrix, NativeStateVector
    return NativeStateVector if kind == "sv" else NativeDensityMatrix


# index bits 2 to 16 live in the kept small buffer, 17 and 18 in memory of their own
@pytest.mark.parametrize("kind,n", [("sv", 2), ("sv", 12), ("sv", 16), ("sv", 17), ("dm", 1), ("dm", 8), ("dm", 9)])
def test_reader_on_another_stream(kind, n):
    make, count = _handles(kind), 1 << (n if kind == "sv" else 2 * n)
    x = np.array([[0, 1], [1, 0]], dtype=complex)
    h = make(n)
    if kind == "sv":
        h.apply_1q(0, x)
    else:
        h.apply_1q_unitary(0, x)
    want = torch.zeros(count, dtype=torch.complex128)
    want[1 if kind == "sv" else (1 << n) + 1] = 1.0
    view = torch.as_tensor(_Array(h.device_ptr(), count), device="cuda")
    h.sync() if kind == "sv" else h.trace()
    out = torch.empty(count, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)   # ~50 ms of a bounded wait before the reader
        out.copy_(view)
    h.close()
    later = [make(n) for _ in range(3)]   # every one resets its state
    for k in later:
        (k.sync if kind == "sv" else k.trace)()
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)
    for k in later:
        k.close()


# scratch of a call: what a live handle keeps is bounded, whatever the call took (2^20 shots fit the bound, 2^21 and 2^24 do not)
@pytest.mark.parametrize("shots", [1 << 20, 1 << 21, 1 << 24])
def test_kept_scratch_is_bounded(shots):
    from invariantq_b200.binding import NativeStateVector
    sv = NativeStateVector(12)
    for q in range(12):
        sv.apply_1q(q, np.array([[1, 1], [1, -1]]) / np.sqrt(2))
    sv.sample_counts(100, 1)
    sv.sample(100, 1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    values, counts = sv.sample_counts(shots, 5)
    outcomes = sv.sample(shots, 5)
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    v, c = np.unique(outcomes, return_counts=True)
    assert np.array_equal(values, v) and np.array_equal(counts, c)
    assert kept <= (64 << 20) + (4 << 20)   # the bound, and the allocator's granularity
    sv.close()
