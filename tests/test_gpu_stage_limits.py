"""Programs on arrays of 2^27 amplitudes and more: plans of at most 4, 5 and 8 stages a pass are compared and one of them
is taken; smaller arrays and an explicit limit keep theirs."""
import numpy as np
import pytest

from tests.test_gpu_handle_lifetime import _Array
from tests.test_scheduler_emulated import brickwall_ops

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(n, gates, limit):
    from invariantq_b200.binding import NativeStateVector
    sv = NativeStateVector(n)
    if limit:
        sv.set_option("max_stages", limit)
    with sv.record() as rec:
        for kind, qs, m in gates:
            sv.apply_1q(qs[0], m) if kind == "1q" else sv.apply_2q(qs[0], qs[1], m)
    info = rec.program.pass_info()
    rec.program.run(sv)
    sv.sync()
    state = torch.as_tensor(_Array(sv.device_ptr(), 1 << n), device="cuda").clone()
    torch.cuda.synchronize()
    sv.close()
    return info, state


@pytest.mark.parametrize("n,depth", [(26, 3), (27, 4)])
def test_choice(n, depth):
    gates = brickwall_ops(n, depth, 1)
    got, state = _run(n, gates, 0)
    plans = {}
    for limit in (8, 5, 4) if n >= 27 else (8,):
        plans[limit], other = _run(n, gates, limit)
        assert max(p["stages"] for p in plans[limit]) <= limit
        # ~150 gates, each a few eps of the norm (at most 1 in any amplitude)
        assert float((state - other).abs().max()) <= 1e-13
    assert got in plans.values()
