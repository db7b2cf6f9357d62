"""Rounding of what the host prepares for the kernels: merged diagonals, and the steady list of a circuit."""
import ctypes

import numpy as np
import pytest

from tests.test_steady_phases import shipped  # noqa: F401  (fixture)


# components of modulus at most 1, formed with 64 bits of mantissa and rounded once: half of 2^-53, and what 64-bit
# products of up to 24 factors add (24 * 2^-63 = 0.03 of 2^-53)
@pytest.mark.parametrize("count", [1, 2, 3, 8, 24])
def test_merged_entries_are_rounded_once(shipped, count):  # noqa: F811
    shipped.merged_entry_error.restype = ctypes.c_double
    for seed in range(4):
        assert shipped.merged_entry_error(count, seed) <= 0.54


# A gate's list holds five numbers rounded to 2^-53 of a modulus of about 1 (two phases, a ratio), 0.3 * 2^-53 rms each: ~2^-53
# a gate at most, so sqrt(gates) * 2^-53 for the state (the gates' own rounding is not counted: both sides start from
# them).  The squared norm is off by as much at most, with no preferred sign: its mean over 300 circuits stays within four
# standard errors of 0.
@pytest.mark.parametrize("n,depth", [(2, 2), (4, 4), (6, 12)])
def test_steady_list(shipped, n, depth):  # noqa: F811
    out, state, norm = (ctypes.c_double * 2)(), [], []
    for seed in range(300):
        shipped.host_rounding(n, depth, seed, out)
        state.append(out[0])
        norm.append(out[1])
    eps = 2.0 ** -53
    assert np.sqrt(np.mean(np.square(state))) <= 1.5 * np.sqrt(n * depth) * eps
    assert abs(np.mean(norm)) <= 4 * np.sqrt(np.mean(np.square(norm)) / len(norm))
