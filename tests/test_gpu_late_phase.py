"""A bounded wait looks once more after its limit has passed.

The limit is in time, and time passes while a context is switched out: a copy
that landed meanwhile is there, however late the clock is.  The self-test's
clock completes the phase and then reads past the limit.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_phase_completed_before_the_limit_was_read_counts():
    import torch

    from ns3dperiodic_b200._lib import lib

    assert torch.cuda.is_available()
    seen = ctypes.c_int(-1)
    assert lib().ns3d_selftest_late_phase(ctypes.byref(seen)) == 0
    assert seen.value == 1
