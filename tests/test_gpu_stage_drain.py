"""A z pass whose staged rows broke down waits for the copies it armed last.

The pass stages the rows of its six transforms on one mbarrier, so stage k
completes the phase of parity k & 1.  When a wait gives up, the last armed
stage can be any of the six; a drain of another parity returns at once and lets
the CTA exit with a copy in flight into its shared memory.  The self-test arms
stages 0 .. last: with the last one open the drain has to run out its bounded
wait, and it must not return before a last one that another thread completes.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", range(6))
def test_drain_follows_the_last_armed_stage(last):
    import torch

    from ns3dperiodic_b200._lib import lib

    assert torch.cuda.is_available()
    drained = ctypes.c_int(-1)
    for complete in (0, 1):
        assert lib().ns3d_selftest_stage_drain(last, complete, ctypes.byref(drained)) == 0
        assert drained.value == complete
