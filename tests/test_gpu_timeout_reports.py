"""Every call that hands results to the host reports a wait that gave up.

ns3d_selftest_expire_wait lets one bounded wait run out on the handle's stream
and flag, as a pass whose copies broke down does.  The next read-back, whichever
it is, has to fail with the timeout and hand out nothing; the one after it
succeeds, with the values of before.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 6  # NS3D_ERR_TIMEOUT


def _calls(tmp_path):
    def saved(name, path):
        def call(s, U):
            getattr(s, name)(str(path), U)
            return np.frombuffer(path.read_bytes(), np.uint8)
        return call
    return {
        "synchronize": lambda s, U: s.synchronize() or 0,
        "diagnostics": lambda s, U: s.diagnostics(U),
        "record": lambda s, U: s.record(U, 0.5, 30.0),
        "spectrum": lambda s, U: s.energy_spectrum(U),
        "shapiro": lambda s, U: s.shapiro_error(U, 0.1, 30.0),
        "save_fourier": saved("save_control_fourier", tmp_path / "f.dat"),
        "save_file": saved("save_control_file", tmp_path / "p.dat"),
    }


@pytest.mark.parametrize("what", ["synchronize", "diagnostics", "record", "spectrum", "shapiro",
                                  "save_fourier", "save_file"])
def test_read_back_reports_the_timeout_once(what, tmp_path):
    from ns3dperiodic_b200 import Solver
    from ns3dperiodic_b200._lib import Ns3dError, lib

    call = _calls(tmp_path)[what]
    with Solver(32, 32, 32) as s:
        U = s.shapiro_state(0.0, 30.0)
        before = call(s, U)
        for p in tmp_path.iterdir():
            p.unlink()
        assert lib().ns3d_selftest_expire_wait(s._h) == 0
        with pytest.raises(Ns3dError) as e:
            call(s, U)
        assert e.value.status == TIMEOUT
        assert not list(tmp_path.iterdir())  # nothing written
        assert np.array_equal(np.asarray(call(s, U)), np.asarray(before))
        s.synchronize()


def test_ensemble_diagnostics_report_the_timeout():
    from ns3dperiodic_b200 import Ensemble
    from ns3dperiodic_b200._lib import Ns3dError, lib

    with Ensemble(2, 16, 16, 16) as e:
        U = [u.clone() for u in e.zeros()]
        before = e.diagnostics(U)
        # an ensemble's first member is the handle it steps
        h = ctypes.cast(e._h, ctypes.POINTER(ctypes.c_void_p))[0]
        assert lib().ns3d_selftest_expire_wait(ctypes.c_void_p(h)) == 0
        with pytest.raises(Ns3dError) as err:
            e.diagnostics(U)
        assert err.value.status == TIMEOUT
        assert np.array_equal(np.asarray(e.diagnostics(U)), np.asarray(before))
