"""Failure detection without a GPU fault: a bounded wait that runs out (an
mbarrier that nothing arms) sets the library's status word, the host reports
it as an error, and the same context keeps working afterwards."""
import numpy as np
import pytest

from bfps_b200 import ic

pytestmark = pytest.mark.gpu


def test_bounded_wait_runs_out_and_context_stays_usable():
    from bfps_b200 import _lib
    from bfps_b200.solver import vorticity_equation
    ve = vorticity_equation(32, precision="single")
    try:
        rc = _lib.lib().bfg_selftest_wait(ve.handle)
        assert rc == _lib.BFG_ECUDA
        assert b"ran out" in _lib.lib().bfg_last_error(ve.handle)
        # the status word was cleared: steps run and report normally
        w0 = ic.vorticity_ic(32, seed=3, dtype=np.complex64)
        ve.set_cvorticity(w0)
        ve.step(0.01, 2)
        assert ve.last_step_ms() > 0
        w = ve.get_cvorticity()
        assert np.isfinite(w).all() and not np.array_equal(w, w0)
    finally:
        ve.close()


@pytest.mark.parametrize("precision", ["single", "double"])
def test_calls_do_not_wait_for_the_callers_streams(precision):
    """Calls without device arrays of the caller return while a kernel that the
    caller queued on the default stream (about a second of sleep) still runs."""
    import torch
    from bfps_b200 import _lib
    from bfps_b200.solver import particles_system, vorticity_equation
    n = 64
    L = _lib.lib()
    ve = vorticity_equation(n, precision=precision)
    w = ic.vorticity_ic(n, seed=3, dtype=ve.cdtype)
    ve.set_cvorticity(w)
    ps = particles_system(ve, ic.tracer_ic(100, seed=1), 2, 0, 2)
    c, r = np.array(w), np.zeros(ve.rshape, ve.rdtype)
    calls = {
        "step": lambda: (ve.step(0.001, 1), ve.last_step_ms()),
        "velocity_rspace": ve.velocity_rspace,
        "do_stats": lambda: ve.do_stats(5.0, 50.0, 32),
        "compute_pressure": ve.compute_pressure,
        "acceleration": ve.compute_Lagrangian_acceleration,
        "field_ift": lambda: _lib.check(L.bfg_field_ift(ve.handle, _lib.FIELD_VELOCITY), ve.handle),
        "ift": lambda: _lib.check(L.bfg_ift(ve.handle, c.ctypes.data, r.ctypes.data), ve.handle),
        "dft": lambda: _lib.check(L.bfg_dft(ve.handle, r.ctypes.data, c.ctypes.data), ve.handle),
        "sample_velocity": ps.sample_velocity,
        "sample_acceleration": ps.sample_acceleration,
        "upload": lambda: ve.set_cvorticity(w),
        "download": ve.get_cvorticity,
    }
    for call in calls.values():  # workspaces, kernels
        call()
    waited = []
    for name, call in calls.items():
        torch.cuda.synchronize()
        torch.cuda._sleep(2 * 10 ** 9)
        call()
        if torch.cuda.current_stream().query():
            waited.append(name)
    torch.cuda.synchronize()
    ps.close()
    ve.close()
    assert not waited
