"""The solve's scalars on the host (CFL maxima, time step): every call that
waits for the stream leaves those of the current state for fvm_read_dt,
whichever way they reached the host (copied, or written by a step's last pass
or by the CFL pass)."""
import ctypes as C

import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Solver, abi  # noqa: E402


def _read_dt(s):
    dt = C.c_float()
    assert s.lib.fvm_read_dt(s.h, C.byref(s.params), C.byref(dt)) == 0
    return dt.value


def _solver(workload, policy):
    p, e = small(workload, 96, 48)
    e.dt_policy = policy
    s = Solver(p, e)
    if policy == abi.DT_FIXED:
        p.dt = 0.5 * s.compute_dt()
    return s


@pytest.mark.parametrize("workload", ["euler_m3_circle", "ns_karman_re200"])
@pytest.mark.parametrize("policy", [abi.DT_FIXED, abi.DT_RECOMPUTE])
@pytest.mark.parametrize("steps", [1, 2, 3, 20, 70, 71])
def test_read_dt_after_steps_and_a_wait(workload, policy, steps):
    """Exact: both come from the same maxima.  20 single steps pass the point
    where step graphs take over; 70 and 71 in one call use them at once."""
    s = _solver(workload, policy)
    for n in ([1] * 20 if steps == 20 else [steps]):
        s.step(n)
    s.synchronize()
    read = _read_dt(s)
    assert read == s.compute_dt()
    assert read == _read_dt(s)


def test_read_dt_after_compute_dt_of_a_new_state():
    s = _solver("euler_m3_circle", abi.DT_FIXED)
    s.step(1)
    s.synchronize()
    U = s.fields()
    U[1:3, 20:30, 40:60] *= 1.5  # faster there
    U[3, 20:30, 40:60] = U[4, 20:30, 40:60] + 0.5 * (U[1] ** 2 + U[2] ** 2)[20:30, 40:60] / U[0, 20:30, 40:60]
    s.write_fields(U)
    dt = s.compute_dt()
    assert _read_dt(s) == dt


def test_queued_dt_is_the_queued_state_s():
    """A step queued behind fvm_queue_dt does not change what was queued until
    a call that reads the scalars waits for it."""
    s = _solver("euler_m3_circle", abi.DT_FIXED)
    s.step(3)
    now = s.compute_dt()
    assert s.lib.fvm_queue_dt(s.h, C.byref(s.params)) == 0
    s.fields()  # waits, reads no scalars
    assert _read_dt(s) == now
