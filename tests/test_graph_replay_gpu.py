"""Replay of captured step graphs against plain launches, bit for bit.  The
graphs take over after 16 plain steps or in a call of more than 64; every mode
here passes that point, and the graph counts show that it did."""
import numpy as np
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Solver, abi  # noqa: E402

TOTAL = 90
# calls of fvm_steps, and the graph launches they make: two steps each, one for an odd remainder
MODES = {
    "single": ([1] * TOTAL, TOTAL - 16),                    # one-step graphs of both buffer parities
    "long": ([70, 20], 45),                                 # two-step graphs alone
    "odd": ([71, 1, 15, 3], 35 + 1 + 1 + 7 + 1 + 1 + 1),    # both kinds, the parity changing in between
    "mixed": ([1] * 15 + [2] + [3, 2, 1, 4, 1, 2, 3, 5, 7, 1, 2, 6, 1, 9, 4, 11, 2, 3, 1, 5], 43),
}


def _run(workload, nx, ny, policy, calls, eager=False):
    p, e = small(workload, nx, ny)
    e.dt_policy = policy
    s = Solver(p, e)
    if policy == abi.DT_FIXED:
        p.dt = 0.5 * s.compute_dt()
    if eager:
        s.set_kernel_timing(True)  # every kernel launched by itself
    for n in calls:
        s.step(n)
    s.synchronize()
    out = (s.fields(), s.compute_dt(), p.dt, p.t_current, p.step, s.nonfinite_count())
    return out, s.debug_graph_count(), s.launch_count()


# the last grid is large enough for the marching stages
@pytest.mark.parametrize("workload,nx,ny", [("euler_m3_circle", 160, 80), ("ns_karman_re200", 160, 80),
                                            ("ns_karman_re200", 1600, 960)])
@pytest.mark.parametrize("policy", [abi.DT_FIXED, abi.DT_RECOMPUTE])
def test_graph_replay_matches_plain_launches(workload, nx, ny, policy):
    ref, counts, launches = _run(workload, nx, ny, policy, [TOTAL], eager=True)
    assert counts == (0, 0)
    for mode, (calls, replays) in MODES.items():
        assert sum(calls) == TOTAL
        if nx > 1000 and mode in ("single", "long"):
            continue
        got, (captured, launched), n = _run(workload, nx, ny, policy, calls)
        assert launched == replays, mode
        assert captured == (2 if mode in ("single", "long") else 4), mode  # per kind one for each buffer parity
        assert n == launches, mode
        assert np.array_equal(got[0].view(np.uint32), ref[0].view(np.uint32)), mode
        assert got[1:] == ref[1:], mode


def test_changing_cfl_numbers_never_capture():
    """A CFL number that changes with every call changes what a captured step
    holds: such a solve keeps to plain launches, and captures once it stays."""
    p, e = small("euler_m3_circle", 160, 80)
    e.dt_policy = abi.DT_RECOMPUTE
    s = Solver(p, e)
    q, _ = small("euler_m3_circle", 160, 80)
    r = Solver(q, e)
    r.set_kernel_timing(True)
    for k in range(40):
        p.cfl = q.cfl = 0.2 + 0.005 * k
        s.step(1)
        r.step(1)
    assert s.debug_graph_count() == (0, 0)
    s.step(20)
    s.step(2)
    r.step(22)
    assert s.debug_graph_count() == (2, 1)
    p.cfl = q.cfl = 0.3  # and a change drops them again
    s.step(3)
    r.step(3)
    assert s.debug_graph_count() == (2, 1)
    assert np.array_equal(s.fields().view(np.uint32), r.fields().view(np.uint32))
    assert p.dt == q.dt and p.t_current == q.t_current


@pytest.mark.parametrize("steps", [6, 80])
def test_autotuner_times_graph_replay(steps):
    """Each candidate captures its graphs while it warms up (3 steps: a
    two-step and a one-step launch, each kind for both parities) and replays
    them in the timed steps."""
    p, e = small("ns_karman_re200", 160, 80)
    s = Solver(p, e)
    p.dt = 0.5 * s.compute_dt()
    U = s.fields()
    assert s.autotune(steps) > 0
    captured, launched = s.debug_graph_count()
    assert captured > 0 and captured % 4 == 0
    assert launched == captured // 4 * (2 + steps // 2)
    assert np.array_equal(s.fields().view(np.uint32), U.view(np.uint32))
    s.step(1)  # the solve itself starts plainly again
    assert s.debug_graph_count() == (captured, launched)
