"""Cells that the stage kernels handle behind a branch, against the FP32
oracle: first-order faces of low-density cells, wall faces, the update's
rollback (a density or internal energy under its floor, NaN and infinite
fields) and its velocity cap.  They sit in both rows of a row pair and at the
ends of a column strip.  Around infinite fields only which cells stay finite
is compared: the values there follow from infinities times approximate
reciprocals."""
import numpy as np
import pytest

from helpers import small, rel_l1, FIELDS

pytestmark = pytest.mark.gpu

from fvm_b200 import Solver, abi  # noqa: E402
from oracle.oracle import Oracle  # noqa: E402

# (row, column) on a 141 x 37 grid: both rows of a pair, the strips' ends
# (column strips are 124 wide), beside the obstacle and in the free flow
PLACES = [(4, 7), (5, 20), (10, 122), (11, 123), (14, 124), (21, 125), (30, 138), (35, 60)]


def _state(p, kind):
    j, i = np.mgrid[0:p.ny, 0:p.nx].astype(np.float32)
    w = 1 + 0.02 * np.sin(0.21 * i + 0.13 * j)
    rho, u, v, pr = p.rho_inf * w, p.u_inf * (2 - w), 30.0 * np.sin(0.3 * j), p.p_inf * w
    for n, (a, b) in enumerate(PLACES):
        if kind == "low_density":      # on both sides of the first-order threshold 0.01, and under the floor 1e-4
            rho[a, b] = (0.004, 0.03, 5e-5)[n % 3]
            pr[a, b] *= rho[a, b]
        elif kind == "fast":           # over the velocity cap of 5000 m/s
            u[a, b], v[a, b] = (7000.0, 100.0) if n % 2 else (3000.0, 6000.0)
        elif kind == "cold":           # internal energy near its floor
            pr[a, b] = 0.02
    U = np.stack([rho, rho * u, rho * v, pr / 0.4 + 0.5 * rho * (u * u + v * v), pr / 0.4]).astype(np.float32)
    if kind == "nonfinite":
        for n, (a, b) in enumerate(PLACES):
            U[n % 5, a, b] = (np.nan, np.inf)[n % 2]
    return U


@pytest.mark.parametrize("flux", [abi.FLUX_HLLC, abi.FLUX_AUSM_PLUS])
@pytest.mark.parametrize("limiter", [abi.LIMITER_MINMOD, abi.LIMITER_VAN_LEER])
@pytest.mark.parametrize("kind", ["low_density", "fast", "cold", "nonfinite"])
def test_rare_cells_match_fp32_oracle(kind, limiter, flux):
    """One step: the same cells finite, and relative L1 <= 1e-4 (the bound of
    the smooth cases' 100 steps: a jump of 1e4 in density costs the precision
    that 100 steps do)."""
    p, e = small("euler_m3_circle", 141, 37, flux_scheme=flux, limiter=limiter)
    s = Solver(p, e)
    o = Oracle(p, e, bits=32)
    o.set_geometry(s.sdf(), s.cell_types())
    U = _state(p, kind)
    s.write_fields(U)
    o.set_fields(U)
    p.dt = 0.02 * min(p.dx, p.dy) / p.u_inf
    s.step(1)
    o.step(p.dt)
    A, R = s.fields(), o.fields()
    assert np.array_equal(np.isfinite(A), np.isfinite(R))
    if kind == "nonfinite":
        return
    l1 = rel_l1(A, R)
    assert l1.max() <= 1e-4, dict(zip(FIELDS, l1))
