"""The marching stage kernels on grids that run on the flat one by default: the
oracle comparisons of the parity, grid-shape and rare-cell tests with a pinned
marching shape, and rare cells at the tile ends of both kernels, flat against
marching bit for bit."""
import numpy as np
import pytest

from helpers import small, rel_l1, FIELDS
import test_grids_gpu as grids
import test_parity_gpu as parity
import test_rare_cells_gpu as rare

pytestmark = pytest.mark.gpu

from fvm_b200 import Solver, abi  # noqa: E402
from oracle.oracle import Oracle  # noqa: E402

SHAPES = [(128, 4, 8), (256, 6, 16)]


@pytest.mark.parametrize("case", list(parity.CASES))
@pytest.mark.parametrize("shape,steps", [(SHAPES[0], 1), (SHAPES[0], 100), (SHAPES[1], 10)])
def test_steps_match_fp32_oracle(case, shape, steps):
    """The parity test's bound: relative L1 <= 1e-4 after up to 100 steps."""
    s, o, p, e, _ = parity._pair(case)
    s.set_tune(*shape)
    if case in parity.CFL_DT_CASES:
        for _ in range(steps):
            p.dt = o.compute_dt()
            s.step(1)
            o.step(p.dt)
    else:
        p.dt = o.compute_dt()
        s.step(steps)
        for _ in range(steps):
            o.step(p.dt)
    U = s.fields()
    assert np.isfinite(U).all()
    l1 = rel_l1(U, o.fields())
    assert l1.max() <= 1e-4, dict(zip(FIELDS, l1))


@pytest.mark.parametrize("name", list(grids.GRIDS))
def test_odd_and_small_grids_match_fp32_oracle(name):
    """The grid test's bound: relative L1 <= 1e-4 after 30 steps."""
    p, e = grids._case(name)
    s = Solver(p, e)
    s.set_tune(*SHAPES[0])
    o = Oracle(p, e, bits=32)
    o.set_geometry(s.sdf(), s.cell_types())
    o.set_fields(s.fields())
    p.dt = o.compute_dt()
    s.step(30)
    for _ in range(30):
        o.step(p.dt)
    l1 = rel_l1(s.fields(), o.fields())
    assert l1.max() <= 1e-4, dict(zip(FIELDS, l1))


KINDS = ["low_density", "fast", "cold", "nonfinite"]
FORMS = [(f, m) for f in (abi.FLUX_HLLC, abi.FLUX_AUSM_PLUS) for m in (abi.LIMITER_MINMOD, abi.LIMITER_VAN_LEER)]


@pytest.mark.parametrize("flux,limiter", FORMS)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape", SHAPES)
def test_rare_cells_match_fp32_oracle(kind, flux, limiter, shape):
    """The rare-cell test's bounds: the same cells finite, relative L1 <= 1e-4
    after one step."""
    p, e = small("euler_m3_circle", 141, 37, flux_scheme=flux, limiter=limiter)
    s = Solver(p, e)
    s.set_tune(*shape)
    o = Oracle(p, e, bits=32)
    o.set_geometry(s.sdf(), s.cell_types())
    U = rare._state(p, kind)
    s.write_fields(U)
    o.set_fields(U)
    p.dt = 0.02 * min(p.dx, p.dy) / p.u_inf
    s.step(1)
    o.step(p.dt)
    A, R = s.fields(), o.fields()
    assert np.array_equal(np.isfinite(A), np.isfinite(R))
    if kind != "nonfinite":
        l1 = rel_l1(A, R)
        assert l1.max() <= 1e-4, dict(zip(FIELDS, l1))


# (row, column) at the ends of the flat kernel's tiles (32 columns; 6 rows on
# the small grid, 14 on the large one), of the marching strips (124) and tiles (8 rows)
ENDS = [(5, 31), (6, 32), (6, 63), (13, 64), (14, 31), (12, 96), (27, 127), (28, 128), (29, 33), (7, 95), (8, 34)]


@pytest.mark.parametrize("nx,ny", [(141, 37), (650, 302)])
@pytest.mark.parametrize("flux,limiter", FORMS)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("workload", ["euler_m3_circle", "ns_karman_re200"])
def test_rare_cells_flat_equals_marching(monkeypatch, kind, flux, limiter, nx, ny, workload):
    """Three steps; states, CFL maxima and non-finite count the same."""
    monkeypatch.setattr(rare, "PLACES", rare.PLACES + ENDS)
    out = []
    for shape in (None, SHAPES[0]):
        p, e = small(workload, nx, ny, flux_scheme=flux, limiter=limiter, mach=3.0)
        s = Solver(p, e)
        if shape:
            s.set_tune(*shape)
        s.write_fields(rare._state(p, kind))
        p.dt = 0.02 * min(p.dx, p.dy) / p.u_inf
        s.step(3)
        out.append((s.fields(), s.compute_dt(), s.nonfinite_count()))
    (A, *a), (B, *b) = out
    if kind == "nonfinite":  # not-a-numbers have no one bit pattern
        assert np.array_equal(A, B, equal_nan=True)
    else:
        assert np.array_equal(A.view(np.uint32), B.view(np.uint32))
    assert np.array_equal(a, b, equal_nan=True)
