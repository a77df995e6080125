"""Whole-field passes (derived fields, colour images, maxima, diagnostics,
cell classes) on grids whose rows do not end on a group of four cells, and
into destinations that are not 16-byte aligned.  References: NumPy on the
same state, the FP64 oracle, the oracle's shader."""
import numpy as np
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Solver, abi  # noqa: E402
from oracle import oracle  # noqa: E402
from oracle.oracle import Oracle  # noqa: E402

torch = pytest.importorskip("torch")


def _solver(nx, ny):
    p, e = small("ns_karman_re200", nx, ny, mach=2.0)
    s = Solver(p, e)
    p.dt = 0.3 * s.compute_dt()
    s.step(6)
    return s, p, e


def _derived(U, kind):
    U = U.astype(np.float64)
    r = U[0] + 1e-10
    T = 0.4 * (U[4] / r) / 287.05
    speed = np.hypot(U[1] / r, U[2] / r)
    return {abi.FIELD_TEMPERATURE: T, abi.FIELD_PRESSURE: 0.4 * U[4], abi.FIELD_DENSITY: U[0],
            abi.FIELD_VELOCITY_MAG: speed, abi.FIELD_MACH: speed / (np.sqrt(1.4 * 287.05 * T) + 1e-10)}[kind]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("nx", [5, 37, 38, 39, 40])
def test_fields_and_images_at_row_remainders(nx, offset):
    """rtol 1e-5 as for the aligned grids (approximate reciprocals and square
    roots); nothing written before or behind the destination."""
    s, p, e = _solver(nx, 21)
    n, U, ct = p.nx * p.ny, s.fields(), s.cell_types()
    buf = torch.full((n + 8,), -7.0, device="cuda")
    for kind in range(5):
        buf.fill_(-7.0)
        torch.cuda.synchronize()
        s.field_to_device(kind, buf.data_ptr() + 4 * offset)
        s.synchronize()
        got = buf.cpu().numpy()
        assert np.allclose(got[offset:offset + n].reshape(p.ny, p.nx), _derived(U, kind), rtol=1e-5), kind
        assert (got[:offset] == -7.0).all() and (got[offset + n:] == -7.0).all()
    s.cell_types_to_device(buf.data_ptr() + 4 * offset)
    s.synchronize()
    assert np.array_equal(buf.cpu().numpy()[offset:offset + n].reshape(p.ny, p.nx), ct.astype(np.float32))
    # RGBA8 (4-byte pixels): the image into an offset destination equals the aligned one
    img = [torch.full((n + 8,), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for k, off in enumerate((0, offset)):
        s.colormap_to_device(abi.FIELD_MACH, abi.CMAP_JET, 0.0, 2.5, img[k].data_ptr() + 4 * off, abi.RGBA_U8)
    s.synchronize()
    a, b = img[0].cpu().numpy(), img[1].cpu().numpy()
    assert np.array_equal(a[:n], b[offset:offset + n]) and (b[offset + n:] == 7).all() and (b[:offset] == 7).all()
    wall = (ct == abi.CELL_SOLID) | (ct == abi.CELL_GHOST)
    ref = oracle.colormap(_derived(U, abi.FIELD_MACH).astype(np.float32), ct, abi.CMAP_JET, 0.0, 2.5, fmt=1)
    got = a[:n].view(np.uint8).reshape(p.ny, p.nx, 4)
    assert np.array_equal(got[wall], ref[wall])
    assert np.abs(got.astype(int) - ref.astype(int)).max() <= 1


@pytest.mark.parametrize("nx,ny", [(5, 21), (37, 20), (38, 19), (39, 33), (40, 8), (1030, 67)])
def test_reductions_at_row_remainders(nx, ny):
    """Totals are exact sums up to FP64 rounding, forces as the aligned grids'
    bound; two calls in a row agree bit for bit (the scratch is left clean)."""
    s, p, e = _solver(nx, ny)
    o = Oracle(p, e, bits=64)
    o.set_geometry(s.sdf(), s.cell_types())
    U = s.fields()
    o.set_fields(U)
    d, r = s.diagnostics(), o.diagnostics()
    wall = np.isin(s.cell_types(), (abi.CELL_SOLID, abi.CELL_GHOST))
    area = float(np.float32(p.dx)) * float(np.float32(p.dy))
    for f, k in (("mass", 0), ("mom_x", 1), ("energy", 3)):
        assert getattr(d, f) == pytest.approx(U[k].astype(np.float64)[~wall].sum() * area, rel=1e-12), f
    scale = max(abs(r.force_x), abs(r.force_y), 1e-300)
    assert abs(d.force_x - r.force_x) <= 1e-4 * scale and abs(d.force_y - r.force_y) <= 1e-4 * scale
    d2 = s.diagnostics()
    assert all(getattr(d, f) == getattr(d2, f) for f in ("force_x", "force_y", "mass", "wall_heat", "wall_heat_max"))
    u, v, pr, T = s.primitives().astype(np.float64)
    mach = np.hypot(u, v) / (np.sqrt(1.4 * pr / (U[0].astype(np.float64) + 1e-10)) + 1e-10)
    for _ in range(2):
        assert s.max_temperature() == pytest.approx(T.max(), rel=1e-6)
        assert s.max_mach() == pytest.approx(mach.max(), rel=1e-5)
