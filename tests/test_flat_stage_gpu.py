"""The flat stage kernel (small grids, both tile heights) gives the marching
kernels' bits: grids narrower and shorter than a tile, odd sizes, tiles that
end inside the grid, every flux and limiter, Euler and Navier-Stokes, the
display field, several steps under the recomputed time step."""
import numpy as np
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Batch, Solver, abi  # noqa: E402

torch = pytest.importorskip("torch")

# the last two have enough 32x14 tiles for the taller tile
GRIDS = [(5, 40), (40, 3), (33, 13), (31, 15), (37, 19), (131, 67), (701, 333), (650, 302)]


def _run(nx, ny, workload, flux, limiter, tune, display=False):
    p, e = small(workload, nx, ny, flux_scheme=flux, limiter=limiter, mach=2.5)
    e.dt_policy = abi.DT_RECOMPUTE
    s = Solver(p, e)
    if tune:
        s.set_tune(*tune)
    out = None
    if display:
        out = torch.zeros(nx * ny, device="cuda")
        torch.cuda.synchronize()
        s.set_display_field(abi.FIELD_MACH, out.data_ptr())
    s.step(5)
    s.synchronize()
    return s.fields(), p.dt, p.t_current, s.nonfinite_count(), None if out is None else out.cpu().numpy()


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("workload", ["euler_m3_circle", "ns_karman_re200"])
@pytest.mark.parametrize("flux,limiter", [(abi.FLUX_HLLC, abi.LIMITER_MINMOD), (abi.FLUX_HLLC, abi.LIMITER_VAN_LEER),
                                          (abi.FLUX_AUSM_PLUS, abi.LIMITER_MINMOD),
                                          (abi.FLUX_AUSM_PLUS, abi.LIMITER_VAN_LEER)])
def test_flat_stages_equal_marching_stages(nx, ny, workload, flux, limiter):
    a = _run(nx, ny, workload, flux, limiter, None)
    b = _run(nx, ny, workload, flux, limiter, (128, 4, 8))
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
    assert a[1:4] == b[1:4]


def test_flat_stage_display_field():
    for workload in ("euler_m3_circle", "ns_karman_re200"):
        a = _run(131, 67, workload, abi.FLUX_HLLC, abi.LIMITER_MINMOD, None, True)
        b = _run(131, 67, workload, abi.FLUX_HLLC, abi.LIMITER_MINMOD, (128, 4, 8), True)
        assert np.array_equal(a[4].view(np.uint32), b[4].view(np.uint32))


@pytest.mark.parametrize("flux,limiter", [(abi.FLUX_HLLC, abi.LIMITER_VAN_LEER),
                                          (abi.FLUX_AUSM_PLUS, abi.LIMITER_MINMOD)])
def test_flat_batch_equals_marching_batch(monkeypatch, flux, limiter):
    """Uneven sizes, Euler and Navier-Stokes mixed: the default (flat tiles)
    against a pinned marching shape."""
    def run():
        cases = [small(w, nx, ny, flux_scheme=flux, limiter=limiter, mach=2.5)
                 for w, nx, ny in (("euler_m3_circle", 131, 67), ("ns_karman_re200", 97, 33), ("euler_m3_circle", 37, 19),
                                   ("ns_karman_re200", 200, 100))]
        ext = cases[0][1]
        ext.dt_policy = abi.DT_RECOMPUTE
        b = Batch(ext)
        ids = [b.add(p) for p, _ in cases]
        b.step(7)
        return [(b.fields(i), b.instance(i).dt, b.instance(i).t_current) for i in ids]
    a = run()
    monkeypatch.setenv("FVM_BATCH_TUNE", "128,6,16")
    for x, y in zip(a, run()):
        assert np.array_equal(x[0].view(np.uint32), y[0].view(np.uint32)) and x[1:] == y[1:]
