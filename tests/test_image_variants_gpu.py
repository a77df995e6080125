"""Images to the last bit, whichever kernel variant writes them: the float
image against the shader's arithmetic in NumPy float32, RGBA8 into aligned and
unaligned destinations against its quantisation.

The ranges are chosen so that the divisor hi - lo + 1e-4 is a power of two in
float32: the division is then exact, and nothing else in the shader is
approximate.  The lower end is no short binary fraction, so a subtraction
fused with the value's last product shows."""
import numpy as np
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

import fvm_b200  # noqa: E402
from fvm_b200 import Solver, abi  # noqa: E402

torch = pytest.importorskip("torch")

F = np.float32
# field: (lower end, divisor)
RANGES = {abi.FIELD_TEMPERATURE: (210.3, 256.0), abi.FIELD_PRESSURE: (41000.7, 131072.0), abi.FIELD_DENSITY: (0.71, 1.0),
          abi.FIELD_VELOCITY_MAG: (313.7, 1024.0), abi.FIELD_MACH: (0.37, 4.0)}


def _range(lo, divisor):
    """(lo, hi) with lo as given up to some last bits and (hi - lo) + 1e-4 == divisor in float32."""
    lo = F(lo)
    for _ in range(64):
        for hi in (lo + F(divisor - 1e-4), np.nextafter(lo + F(divisor - 1e-4), F(np.inf))):
            if (hi - lo) + F(1e-4) == F(divisor):
                return lo, hi
        lo = np.nextafter(lo, F(np.inf))
    raise AssertionError("no such range")


def _shade(v, wall, table, lo, divisor):
    s = np.clip((v - lo) / F(divisor), F(0), F(1))
    u = s * F(256) - F(0.5)
    fl = np.floor(u)
    w = (u - fl)[..., None]
    i0, i1 = np.clip(fl.astype(int), 0, 255), np.clip(fl.astype(int) + 1, 0, 255)
    a, b = table[i0], table[i1]
    # fma(w, b, (1 - w) a): the product is exact in float64
    rgb = (w.astype(np.float64) * b + ((F(1) - w) * a).astype(np.float64)).astype(F)
    rgb[wall] = F(0.3)
    return np.concatenate([rgb, np.ones_like(rgb[..., :1])], axis=-1)


@pytest.mark.parametrize("nx,ny", [(400, 203), (401, 203)])
@pytest.mark.parametrize("field", sorted(RANGES))
@pytest.mark.parametrize("colormap", [abi.CMAP_JET, abi.CMAP_VIRIDIS])
def test_image_bits(field, colormap, nx, ny):
    p, e = small("euler_m3_circle", nx, ny)
    s = Solver(p, e)
    j, i = np.mgrid[0:ny, 0:nx].astype(F)
    w = 1 + 0.3 * np.sin(0.13 * i + 0.17 * j)
    rho, u, v, pr = p.rho_inf * w, p.u_inf * (1.2 - 0.4 * w), 50 * np.sin(0.3 * j), p.p_inf * w ** 1.3
    s.write_fields(np.stack([rho, rho * u, rho * v, pr / 0.4 + 0.5 * rho * (u * u + v * v), pr / 0.4]).astype(F))
    divisor = RANGES[field][1]
    lo, hi = _range(*RANGES[field])
    n = nx * ny
    buf = torch.zeros(4 * n + 4, device="cuda")
    torch.cuda.synchronize()
    s.field_to_device(field, buf.data_ptr())
    s.synchronize()
    value = buf[:n].cpu().numpy().reshape(ny, nx)
    ct = s.cell_types()
    ref = _shade(value, (ct == abi.CELL_SOLID) | (ct == abi.CELL_GHOST), fvm_b200.colormap_table(colormap), lo, divisor)
    assert len(np.unique(ref)) > 1000  # the range cuts into the values
    s.colormap_to_device(field, colormap, float(lo), float(hi), buf.data_ptr(), abi.RGBA_F32)
    s.synchronize()
    got = buf[:4 * n].cpu().numpy().reshape(ny, nx, 4)
    assert np.array_equal(got, ref), (np.abs(got - ref).max(), (got != ref).sum())
    q = np.rint(np.clip(ref, F(0), F(1)) * F(255)).astype(np.uint8)
    for offset in (0, 1):
        buf.zero_()
        torch.cuda.synchronize()
        s.colormap_to_device(field, colormap, float(lo), float(hi), buf.data_ptr() + 4 * offset, abi.RGBA_U8)
        s.synchronize()
        img = buf[offset:offset + n].cpu().numpy().view(np.uint8).reshape(ny, nx, 4)
        assert np.array_equal(img, q), (offset, (img != q).sum())
