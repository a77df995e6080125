"""Which stage kernels a batch runs on: flat tiles for few cells or for narrow
grids that would leave lanes of the marching strips idle, else the march.
Measured flat against marching step times are with the rule (fvm_batch.cu);
the grids here are those of its clear cases."""
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Batch  # noqa: E402


@pytest.mark.parametrize("sizes,flat", [
    ([(128, 64)] * 16, True),
    ([(1240, 620)] * 3, True),       # 2.3 million cells
    ([(2048, 1024)] * 4, False),     # 8.4 million, strips 3 % idle: flat was 5 % slower
    ([(3100, 1550)] * 2, False),     # 9.6 million, strips full: 8 % slower
    ([(1024, 512)] * 15, True),      # 7.9 million, 9 % idle: flat is 2-4 % faster
    ([(512, 256)] * 61, True),       # 8 million, 21 % idle: 15 % faster
    ([(512, 256)] * 130, False),     # 17 million
])
def test_batch_route(sizes, flat):
    b = Batch()
    for nx, ny in sizes:
        b.add(small("euler_m3_circle", nx, ny)[0])
    assert b.debug_flat() is flat
