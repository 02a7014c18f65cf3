"""The 7-point Laplacian's tiles (fb_stencil.cu) where they can go wrong:
grids around the 32 x 16 tile, the 8-plane ring and the 16-plane pieces,
several columns with a leading dimension past the grid. Each output is a sum
of seven products, so 16 eps times the largest magnitude covers the rounding of
both sides."""
import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu


def laplace(v, grid, shift):
    nx, ny, nz = grid
    x = v.reshape((nx, ny, nz), order="F")
    p = np.pad(x, 1)
    s = (p[:-2, 1:-1, 1:-1] + p[2:, 1:-1, 1:-1] + p[1:-1, :-2, 1:-1] + p[1:-1, 2:, 1:-1] + p[1:-1, 1:-1, :-2]
         + p[1:-1, 1:-1, 2:])
    return ((6 + shift) * x - s).reshape(-1, order="F")


@pytest.mark.parametrize("grid", [(1, 1, 1), (32, 16, 1), (33, 17, 2), (31, 15, 6), (32, 16, 7), (65, 33, 8), (2, 40, 9),
                                  (64, 1, 31), (1, 16, 32), (30, 18, 33), (96, 48, 49)])
@pytest.mark.parametrize("cols", [1, 3])
def test_tiles(fb, backend, grid, cols):
    n = grid[0] * grid[1] * grid[2]
    rng = np.random.default_rng(n + cols)
    X = randmatrix(rng, n + 5, cols)
    shift = 0.5 + 0.1j
    Xd = backend.todevice(X)
    Yd = backend.todevice(np.full((n + 7, cols), np.nan + 0j, dtype=np.complex128, order="F"))
    x, y = Xd.view(slice(0, n)), Yd.view(slice(0, n))
    fb.kernels.laplace7_apply(backend, y, x, grid, shift)
    backend.sync_all()
    out = Yd.to_host()
    for c in range(cols):
        ref = laplace(X[:n, c], grid, shift)
        assert np.max(np.abs(out[:n, c] - ref)) <= 16 * np.finfo(np.float64).eps * 13
    assert np.all(np.isnan(out[n:]))   # nothing past the grid is written
