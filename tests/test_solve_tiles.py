"""rdiv_upper! as a product by the inverse (trsm_inv_kernel): around the widths
where the 4-column n-tiles and the depth of a warp's ring change, and the row
counts where 8-row units, a CTA's warps, the GPU's CTAs and the ring begin to
repeat. Every entry is checked: a copy that overtook the reads of the rows
before it would show in single rows.

Tolerance: |X - Y R^-1| <= (k + 8) eps sum_l |y_l| |R^-1|_lj, with a cond_1(R)
below 4, so 16 (k + 8) eps times the row's largest entry times k covers it."""
import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def factor(rng, k):
    R = np.triu(randmatrix(rng, k, k)) * (0.2 / k)
    R[np.diag_indices(k)] = 1.0 + 0.1 * rng.random(k)
    return np.asfortranarray(R)


@pytest.mark.parametrize("N", [1, 7, 8, 9, 1184, 1185, 18_944, 18_953, 75_776, 75_801, 300_007])
@pytest.mark.parametrize("k", [1, 4, 5, 8, 12, 16, 20, 28, 32, 33, 40, 44, 48, 52, 60, 61, 64])
def test_every_row(fb, backend, N, k):
    rng = np.random.default_rng(100 * k + N)
    R, Y = factor(rng, k), randmatrix(rng, N, k)
    Yd = backend.todevice(Y)
    fb.kernels.rdiv_upper(backend, Yd, backend.todevice(R))
    backend.sync_all()
    want = Y @ np.linalg.inv(R)
    err = np.abs(Yd.to_host() - want).max(axis=1)
    assert np.all(err <= 16 * (k + 8) * EPS * k * np.abs(Y).max(axis=1))


@pytest.mark.parametrize("k", [3, 16, 44])
def test_a_view_touches_only_its_entries(fb, backend, k):
    rng = np.random.default_rng(k)
    N = 5003
    R, Y = factor(rng, k), randmatrix(rng, N, k)
    P = np.full((N + 24, k + 5), np.nan + 1j * np.nan, dtype=np.complex128, order="F")
    P[9:9 + N, 2:2 + k] = Y
    Pd = backend.todevice(P)
    fb.kernels.rdiv_upper(backend, Pd[9:9 + N, 2:2 + k], backend.todevice(R))
    backend.sync_all()
    got = Pd.to_host()
    assert np.abs(got[9:9 + N, 2:2 + k] - Y @ np.linalg.inv(R)).max() <= 16 * (k + 8) * EPS * k * np.abs(Y).max()
    got[9:9 + N, 2:2 + k] = np.nan + 1j * np.nan
    assert np.all(np.isnan(got))
