"""The tall product D <- A C (rmul_pair_kernel) at the row count where it takes
over, with remainders of its 16-row pairs and 8-row units, and around the
widths where 16-column stages, 2-column steps and 4-column n-tiles begin.

Tolerance: both sides add K products, so 4 (K + 8) eps ||a_row|| ||c_col||."""
import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
LINE = 1 << 18


@pytest.mark.parametrize("N", [LINE - 1, LINE, LINE + 7, LINE + 9])
@pytest.mark.parametrize("K,n", [(7, 9), (8, 1), (9, 4), (15, 16), (16, 17), (17, 20), (33, 5), (50, 20), (63, 33),
                                 (64, 61), (64, 64), (20, 64)])
def test_rightmul(fb, backend, N, K, n):
    rng = np.random.default_rng(N + 100 * K + n)
    A, C = randmatrix(rng, N, K), randmatrix(rng, K, n)
    P = np.full((N + 5, n + 2), np.nan + 1j * np.nan, dtype=np.complex128, order="F")
    Pd = backend.todevice(P)
    fb.kernels.rightmul_gemm(backend, Pd[3:3 + N, 1:1 + n], backend.todevice(A), backend.todevice(C))
    backend.sync_all()
    got = Pd.to_host()
    bound = 4 * (K + 8) * EPS * np.outer(np.linalg.norm(A, axis=1), np.linalg.norm(C, axis=0))
    assert np.all(np.abs(got[3:3 + N, 1:1 + n] - A @ C) <= bound)
    got[3:3 + N, 1:1 + n] = np.nan + 1j * np.nan
    assert np.all(np.isnan(got))
