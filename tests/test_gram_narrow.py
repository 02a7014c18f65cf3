"""gram_accumulate! of one panel with at most 48 columns (gram_narrow_kernel):
around the widths where the number of 8-column strips changes and the row
counts where a warp's 8-row boxes, a chunk's 32-row stages, a warp's ring and
the chunks of a whole GPU begin and end. At the end, both sides of the lines
where the split form takes over.

Tolerance, relative to ||a_i|| ||a_j||: the oracle's and the library's sums of
N terms round as a random walk, so 4 eps sqrt(N) covers both (with at least 16
terms' worth for the shortest)."""
import numpy as np
import pytest

from conftest import randmatrix
from test_gram_split import EPS, gram, norms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 7, 8, 9, 31, 33, 64, 65, 4736, 4737, 4800, 90_001])
@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 48, 49])
def test_widths_and_rows(fb, backend, N, k):
    rng = np.random.default_rng(1000 * k + N)
    A = randmatrix(rng, N, k)
    C0 = randmatrix(rng, k, k)
    n = norms(A)
    ref, scale, tol = A.conj().T @ A, np.outer(n, n), 4 * EPS * np.sqrt(max(N, 16))
    G = gram(fb, backend, A)
    assert np.max(np.abs(G - ref) / scale) <= tol
    assert np.array_equal(G, G.conj().T)
    H = gram(fb, backend, A, None, 0.5 - 2j, 1.0 + 1j, C0)
    assert np.max(np.abs(H - ((0.5 - 2j) * ref + (1.0 + 1j) * C0)) / (3 * scale + 2)) <= tol


@pytest.mark.parametrize("k", [1, 12, 20, 32, 40, 48])
def test_a_view_reads_only_its_rows_and_columns(fb, backend, k):
    # Everything around the view is NaN: a box past its last row or column is
    # filled with zeros, not with what lies there.
    rng = np.random.default_rng(k)
    N = 1003
    P = np.full((N + 40, k + 9), np.nan + 1j * np.nan, dtype=np.complex128, order="F")
    A = randmatrix(rng, N, k)
    P[16:16 + N, 1:1 + k] = A
    V = backend.todevice(P)[16:16 + N, 1:1 + k]
    C = backend.alloc_device(np.complex128, (k, k))
    fb.kernels.gram_accumulate(backend, C, V, V, 1.0, 0.0)
    backend.sync_all()
    n = norms(A)
    assert np.max(np.abs(C.to_host() - A.conj().T @ A) / np.outer(n, n)) <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("N,kA,kB", [(499_999, 48, 0), (500_000, 41, 0), (299_999, 49, 0), (300_000, 49, 0),
                                     (300_000, 200, 0), (249_999, 64, 36), (250_000, 64, 36), (399_999, 41, 41),
                                     (400_000, 41, 41), (400_000, 64, 32)])
def test_lines_between_fp64_and_split(fb, backend, N, kA, kB):
    rng = np.random.default_rng(N + kA)
    A = randmatrix(rng, N, kA)
    B = randmatrix(rng, N, kB) if kB else None
    G = gram(fb, backend, A, B)
    B = A if B is None else B
    assert np.max(np.abs(G - A.conj().T @ B) / np.outer(norms(A), norms(B))) <= 4 * EPS * np.sqrt(N)
