"""gram_accumulate! in its split form (slices on the integer tensor cores,
fb_ozaki_gram.cu), which the library takes for wide and tall products: around
the row and column counts where the choice and the tiles change, and where the
device's own verdict must refuse the sums and the FP64 kernels take over.

Tolerances, relative to sqrt(G_ii G_jj) or ||a_i|| ||b_j||: the slices leave
out less than 2^-53 of it and both the oracle's and the library's FP64 sums of
N terms round as a random walk, so 4 eps sqrt(N) covers all three."""
import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def gram(fb, backend, A, B=None, alpha=1.0, beta=0.0, C0=None):
    Ad = backend.todevice(np.asfortranarray(A))
    Bd = Ad if B is None else backend.todevice(np.asfortranarray(B))
    shape = (A.shape[1], (A if B is None else B).shape[1])
    C = backend.alloc_device(np.complex128, shape) if C0 is None else backend.todevice(np.asfortranarray(C0))
    fb.kernels.gram_accumulate(backend, C, Ad, Bd, alpha, beta)
    backend.sync_all()
    return C.to_host()


def norms(A):
    return np.linalg.norm(A, axis=0)


@pytest.mark.parametrize("N", [299_999, 300_000, 300_001, 300_015])
@pytest.mark.parametrize("k", [40, 41, 64, 65, 128, 130])
def test_folded(fb, backend, N, k):
    rng = np.random.default_rng(N + k)
    A = randmatrix(rng, N, k)
    C0 = randmatrix(rng, k, k)
    ref = A.conj().T @ A
    scale = np.outer(norms(A), norms(A))
    G = gram(fb, backend, A)
    assert np.max(np.abs(G - ref) / scale) <= 4 * EPS * np.sqrt(N)
    assert np.array_equal(G, G.conj().T)
    H = gram(fb, backend, A, None, 0.5 - 2j, 1.0 + 1j, C0)
    want = (0.5 - 2j) * ref + (1.0 + 1j) * C0
    assert np.max(np.abs(H - want) / (3 * scale + 2)) <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("N,kA,kB", [(249_999, 64, 64), (250_000, 64, 64), (400_017, 48, 48), (250_001, 64, 36),
                                     (250_003, 100, 70), (250_002, 129, 64)])
def test_cross(fb, backend, N, kA, kB):
    rng = np.random.default_rng(N + kA + kB)
    A, B = randmatrix(rng, N, kA), randmatrix(rng, N, kB)
    G = gram(fb, backend, A, B)
    assert np.max(np.abs(G - A.conj().T @ B) / np.outer(norms(A), norms(B))) <= 4 * EPS * np.sqrt(N)


def test_zero_columns_and_rows_that_grow(fb, backend):
    # Scales adapt as the rows grow by 2^40; zero columns stay exactly zero.
    rng = np.random.default_rng(3)
    N, k = 300_000, 64
    A = randmatrix(rng, N, k) * (2.0 ** (40 * np.arange(N) / N))[:, None]
    A[:, 5] = 0
    A[:200_000, 9] = 0
    G = gram(fb, backend, A)
    n = norms(A)
    n[5] = 1.0
    assert np.max(np.abs(G - A.conj().T @ A) / np.outer(n, n)) <= 4 * EPS * np.sqrt(N)
    assert np.all(G[5] == 0) and np.all(G[:, 5] == 0)


@pytest.mark.parametrize("same", [True, False])
def test_a_spike_is_summed_in_fp64(fb, backend, same):
    # One entry of 2^40 in a column of unit entries. Against the exact product
    # the FP64 sums are off by at most (rows of a chunk) eps 2^40; slices scaled
    # for the spike would round every other entry of the column to 2^-11.
    rng = np.random.default_rng(4)
    N, k = 300_000, 64
    A = (rng.standard_normal((N, k)) + 1j * rng.standard_normal((N, k))) / np.sqrt(2)
    A[77, 3] = 2.0 ** 40
    B = A if same else (rng.standard_normal((N, k)) + 1j * rng.standard_normal((N, k))) / np.sqrt(2)
    rest = A[:, 3].copy()
    rest[77] = 0
    G = gram(fb, backend, A, None if same else B)
    chunk = -(-N // 148 // 32) * 32
    for j in (0, 1, 2, 10, 40, 63):
        exact = rest.conj() @ B[:, j] + 2.0 ** 40 * B[77, j]
        assert abs(G[3, j] - exact) <= chunk * EPS * 2.0 ** 40


@pytest.mark.parametrize("value", [np.nan, np.inf, 2.0 ** 480])
@pytest.mark.parametrize("same", [True, False])
def test_what_slices_cannot_hold_is_summed_in_fp64(fb, backend, value, same):
    # A NaN, an infinity or a magnitude whose products leave the slices' range
    # reaches only the rows and columns it belongs to.
    rng = np.random.default_rng(5)
    N, k = 300_001, 56
    A = randmatrix(rng, N, k)
    B = A if same else randmatrix(rng, N, k)
    ref = A.conj().T @ B
    scale = np.outer(norms(A), norms(B))
    A2 = A.copy()
    A2[123_456, 7] = value
    G = gram(fb, backend, A2, None if same else B)
    keep = np.ones((k, k), dtype=bool)
    keep[7, :] = False
    if same:
        keep[:, 7] = False
    assert np.max((np.abs(G - ref) / scale)[keep]) <= 4 * EPS * np.sqrt(N)
    if np.isfinite(value):
        want = (A2[:, 7].conj() @ B) if not same else A2[:, 7].conj() @ A2
        assert np.all(np.abs(G[7] - want) <= 1e-12 * np.abs(want))
    else:
        assert not np.any(np.isfinite(G[7]))
