"""What the device's verdict on the split Gram (fb_ozaki_gram.cu) accepts and
refuses, read from the workspace, and the entries that come out either way,
each against its own sum_r |a_ri| |b_rj| in extended precision.

Accepted sums: each of the two terms of the verdict's bound is below
2^-54 ||a|| ||b||, and the 148 chunk sums are added in runs of 19 and 8, so 8 eps
||a|| ||b|| covers them (a lost slice costs 20 eps or more). Refused ones are FP64
sums of N terms, which round as a random walk: 4 eps sqrt(N) of sum |a| |b|."""
import ctypes

import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
PAIRS = [(0, 0), (0, 1), (1, 2), (3, 8), (5, 40), (17, 30), (20, 21), (35, 34)]


def gram(fb, backend, A, B=None):
    """G, the verdict of every output tile (the first words of the workspace) and
    what the screen refused (four words a column from the next 256 bytes on)."""
    vp = ctypes.c_void_p
    Ad = backend.todevice(np.asfortranarray(A))
    Bd = Ad if B is None else backend.todevice(np.asfortranarray(B))
    need = ctypes.c_size_t(0)
    fb._lib.call("fb_zgram_workspace_size", ctypes.c_int64(Ad.rows), Ad.cols, Bd.cols, int(B is None),
                 ctypes.byref(need))
    ws = backend.todevice(np.full((need.value // 16 + 1, 1), np.nan + 0j, order="F"))
    C = backend.alloc_device(np.complex128, (Ad.cols, Bd.cols))
    fb._lib.check(fb._lib.load().fb_zgram(vp(C.ptr), C.ld, vp(Ad.ptr), Ad.ld, vp(Bd.ptr), Bd.ld, Ad.rows, Ad.cols,
                                          Bd.cols, fb._lib.z128(1.0), fb._lib.z128(0.0), vp(ws.ptr), need.value, None),
                  "fb_zgram")
    fb._lib.call("fb_sync_all")
    na, nb = -(-Ad.cols // 64), -(-Bd.cols // 64)
    words = ws.to_host().view(np.int32).ravel()
    tiles = na * (na + 1) // 2 if B is None else na * nb
    screen = -(-tiles // 64) * 64
    return C.to_host(), words[:tiles], words[screen:screen + 4 * (Ad.cols if B is None else Ad.cols + Bd.cols)]


def errors(G, A, B, pairs):
    """Largest |G_ij - exact| over the pairs, against ||a|| ||b|| and against sum |a| |b|."""
    L = np.longdouble
    norm = size = 0.0
    for i, j in pairs:
        ar, ai, br, bi = (np.asarray(v, dtype=L) for v in (A[:, i].real, A[:, i].imag, B[:, j].real, B[:, j].imag))
        d = np.hypot(float(G[i, j].real - ((ar * br).sum() + (ai * bi).sum())),
                     float(G[i, j].imag - ((ar * bi).sum() - (ai * br).sum())))
        norm = max(norm, d / (np.linalg.norm(A[:, i]) * np.linalg.norm(B[:, j])))
        size = max(size, d / (np.abs(A[:, i]) @ np.abs(B[:, j])))
    return norm, size


def gaussian(rng, N, k):
    return rng.standard_normal((N, k)) + 1j * rng.standard_normal((N, k))


def flat(kind, rng, N, k):
    r, j = np.arange(N)[:, None] / N, np.arange(1, k + 1)[None, :]
    if kind == "gaussian":
        return gaussian(rng, N, k)
    if kind == "uniform":
        return randmatrix(rng, N, k)
    if kind == "waves":
        return np.exp(2j * np.pi * j * r)
    if kind == "modes":
        return np.sin(np.pi * j * r) + 1j * np.cos(np.pi * j * r)
    X = gaussian(rng, N, k)     # "zeros": a zero column, and one that starts late, on a chunk's first row
    X[:, 3] = 0
    X[:2032 * 70, 8] = 0
    return X


@pytest.mark.parametrize("kind", ["gaussian", "uniform", "waves", "modes", "zeros"])
@pytest.mark.parametrize("N,kA,kB", [(300_000, 64, None), (250_007, 64, 64), (300_017, 130, None), (250_001, 100, 64)])
def test_flat_columns_are_accepted(fb, backend, kind, N, kA, kB):
    rng = np.random.default_rng(N + kA)
    A = flat(kind, rng, N, kA)
    B = A if kB is None else flat(kind, rng, N, kB)
    G, verdict, screen = gram(fb, backend, A, None if kB is None else B)
    if kind != "zeros" or (N, kA, kB) == (300_000, 64, None):
        assert not screen.any() and not verdict.any()
    pairs = [p for p in PAIRS + [(kA - 1, B.shape[1] - 2), (kA - 1, 2)] if 3 not in p]
    assert errors(G, A, B, pairs)[0] <= 8 * EPS


def graded(kind, rng, N, k, first):
    X, r = gaussian(rng, N, k), np.arange(N)
    odd = (np.arange(k) + first) % 2 == 1
    low = {"halves": r < N // 2, "runs": r % 64 < 32, "rows": r % 2 == 0}.get(kind)
    if low is not None:          # every other column small where the others are large
        return X * np.where(low[:, None] ^ odd, 2.0 ** -48, 1.0)
    if kind == "sparse":
        return X * (rng.random((N, k)) < 0.05)
    if kind == "spike":          # where the others are zero
        X[77] = 0
        X[77, 3] = 2.0 ** 60
        return X
    if kind == "range":
        return X * 2.0 ** 460
    raise AssertionError(kind)


@pytest.mark.parametrize("kind", ["halves", "runs", "rows", "sparse", "spike", "range"])
@pytest.mark.parametrize("N,kA,kB", [(300_000, 64, None), (250_007, 64, 48), (300_017, 70, None)])
def test_columns_that_share_no_rows_at_their_scale_are_refused(fb, backend, kind, N, kA, kB):
    rng = np.random.default_rng(N + kA)
    A = graded(kind, rng, N, kA, 0)
    B = A if kB is None else graded(kind, rng, N, kB, 0)
    G, verdict, _ = gram(fb, backend, A, None if kB is None else B)
    assert verdict.any()
    assert errors(G, A, B, PAIRS)[1] <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("modulus,accepted", [(0.82, False), (1.05, True)])
@pytest.mark.parametrize("same", [True, False])
def test_the_norm_a_scale_asks_for(fb, backend, modulus, accepted, same):
    # What the slices leave out stays below 2^-54 ||a|| ||b|| from ||a||^2 =
    # 0.29 sqrt(N) 4^E on, checked with 1.4 times that to spare (0.41). The
    # entry of 20 sets 2^E = 32: modulus 0.82 has 0.36 sqrt(N) 4^E, 1.05 has 0.59.
    rng = np.random.default_rng(6)
    N, k = 300_000, 64
    wave = lambda: np.exp(2j * np.pi * rng.random((N, k)))
    A = wave()
    A[:, 5] *= modulus
    A[1_000, 5] = 20.0
    G, verdict, _ = gram(fb, backend, A, None if same else wave())
    assert bool(verdict.any()) != accepted


def uneven(kind, rng, N, k):
    r, j = np.arange(N)[:, None] / N, np.arange(1, k + 1)[None, :]
    if kind == "sines":
        return np.sin(np.pi * j * r) * (1 + 0.5j)
    if kind == "envelopes":
        return gaussian(rng, N, k) * np.exp(-(r - j / (k + 1)) ** 2 / (2 * 0.02 ** 2))
    if kind == "heavy tails":
        return gaussian(rng, N, k) / np.sqrt(rng.random((N, k)))
    if kind == "sparse":
        return gaussian(rng, N, k) * (rng.random((N, k)) < 0.2)
    X = gaussian(rng, N, k)      # "one": a single column of them all
    X[:, k - 1] *= rng.random(N) < 0.2
    return X


@pytest.mark.parametrize("kind", ["sines", "envelopes", "heavy tails", "sparse", "one"])
@pytest.mark.parametrize("N,kA,kB", [(300_000, 64, None), (250_007, 48, 64), (300_017, 70, None)])
def test_what_slices_are_slow_on_is_refused_by_its_sample(fb, backend, kind, N, kA, kB):
    rng = np.random.default_rng(N + kA)
    A = uneven(kind, rng, N, kA)
    B = A if kB is None else gaussian(rng, N, kB) if kind == "one" else uneven(kind, rng, N, kB)
    G, verdict, screen = gram(fb, backend, A, None if kB is None else B)
    assert screen.any() and verdict.all()
    if kind == "one":
        assert np.flatnonzero(screen)[0] >= 4 * (kA - 1)
    assert errors(G, A, B, PAIRS)[1] <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("spiked,accepted", [(8, True), (64, False)])
@pytest.mark.parametrize("same", [True, False])
def test_a_chunk_whose_scales_keep_growing_is_left_to_fp64(fb, backend, spiked, accepted, same):
    # Entries of 20 among waves of modulus 1, each in another stage of one chunk
    # and past the sampled rows: a new epoch each, 16 at most.
    rng = np.random.default_rng(8)
    N, k, chunk, rows = 300_000, 64, 5, 2032
    wave = lambda: np.exp(2j * np.pi * rng.random((N, k)))
    A, B = wave(), wave()
    half = (rows - 16) // 2
    sampled = {o + i for r in (1, 2) for i in range(16)
               for o in [(r - 1) * half + (((4 * chunk + r) * 2654435761 % 2 ** 32) * half >> 32)]}
    free = [s for s in range(17, rows - 32, 16) if s not in sampled]
    for j in range(spiked):
        A[chunk * rows + free[j], j] = 20.0
    G, verdict, screen = gram(fb, backend, A, None if same else B)
    assert not screen.any() and bool(verdict.any()) != accepted
    assert errors(G, A, A if same else B, PAIRS)[1] <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("N,kA,kB", [(300_000, 64, None), (300_017, 130, None), (250_001, 64, 48)])
def test_the_gram_of_real_columns_is_real(fb, backend, N, kA, kB):
    rng = np.random.default_rng(N + kA)
    real = lambda k: (0.5 + rng.random((N, k))) * rng.choice([-1.0, 1.0], (N, k)) + 0j
    A = real(kA)
    B = A if kB is None else real(kB)
    G, _, _ = gram(fb, backend, A, None if kB is None else B)
    assert not G.imag.any()
    assert errors(G, A, B, PAIRS)[1] <= 4 * EPS * np.sqrt(N)


@pytest.mark.parametrize("small", [2.0 ** -20, 2.0 ** -40])
def test_a_small_imaginary_part_keeps_its_digits(fb, backend, small):
    # Im G_ij sums re_i im_j - im_i re_j: 2 N terms, against their own size.
    rng = np.random.default_rng(12)
    N, k = 300_000, 64
    A = 0.5 + rng.random((N, k)) + 1j * small * (0.5 + rng.random((N, k)))
    G, _, _ = gram(fb, backend, A)
    L = np.longdouble
    for i, j in PAIRS + [(0, 63), (9, 60)]:
        if i // 8 == j // 8:     # the folded 8 x 8 diagonal blocks of the FP64 form carry Re + Im
            continue
        ar, ai, br, bi = (np.asarray(v, dtype=L) for v in (A[:, i].real, A[:, i].imag, A[:, j].real, A[:, j].imag))
        exact, size = (ar * bi).sum() - (ai * br).sum(), float((ar * bi).sum() + (ai * br).sum())
        assert abs(float(L(G[i, j].imag) - exact)) <= 4 * EPS * np.sqrt(2 * N) * size
