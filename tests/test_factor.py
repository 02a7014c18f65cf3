"""The k x k factor step (fb_factor.cuh) at the sizes where its blocks, its
stores and its inverse's levels change: the Cholesky and R_new = U R_old
through fb_zpotrf_shifted, the solve plan through rdiv_upper!.

||U^H U - G|| <= 4 k eps ||G|| (each entry is a sum of at most k products, real
and imaginary parts); the solve's residual ||X R - Y|| <= 8 k eps ||X|| ||R||."""
import numpy as np
import pytest

from conftest import randmatrix

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
SIZES = [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 33, 40, 56, 63, 64, 65, 100, 127, 128, 160, 161, 200]


def gram(rng, k, kappa):
    A = randmatrix(rng, 3 * k + 8, k) @ np.diag(10.0 ** -np.linspace(0, np.log10(kappa), k))
    return A.conj().T @ A


@pytest.mark.parametrize("k", SIZES)
@pytest.mark.parametrize("kappa", [1.0, 1e5])
def test_cholesky_and_update(fb, backend, k, kappa):
    rng = np.random.default_rng(k)
    G = gram(rng, k, kappa)
    Rin = np.triu(randmatrix(rng, k, k))
    dev = lambda a: backend.todevice(np.asfortranarray(a))
    U, Rout = backend.alloc_device(np.complex128, (k, k)), backend.alloc_device(np.complex128, (k, k))
    shifted, _ = fb.kernels.cholesky_upper_device(backend, dev(G), 1000, k, U, dev(Rin), Rout)
    u, r = U.to_host(), Rout.to_host()
    assert not shifted
    assert np.array_equal(u, np.triu(u)) and np.all(np.diag(u).imag == 0) and np.all(np.diag(u).real > 0)
    assert np.linalg.norm(u.conj().T @ u - G) <= 4 * k * EPS * np.linalg.norm(G)
    assert np.linalg.norm(r - u @ Rin) <= 4 * k * EPS * np.linalg.norm(u) * np.linalg.norm(Rin)


@pytest.mark.parametrize("k", [1, 5, 8, 13, 16, 23, 32, 37, 40, 48, 57, 64, 65, 72, 128, 150])
@pytest.mark.parametrize("kappa", [1.0, 1e6, 1e9])
def test_plan_and_solve(fb, backend, k, kappa):
    # kappa 1 solves by the inverse, 1e6 by blocks, 1e9 (graded inside the 8 x 8
    # blocks of a narrow factor) also by substitution.
    rng = np.random.default_rng(100 + k)
    R = np.triu(randmatrix(rng, k, k)) * 0.1 + np.diag(10.0 ** -np.linspace(0, np.log10(kappa), k))
    Y = randmatrix(rng, 501, k)
    Yd = backend.todevice(np.asfortranarray(Y))
    fb.kernels.rdiv_upper(backend, Yd, backend.todevice(np.asfortranarray(R)))
    backend.sync_all()
    X = Yd.to_host()
    assert np.linalg.norm(X @ R - Y) <= 8 * k * EPS * np.linalg.norm(X) * np.linalg.norm(R)


def test_a_failing_pivot_is_found_in_every_block(fb, backend):
    rng = np.random.default_rng(9)
    for k, bad in [(64, 0), (64, 7), (64, 8), (64, 63), (40, 39), (128, 100)]:
        G = gram(rng, k, 1.0)
        G[bad, bad] = -abs(G[bad, bad]) * 1e3
        with pytest.raises(fb.NotPositiveDefinite):
            fb.kernels.cholesky_upper_device(backend, backend.todevice(np.asfortranarray(G)), 10, k,
                                             backend.alloc_device(np.complex128, (k, k)))


@pytest.mark.parametrize("k", [1, 9, 64, 65, 160, 161, 200])
@pytest.mark.parametrize("forced", [None, 2.0 ** -53])
def test_r_may_take_the_place_of_u(fb, backend, k, forced):
    # Only Rin must not alias Rout: R = U Rin written over U itself, or over
    # memory that U's columns run through, holds what separate arrays hold.
    # Two sums of at most k products in different orders: 4 k eps each.
    rng = np.random.default_rng(200 + k)
    G, Rin = gram(rng, k, 1e3), np.triu(randmatrix(rng, k, k))
    dev = lambda a: backend.todevice(np.asfortranarray(a))
    factor = lambda U, R: fb.kernels.cholesky_upper_device(backend, dev(G), 1000, k, U, dev(Rin), R, forced)
    U, R = backend.alloc_device(np.complex128, (k, k)), backend.alloc_device(np.complex128, (k, k))
    factor(U, R)
    u, r = U.to_host(), R.to_host()
    bound = 8 * k * EPS * np.linalg.norm(u) * np.linalg.norm(Rin)
    same = backend.alloc_device(np.complex128, (k, k))
    factor(same, same)
    assert np.linalg.norm(same.to_host() - r) <= bound
    both = backend.alloc_device(np.complex128, (k + 1, k))     # U from the first row on, R from the second
    at = lambda row: fb.DeviceMatrix(both.ptr + 16 * row, (k, k), both.ld, np.dtype(np.complex128), both)
    factor(at(0), at(1))
    assert np.linalg.norm(both.to_host()[1:] - r) <= bound
