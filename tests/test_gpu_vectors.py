"""Eigenvectors of matrices whose tridiagonal form falls into blocks, some of them zero or far from one in size."""
import numpy as np
import pytest

from nrltb import abi

pytestmark = pytest.mark.gpu


def _hermitian(n, rng):
    G = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    return (G + G.conj().T) / 2


def _two_blocks(n, size, seed):
    """Half of the orbitals coupled among themselves, the others too, `size` times as strongly; and the same shuffled."""
    rng, h = np.random.default_rng(seed), n // 2
    G = _hermitian(n, rng)
    G[:h, h:] = G[h:, :h] = 0
    G[h:, h:] *= size
    at = rng.permutation(n)
    return [G, G[np.ix_(at, at)]]


def _check(ctx, H, precision, norm=None):
    """Residuals within 64 n units of the norm, as for any matrix (the mixed form's 1e-9), and orthonormal vectors
    (within 1e-9: dstein's bound goes by the gaps)."""
    n = len(H[0])
    e, z, st = ctx.diag(np.array(H), np.tile(np.eye(n) + 0j, (len(H), 1, 1)), precision=precision)
    assert (st == 0).all() and np.isfinite(e).all() and np.isfinite(z).all()
    tol = 64 * n * 2.0 ** -53 if precision == abi.PREC_FP64 else 1e-9
    for h, ej, zj in zip(H, e, z):
        assert np.abs(h @ zj - zj * ej).max() <= tol * np.abs(np.linalg.eigvalsh(h)).max()
        assert np.abs(zj.conj().T @ zj - np.eye(n)).max() <= 1e-9
    return e


# (the mixed form refines clusters of up to 16 vectors)
@pytest.mark.parametrize("precision,n", [(abi.PREC_FP64, n) for n in (1, 2, 9, 20, 64, 128, 200)] +
                         [(abi.PREC_MIXED, n) for n in (1, 2, 9, 16)])
def test_zero_blocks(ctx, precision, n):
    H = [np.zeros((n, n), complex)]
    if n > 1:
        H += _two_blocks(n, 0.0, n) + _two_blocks(n, 1e-15, n)
    _check(ctx, H, precision)


@pytest.mark.parametrize("n", [9, 20, 64, 128, 200])
def test_graded(ctx, n):
    """Rows and columns falling by 2^-80: the reduction leaves zero blocks of the smallest."""
    D = 2.0 ** -(np.arange(n) * 80.0 / n)
    G = _hermitian(n, np.random.default_rng(n)) * D[:, None] * D
    at = np.random.default_rng(n).permutation(n)
    _check(ctx, [G, G[::-1, ::-1], G[np.ix_(at, at)]], abi.PREC_FP64)


@pytest.mark.parametrize("n", [4, 9, 20, 64, 128, 200])
@pytest.mark.parametrize("size", [1e-15, 1e-40, 1e-70, 1e-100, 1e-150])
def test_small_blocks_have_their_own_scale(ctx, n, size):
    """A decoupled block's eigenvalues are good to 32 n units of the block's norm, however small it is beside the
    other's (e^2 stays a normal number), and its vectors orthonormal; shuffled, the reduction mixes the blocks and
    the matrix's norm counts."""
    H = _two_blocks(n, size, n)
    e = _check(ctx, H, abi.PREC_FP64)
    w = np.linalg.eigvalsh(H[0][n // 2:, n // 2:] / size)
    got = np.sort(e[0][np.argsort(np.abs(e[0]))[:n - n // 2]]) / size
    assert np.abs(got - w).max() <= 32 * n * 2.0 ** -53 * np.abs(w).max()


@pytest.mark.parametrize("n", [2, 9, 33, 64, 160])
@pytest.mark.parametrize("precision,size", [(abi.PREC_MIXED, s) for s in (1e-18, 1e-22, 1e-24, 1e-30)] +
                         [(abi.PREC_FP64, s) for s in (1e-24, 1e-155, 1e-165, 1e-200)])
def test_couplings_whose_squares_vanish(ctx, n, precision, size):
    """Levels coupled by so little that the squares of a whole column are no longer numbers of the form's range."""
    G = _hermitian(n, np.random.default_rng(n)) * size
    G[np.arange(n), np.arange(n)] = np.cos(np.arange(n))
    _check(ctx, [G], precision)
