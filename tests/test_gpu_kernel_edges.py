"""Kernels at the sizes where their tiling can go wrong: edges of tiles, remainders, the smallest and the
largest of a range."""
import ctypes as C

import numpy as np
import pytest

import oracle
from nrltb import KMesh, abi, synth

pytestmark = pytest.mark.gpu


def _atoms(n, basis, seed):
    """n displaced atoms of one species in a row of simple cubic cells."""
    st = synth.supercell(synth.SC_BASIS, 4.6, (n, 1, 1), lambda b: 1, 0.1, np.random.default_rng(seed))
    return st, synth.make_params([basis], [4.0], synth.PARAM_SEED)


@pytest.mark.parametrize("natoms,basis", [(1, 1), (1, 9), (8, 4), (11, 9), (7, 9), (16, 4)])
@pytest.mark.parametrize("nk", [1, 3, 4, 5, 9])
def test_bloch_sums_over_k_groups_and_tiles(ctx, natoms, basis, nk):
    """H and S of every k: matrix orders 1, 9, 32, 99, 63, 64 against tiles of 32, k lists around groups of 4.
    Each element is a sum of at most a few hundred FP64 products in the oracle's order: 1e-13 of the largest."""
    st, par = _atoms(natoms, basis, 5)
    km = KMesh(np.random.default_rng(nk).uniform(-0.5, 0.5, (nk, 3)), np.full(nk, 1.0 / nk))
    for which in (0, 1):
        got = ctx.setham(st, par, km, which)
        want = oracle.setham(st, par, km, which)
        for g, o in zip(got, want):
            assert np.abs(g - o).max() <= 1e-13 * max(np.abs(o).max(), 1e-300)


def _cplx(rng, shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def _zgemm(ctx, method, opA, opB, tri, alpha, beta, A, B, Cm):
    """C = alpha op(A) op(B) + beta C; A, B, C as (batch, column, row) arrays."""
    m, n = Cm.shape[2], Cm.shape[1]
    k = A.shape[2] if opA else A.shape[1]
    A, B, out = np.ascontiguousarray(A), np.ascontiguousarray(B), np.ascontiguousarray(Cm).copy()
    rc = ctx.lib.nrltb_bench_zgemm_run(ctx.h, method, m, n, k, out.shape[0], opA, opB, *tri, alpha, beta,
                                       C.c_void_p(A.ctypes.data), A.shape[2], C.c_void_p(B.ctypes.data), B.shape[2],
                                       C.c_void_p(out.ctypes.data), m)
    assert rc == 0 and ctx.lib.nrltb_bench_umma_fault(0) == 0
    return out


def _zgemm_check(got, M, N, Cm, tri, alpha, beta):
    """Bound of the digit products: the operands' rounding (2^-56 of a power of two that is at most twice the row's
    or column's largest part, for both factors), the pairs dropped and the unit of the 64-bit sums, below
    K 2^-51 row maximum x column maximum in all; and two roundings of the result.  Held by 200 elements against
    extended precision, by all against double precision with that reference's own K 2^-52 |M| |N|."""
    K = M.shape[2]
    want = alpha * (M @ N) + beta * Cm.transpose(0, 2, 1)
    part = lambda x: np.maximum(np.abs(x.real), np.abs(x.imag))
    bound = K * 2.0 ** -51 * part(M).max(2)[:, :, None] * part(N).max(1)[:, None, :]
    bound = bound + 2.0 ** -52 * (np.abs(want) + np.abs(M @ N))
    m, n = want.shape[1:]
    use = np.tril(np.ones((m, n), bool)) if tri[2] == 1 else np.triu(np.ones((m, n), bool)) if tri[2] == 2 else \
        np.ones((m, n), bool)
    got = got.transpose(0, 2, 1)
    assert ((np.abs(got - want) <= bound + K * 2.0 ** -52 * (np.abs(M) @ np.abs(N))) | ~use).all()
    rng = np.random.default_rng(0)
    at = np.argwhere(np.broadcast_to(use, want.shape))
    L = np.clongdouble
    for b, i, j in at[rng.integers(0, len(at), 200)]:
        v = alpha * (M[b, i].astype(L) * N[b, :, j].astype(L)).sum() + beta * Cm[b, j, i]
        assert abs(complex(got[b, i, j] - v)) <= bound[b, i, j]


@pytest.mark.parametrize("m,n,k,batch", [(16, 16, 16, 3), (128, 64, 32, 1), (129, 65, 33, 2), (127, 63, 31, 2),
                                         (300, 200, 257, 2), (15, 16, 16, 1), (700, 33, 64, 5)])
@pytest.mark.parametrize("opA,opB", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_fp64_product_shapes(ctx, m, n, k, batch, opA, opB):
    """The digit products at the edges of their 128 x 64 x 32 tiles and of the rule that selects them."""
    rng = np.random.default_rng(m + n + k)
    A, B = _cplx(rng, (batch, m, k) if opA else (batch, k, m)), _cplx(rng, (batch, k, n) if opB else (batch, n, k))
    Cm = _cplx(rng, (batch, n, m))
    M = A.conj() if opA else A.transpose(0, 2, 1)
    N = B.conj() if opB else B.transpose(0, 2, 1)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0)):
        _zgemm_check(_zgemm(ctx, 1, opA, opB, (0, 0, 0), alpha, beta, A, B, Cm), M, N, Cm, (0, 0, 0), alpha, beta)


@pytest.mark.parametrize("m,n,k,batch", [(1, 1, 1, 300), (9, 9, 9, 57), (15, 15, 1, 4), (15, 15, 200, 2), (3, 15, 40, 5),
                                         (16, 15, 20, 2)])
@pytest.mark.parametrize("opA,opB", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("triA,triB", [(0, 0), (1, 0), (2, 0), (0, 1), (0, 2)])
def test_fp64_small_products(ctx, m, n, k, batch, opA, opB, triA, triB):
    """A thread per element: several matrices a CTA, a remainder of CTAs, the largest order and the next one."""
    rng = np.random.default_rng(m + n + k)
    A, B = _cplx(rng, (batch, m, k) if opA else (batch, k, m)), _cplx(rng, (batch, k, n) if opB else (batch, n, k))
    Cm = _cplx(rng, (batch, n, m))
    M = A.conj() if opA else A.transpose(0, 2, 1)
    N = B.conj() if opB else B.transpose(0, 2, 1)
    r, s = np.arange(m)[:, None] - np.arange(k), np.arange(k)[:, None] - np.arange(n)
    M = M * (r >= 0 if triA == 1 else r <= 0 if triA == 2 else True)
    N = N * (s <= 0 if triB == 1 else s >= 0 if triB == 2 else True)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0)):
        got = _zgemm(ctx, 1, opA, opB, (triA, triB, 0), alpha, beta, A, B, Cm).transpose(0, 2, 1)
        want = alpha * (M @ N) + beta * Cm.transpose(0, 2, 1)
        assert (np.abs(got - want) <= (k + 2) * 2.0 ** -51 * (np.abs(M) @ np.abs(N) + np.abs(Cm.transpose(0, 2, 1)))).all()


@pytest.mark.parametrize("n,batch", [(65, 1), (200, 6), (385, 5)])
@pytest.mark.parametrize("tri", [(1, 0, 0), (2, 0, 0), (0, 1, 0), (0, 2, 0), (0, 0, 1), (0, 0, 2), (1, 0, 1), (2, 0, 2)])
def test_fp64_product_triangles(ctx, n, batch, tri):
    """Every triangle form: the other half of a triangular operand is never read (NaN there)."""
    rng = np.random.default_rng(n)
    A, B, Cm = (_cplx(rng, (batch, n, n)) for _ in range(3))
    M, N = A.transpose(0, 2, 1).copy(), B.transpose(0, 2, 1).copy()
    low = np.tril(np.ones((n, n), bool))
    if tri[0]:
        M[:, ~(low if tri[0] == 1 else low.T)] = np.nan
    if tri[1]:
        N[:, ~(low.T if tri[1] == 1 else low)] = np.nan
    got = _zgemm(ctx, 1, 0, 0, tri, 1.0, 0.0, M.transpose(0, 2, 1), N.transpose(0, 2, 1), Cm)
    _zgemm_check(got, np.nan_to_num(M), np.nan_to_num(N), Cm, tri, 1.0, 0.0)


@pytest.mark.parametrize("scale", [0.0, 1e-320, 1e-160, 1e-30, 1e150, 1e300])
def test_fp64_product_scales_and_specials(ctx, scale):
    """Row scales from subnormal to near overflow; zero rows; one large element; infinities and NaN reach every
    element of their row and column and no other."""
    rng = np.random.default_rng(3)
    A, B, Cm = _cplx(rng, (1, 70, 150)), _cplx(rng, (1, 80, 70)), np.zeros((1, 80, 150), complex)
    A[0, :, 7] *= scale
    A[0, 3, 9] = 1e6
    M, N = A.transpose(0, 2, 1), B.transpose(0, 2, 1)
    got = _zgemm(ctx, 1, 0, 0, (0, 0, 0), 1.0, 0.0, A, B, Cm).transpose(0, 2, 1)
    # (the scaled row against itself unscaled: digits and sums depend on the scale by an exponent only)
    unit = scale if scale else 1.0
    by_unit = lambda x: x.real / unit + 1j * (x.imag / unit)   # (numpy's complex quotient overflows at 1e-320)
    want = np.vstack([M[0, :7] @ N[0], by_unit(M[0, 7:8]) @ N[0], M[0, 8:] @ N[0]])
    have = got[0].copy()
    have[7] = by_unit(have[7])
    size = np.abs(M[0]).max(1) * np.abs(N).max()
    size[7] /= unit
    tiny = 70 * 2.0 ** -1073 / unit * np.abs(N).max()   # a subnormal row has no more bits
    assert (np.abs(have - want) <= (70 * 2.0 ** -49 * size + (np.arange(150) == 7) * tiny)[:, None]).all()
    for special in (np.inf, np.nan):
        A2, B2 = A.copy(), B.copy()
        A2[0, 5, 140], B2[0, 11, 20] = special, complex(0, special)
        got = _zgemm(ctx, 1, 0, 0, (0, 0, 0), 1.0, 0.0, A2, B2, Cm).transpose(0, 2, 1)[0]
        hit = np.zeros((150, 80), bool)
        hit[140], hit[:, 11] = True, True
        assert (np.isfinite(got) == ~hit).all()


def _pencils(n, nk, seed):
    """nk Hermitian H and positive definite S = 1 + small, as (nk, n, n) arrays."""
    rng = np.random.default_rng(seed)
    H, S = _cplx(rng, (nk, n, n)), _cplx(rng, (nk, n, n)) * (0.1 / n)
    H = H + H.conj().transpose(0, 2, 1)
    return H, np.eye(n) + S @ S.conj().transpose(0, 2, 1)


@pytest.mark.parametrize("n,batches", [(1, (2,)), (2, (3,)), (31, (160,)), (32, (310,)), (33, (80, 160)),
                                       (64, (60, 330)), (65, (60, 160)), (128, (30, 40)), (129, (16, 40)),
                                       (160, (160,)), (161, (30, 160)), (257, (12, 30)), (545, (6,)), (801, (20,))])
def test_mixed_solve_does_not_depend_on_the_batch(ctx, n, batches):
    """Cluster sizes 1, 2, 4 and 8 of the panel kernel, with 8 and 16 warps, one wave and more: the first two
    matrices have the same eigenvalues and vectors, bit for bit, by themselves and ahead of others (the start of
    the inverse iteration goes by a matrix's place); the values within the form's 1e-9 of the matrix norm."""
    H, S = _pencils(n, 2, n)
    first = ctx.diag(H, S, precision=abi.PREC_MIXED)
    want = oracle.diag(H, S, vectors=False)[0]
    assert (first[2] == 0).all() and np.abs(first[0] - want).max() <= 1e-9 * np.abs(want).max()
    for nb in batches:
        at = np.arange(nb) % 2
        e, z, st = ctx.diag(H[at], S[at], precision=abi.PREC_MIXED)
        assert (st == 0).all() and np.array_equal(e[:2], first[0]) and np.array_equal(z[:2], first[1])
        assert np.abs(e - want[at]).max() <= 1e-9 * np.abs(want).max()


def _spectra(n, rng):
    """Hermitian matrices whose tridiagonal form is a hard one for bisection: (name, matrix, eigenvalues)."""
    Q = np.linalg.qr(_cplx(rng, (n, n)))[0]
    k = np.arange(n)
    yield "zero", np.zeros((n, n), complex), np.zeros(n)
    yield "multiple of one", -3.0 * np.eye(n) + 0j, np.full(n, -3.0)
    yield "diagonal", np.diag(np.cos(k) + 0j), np.sort(np.cos(k))
    for name, w in (("clusters", np.round(np.sin(k) * 2) + 1e-14 * k), ("graded", 2.0 ** -(k * 40.0 / max(n, 40))),
                    ("one far", np.where(k == 0, 1e3, 1e-3 * k)), ("plus minus", np.where(k % 2, 1.0, -1.0))):
        H = (Q * w) @ Q.conj().T
        yield name, (H + H.conj().T) / 2, np.sort(w)


@pytest.mark.parametrize("n", [1, 2, 3, 9, 31, 32, 33, 63, 64, 65, 129, 200])
@pytest.mark.parametrize("size", [1.0, 1e6, 1e-100, 1e120])
def test_fp64_spectra(ctx, n, size):
    """The FP64 form on spectra with clusters, zeros, grades and outliers.  Forming H, the reduction and the
    bisection are backward stable: each within 8 n 2^-53 of the norm, 32 in all."""
    rng = np.random.default_rng(n)
    names, H, want = zip(*_spectra(n, rng))
    S = np.tile(np.eye(n) + 0j, (len(H), 1, 1))
    e, _, st = ctx.diag(np.array(H) * size, S)
    e2, _, st2 = ctx.diag(np.array(H) * size, S, vectors=False)
    assert (st == 0).all() and (st2 == 0).all() and np.array_equal(e, e2)
    for name, got, w in zip(names, e, want):
        assert np.abs(got / size - w).max() <= 32 * n * 2.0 ** -53 * np.abs(w).max(), name


@pytest.mark.parametrize("n", [2, 33, 64, 129, 200])
@pytest.mark.parametrize("decades", [3, 30])
def test_fp64_scaled_basis(ctx, n, decades):
    """Basis functions scaled by powers of two: the same eigenvalues and, scaled back, the same vectors, bit for
    bit, since every step is exact in such a scale."""
    H, S = _pencils(n, 3, n)
    D = 2.0 ** np.random.default_rng(n).integers(-3 * decades, 3 * decades + 1, (3, n))
    e, z, st = ctx.diag(H, S)
    e2, z2, st2 = ctx.diag(H * D[:, :, None] * D[:, None, :], S * D[:, :, None] * D[:, None, :])
    assert (st == 0).all() and (st2 == 0).all()
    assert np.array_equal(e, e2) and np.array_equal(z, z2 * D[:, :, None])


@pytest.mark.parametrize("n,batches", [(1, (70,)), (16, (9,)), (17, (300,)), (32, (40,)), (33, (4,)), (65, (160,)),
                                       (112, (20,)), (113, (20, 60)), (160, (20, 80)), (161, (12, 40)), (192, (20, 80)),
                                       (193, (20, 60)), (225, (30,)), (300, (12,))])
def test_fp64_solve_does_not_depend_on_the_batch(ctx, n, batches):
    """One CTA, clusters of 8, 4 and 2, and columns ahead of a cluster: the first two matrices have the same
    eigenvalues and vectors, bit for bit, by themselves and ahead of others; values, residuals and S-orthonormality
    as a backward stable solve leaves them, 64 n 2^-53 of the norm (S is within 2 of one)."""
    H, S = _pencils(n, 2, n)
    first = ctx.diag(H, S)
    want = oracle.diag(H, S, vectors=False)[0]
    norm, tol = np.abs(want).max(), 64 * n * 2.0 ** -53
    assert (first[2] == 0).all() and np.abs(first[0] - want).max() <= tol * norm
    for j in (0, 1):
        e, z = first[0][j], first[1][j]
        assert np.abs(H[j] @ z - (S[j] @ z) * e).max() <= tol * norm
        assert np.abs(z.conj().T @ S[j] @ z - np.eye(n)).max() <= 1e-9   # (dstein's: eps norm / gap outside clusters)
    for nb in batches:
        at = np.arange(nb) % 2
        e, z, st = ctx.diag(H[at], S[at])
        assert (st == 0).all() and np.array_equal(e[:2], first[0]) and np.array_equal(z[:2], first[1])
        assert np.abs(e - want[at]).max() <= tol * norm
