"""The tensor-core products at their limits: barrier waits that run out, digit scratch for a part of the batch."""
import ctypes as C

import numpy as np
import pytest

from nrltb import abi

pytestmark = pytest.mark.gpu


def _zgemm(ctx, A, B, scratch=None):
    """A B by the FP64 form's dispatch; A, B as (batch, column, row) arrays."""
    batch, k, m = A.shape
    n = B.shape[1]
    out = np.zeros((batch, n, m), complex)
    p = lambda a: C.c_void_p(a.ctypes.data)
    args = [ctx.h, 1, m, n, k, batch, 0, 0, 0, 0, 0, 1.0, 0.0, p(A), m, p(B), k, p(out), m]
    f = ctx.lib.nrltb_bench_zgemm_run if scratch is None else ctx.lib.nrltb_bench_zgemm_scratch
    assert f(*args, *([] if scratch is None else [scratch])) == abi.NRLTB_OK
    assert ctx.lib.nrltb_bench_umma_fault(0) == 0
    return out


def _operands(m, n, k, batch):
    rng = np.random.default_rng(m + n + k)
    draw = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
    return draw(batch, k, m), draw(batch, n, k)


def _scratch(m, n, k, matrices):
    mt, nt, kc = -(-m // 128), -(-n // 64), -(-k // 32)
    return ((mt + nt) * kc * 7 * 16384 + 8 * (mt * 128 + nt * 64)) * matrices + 1024


# (the FP32 product's CTAs wait one wave after another: no batch above one wave)
@pytest.mark.parametrize("kernel,n,batch", [(0, 128, 1), (0, 385, 5)] +
                         [(k, n, batch) for k in (1, 2) for n, batch in ((128, 1), (160, 300), (385, 5))])
def test_wait_that_runs_out_is_reported_and_leaves_nothing_behind(ctx, kernel, n, batch):
    """The wait for an accumulator that is never said to be empty: the kernel gives up after its two seconds, says so,
    and the products after it are those before it, bit for bit."""
    A, B = _operands(n, n, n, 3)
    before = _zgemm(ctx, A, B)
    assert ctx.lib.nrltb_bench_wait_runs_out(ctx.h, kernel, n, batch) == abi.NRLTB_E_TIMEOUT
    assert np.array_equal(_zgemm(ctx, A, B), before)


@pytest.mark.parametrize("m,n,k", [(129, 65, 33), (300, 200, 257), (16, 16, 16), (385, 385, 64)])
def test_products_in_parts(ctx, m, n, k):
    """Scratch for 1, 2, 4 and 5 of 5 matrices (parts of 1, of 2, 2 and 1, of 4 and 1): the same bits.  For none: the
    FMA pipe, whose own errors are below K 2^-51 |A| |B|, as the digit products' are of row and column maxima."""
    A, B = _operands(m, n, k, 5)
    want = _zgemm(ctx, A, B)
    for fit in (5, 4, 2, 1):
        assert np.array_equal(_zgemm(ctx, A, B, _scratch(m, n, k, fit)), want)
    part = lambda x: np.maximum(np.abs(x.real), np.abs(x.imag))
    a, b = np.abs(A.transpose(0, 2, 1)), np.abs(B.transpose(0, 2, 1))
    bound = k * 2.0 ** -51 * (a @ b + part(A).max(1)[:, :, None] * part(B).max(2)[:, None, :])
    assert (np.abs(_zgemm(ctx, A, B, 1024) - want).transpose(0, 2, 1) <= bound).all()
