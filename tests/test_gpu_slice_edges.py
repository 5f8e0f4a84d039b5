"""The sliced FP64 GEMM at the ends of its range and on the calls that reach it in
other ways than a plain contraction."""
import time

import numpy as np
import pytest

from test_gpu_slice import ctx, dense, product  # noqa: F401
from ultradmrg_gb300 import api
from ultradmrg_gb300.tensor_data import IN, OUT, BlockTensorData, Index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ea,eb", [(-498, -498), (-477, -476), (-475, -475), (-474, -520),
                                   (475, 475), (475, -475), (499, 499), (-476, 477)])
def test_ends_of_the_range(ctx, ea, eb):  # noqa: F811
    """Lines whose maxima are near 2^ea and 2^eb, with sums that cancel down to the
    last bits: results below 2^-1022 are FP64's, not wrapped exponents.  Bound: the
    sliced form's, or the FMAs' K roundings at the largest product and below the
    normal range."""
    rng = np.random.default_rng(abs(ea - 3 * eb))
    m, n, k = 70, 66, 96
    a, b = rng.integers(-2 ** 20, 2 ** 20, (m, k)), rng.integers(-2 ** 20, 2 ** 20, (k, n))
    # pairs that cancel: wholly where a is large, but for b's last bit where a is
    # small, so that results are a few units of 2^(ea + eb - 40)
    a[:, k // 2:] = rng.integers(-3, 4, (m, k // 2))
    a[:, 1::2] = a[:, 0::2]
    b[1::2] = -b[0::2]
    b[k // 2 + 1::2] += rng.integers(-1, 2, (k // 4, n))
    a, b = np.ldexp(a.astype(float), ea - 20), np.ldexp(b.astype(float), eb - 20)
    got = product(ctx, a, b)
    ref = a.astype(np.longdouble) @ b.astype(np.longdouble)
    top = np.abs(a).max(1).astype(np.longdouble)[:, None] * np.abs(b).max(0)[None, :]
    tiny = np.ldexp(np.longdouble(1), -1074)
    assert np.all(np.isfinite(got))
    assert np.all(np.abs(got - ref) <= 2.0 ** -53 * np.abs(ref) + k * (2.0 ** -52 * top + tiny))


@pytest.mark.parametrize("k", [256, 512, 1040])
def test_coherent_low_digits(ctx, k):  # noqa: F811
    """Leading digits that cancel over lower ones of one sign: the largest sums of
    the lower levels, beyond 2^24 in level 5.  Bound: one rounding of the result and
    four units of level 5 (2^-50 of the lines' scales, here 1) per product."""
    s, t = (np.where(np.arange(k) // w % 2, -1, 1) for w in (1, 2))
    low = sum(127 * 2.0 ** -(6 + 8 * d) for d in range(1, 5))
    a = s * 63 / 64 + low + t * 127 * 2.0 ** -46
    b = t * 63 / 64 + low + s * 127 * 2.0 ** -46
    a, b = np.tile(a, (130, 1)), np.tile(b[:, None], (1, 66))
    b[:, 1] *= -1.0
    got = product(ctx, a, b)
    ref = np.array([[sum(int(x) * int(y) for x, y in zip(a[0] * 2.0 ** 46, b[:, j] * 2.0 ** 46))
                     for j in (0, 1)]], dtype=object)
    for j in (0, 1):
        exact = np.longdouble(float(ref[0, j] >> 40)) * np.ldexp(np.longdouble(1), 40 - 92)
        cols = got[:, j::2] if j == 0 else got[:, 1:2]
        assert np.all(np.abs(cols - exact) <= 2.0 ** -52 * np.abs(exact) + k * 2.0 ** -50)


def two_sectors(shapes, decades, seed, dtype=np.float64):
    """A block-diagonal matrix (one block per charge) and its blocks; singular values
    decay over `decades`."""
    rng = np.random.default_rng(seed)
    blocks = {}
    for q, (r, c) in enumerate(shapes):
        k = min(r, c)
        def orth(n):
            x = rng.standard_normal((n, k))
            if dtype == np.complex128:
                x = x + 1j * rng.standard_normal((n, k))
            return np.linalg.qr(x)[0]
        s = 10.0 ** (-decades * np.arange(k) / k) / (q + 1)
        blocks[q, q] = (orth(r) * s) @ orth(c).conj().T
    idx = [Index.make([((q,), s[i]) for q, s in enumerate(shapes)], (IN, OUT)[i]) for i in (0, 1)]
    return BlockTensorData(idx, blocks, dtype), blocks


def rebuilt(ctx, u, s, vt):  # noqa: F811
    return api.contract(ctx, api.contract(ctx, u, s, [1], [0]), vt, [1], [0]).to_data().blocks


@pytest.mark.parametrize("shapes", [((129, 300), (40, 65)), ((260, 193), (64, 64))])
def test_randomized_svd(ctx, shapes):  # noqa: F811
    """Products that add to their result (the residuals) run on the FMAs whatever
    the form; the truncated matrix is the exact SVD's to the sketch's accuracy."""
    t, _ = two_sectors(shapes, 8, sum(shapes[0]))
    d = api.DeviceTensor.from_data(ctx, t)
    u, s, vt, err, kept = api.svd(ctx, d, 1, (0,), 1e-10, 1, 1000)
    x, y, z, err2, kept2, _ = api.svd_randomized(ctx, d, 1, (0,), 1e-10, 1, 1000,
                                                 [((q,), 30) for q in range(2)])
    assert kept == kept2 and abs(err - err2) <= 1e-12
    a, b = rebuilt(ctx, u, s, vt), rebuilt(ctx, x, y, z)
    for k in a:
        assert np.abs(a[k] - b[k]).max() <= 1e-6


@pytest.mark.parametrize("m,n", [(60000, 8), (8, 60000)])
def test_narrow_out_of_range_product(ctx, m, n):  # noqa: F811
    """An operand outside the range, narrow result: the FMAs' result bit for bit, from
    tiles of its shape (64 x 64 ones would take four times the work): not three
    times as long as the FMA form itself, at a K that leaves the plan's host time
    behind."""
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((m, 1024)), rng.standard_normal((1024, n))
    (a if m > n else b)[3, 5] = 1e200
    x, y = (api.DeviceTensor.from_data(ctx, dense(v, (IN, OUT))) for v in (a, b))

    def timed(form):
        ctx.set_gemm_form(form)
        best = 1e9
        for _ in range(8):
            ctx.sync()
            t = time.perf_counter()
            c = api.contract(ctx, x, y, [1], [0])
            ctx.sync()
            best = min(best, time.perf_counter() - t)
        return best, c.download_packed()

    t0, want = timed(0)
    t1, got = timed(1)
    assert np.array_equal(got, want)
    assert t1 <= 3 * t0, (t0, t1)
