"""The sliced FP64 GEMM at the ends of its range and on the calls that reach it in
other ways than a plain contraction."""
import time

import numpy as np
import pytest

from test_gpu_slice import check, ctx, dense, product  # noqa: F401
from ultradmrg_gb300 import api
from ultradmrg_gb300 import models as M
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


# ---- the calls that reach the form in other ways --------------------------------

@pytest.mark.parametrize("k", [1153, 2501])
def test_complex_k_parts(ctx, k):  # noqa: F811
    """Few tiles of a long complex contraction, whose embedded K is cut into parts."""
    rng = np.random.default_rng(k)
    a = rng.standard_normal((70, k)) + 1j * rng.standard_normal((70, k))
    b = rng.standard_normal((k, 33)) + 1j * rng.standard_normal((k, 33))
    check(product(ctx, a, b), a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("shapes", [((63, 129), (65, 64)), ((128, 300), (200, 127)),
                                    ((257, 193), (30, 7)), ((320, 320), (160, 131))])
@pytest.mark.parametrize("mode", [api.SVD_SPLIT_LEFT, api.SVD_SPLIT_RIGHT])
def test_svd_products(ctx, shapes, dtype, mode):  # noqa: F811
    """Gram products of the upper triangle, Newton-Schulz and factor products in the
    sliced form, at sizes around the tiles' edges and in both orientations.  Bounds
    of the Gram route: squared singular values to 1e-14 sqrt(n) of the largest, the
    factors' product (all states kept) to 1e-13 n of it."""
    t, blocks = two_sectors(shapes, 4, shapes[0][0] + shapes[1][1], dtype)
    u, s, vt, err, kept = api.svd(ctx, api.DeviceTensor.from_data(ctx, t), 1, (0,), 0.0, 1, 10000,
                                  mode)
    assert kept == sum(min(x) for x in shapes)
    sv = {k[0]: np.diag(b).real for k, b in s.to_data().blocks.items()}
    state = api.contract(ctx, u, vt, [1], [0]).to_data().blocks
    top = max(np.linalg.norm(b, 2) for b in blocks.values())
    got = np.sort(np.concatenate([sv[k] for k in sorted(sv)]))[::-1]
    want = np.sort(np.concatenate([np.linalg.svd(b, compute_uv=False)
                                   for b in blocks.values()]))[::-1]
    n = max(max(x) for x in shapes)
    assert np.abs(got ** 2 - want ** 2).max() <= 1e-14 * np.sqrt(n) * top ** 2
    for k, b in blocks.items():
        assert np.abs(state[k] - b).max() <= 1e-13 * n * top


@pytest.fixture(scope="module", params=[np.float64, np.complex128], ids=["real", "complex"])
def bond(request, ctx):  # noqa: F811
    """(L, W1, W2, R, two site tensors) at the centre of a 3 x 2 Hubbard cylinder."""
    dtype = request.param
    mpo, pb = M.hubbard_cylinder_mpo(3, 2, t=1.0, U=8.0, dtype=dtype)
    mps = M.random_canonical_mps([pb] * 6, (5, 1), 60, 2, seed=3, dtype=dtype)
    up = lambda t: api.DeviceTensor.from_data(ctx, t)  # noqa: E731
    ctx.set_gemm_form(0)
    L, R = api.build_envs(ctx, mpo, mps, 2)
    ctx.set_gemm_form(1)
    return L, up(mpo[2]), up(mpo[3]), R, up(mps[2]), up(mps[3])


def scaled(ctx, t, f):  # noqa: F811
    d = t.to_data()
    d.blocks = {k: v * f for k, v in d.blocks.items()}
    return api.DeviceTensor.from_data(ctx, d)


def both_forms(ctx, fn):  # noqa: F811
    out = []
    for form in (0, 1):
        ctx.set_gemm_form(form)
        out.append(fn().to_data().blocks)
    return out


def agree(x, y, tol):
    scale = max(np.abs(v).max() for v in x.values())
    assert scale > 0 and sorted(x) == sorted(y)
    for k in x:
        assert np.abs(x[k] - y[k]).max() <= tol * scale


@pytest.mark.parametrize("p", [0, -60, 300, -430])
def test_one_site_product(ctx, bond, p):  # noqa: F811
    """The one-site product, whose MPO step finds the last GEMM's scales, for states
    of several magnitudes in a row (at 2^-430 the scales that the step finds are
    outside the range, those of the state are not)."""
    L, w1, _, R1, a, _ = bond
    L = scaled(ctx, L, 2.0 ** -60) if p == -430 else L
    # its right environment: one more update from the two-site one
    ctx.set_gemm_form(0)
    R = api.update_site_renvs(ctx, R1, bond[5], bond[2])
    for q in (p, 0, p):
        x, y = both_forms(ctx, lambda: api.eff_ham_mul_single_site_state(
            ctx, [L, w1, R], scaled(ctx, a, 2.0 ** q)))
        agree(x, y, 1e-13)


def test_two_site_scales_out_of_range(ctx, bond):  # noqa: F811
    """A state and an environment inside the range whose product is not."""
    L, w1, w2, R, a, b = bond
    psi = api.contract(ctx, a, b, [2], [0])
    big = scaled(ctx, L, 2.0 ** -240)
    x, y = both_forms(ctx, lambda: api.eff_ham_mul_two_site_state(
        ctx, [big, w1, w2, R], scaled(ctx, psi, 2.0 ** -250)))
    agree(x, y, 1e-13)


def test_double_word_fallback(ctx, bond):  # noqa: F811
    """A sliced anchor whose operand is not finite: the double-word tiles' result."""
    L, w1, w2, R, a, b = bond
    psi = api.contract(ctx, a, b, [2], [0])
    bad = psi.to_data()
    k = sorted(bad.blocks)[len(bad.blocks) // 2]
    bad.blocks[k] = np.full_like(bad.blocks[k], np.inf)
    bad = api.DeviceTensor.from_data(ctx, bad)

    def run():
        plan = api.MatvecPlan(ctx, [L, w1, w2, R], psi, precision=api.PREC_MIXED)
        x, y = plan.embed(bad), plan.embed(psi)
        plan.apply_anchor(x, y)
        return y

    x, y = both_forms(ctx, run)
    for k in x:
        assert np.array_equal(np.isfinite(x[k]), np.isfinite(y[k]))
        ok = np.isfinite(x[k])
        assert np.abs(x[k][ok] - y[k][ok]).max(initial=0.0) <= 1e-12
