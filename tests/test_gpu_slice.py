"""Digit-sliced FP64 GEMM on the tensor cores against extended-precision sums.

The bound per output is derived from the splitting: the digits of both
operands end 2^-63 below their line's power-of-two scale (up to twice the
line's maximum), the dropped digit pairs sum below 2^-61 of the scales' product,
levels 4 .. 7 round below 2^-58 of it per step of sixteen products, and the
result is rounded once: |err| <= 2^-53 |c| + K 2^-57 rowmax colmax.
"""
import numpy as np
import pytest

from ultradmrg_gb300 import api
from ultradmrg_gb300 import models as M
from ultradmrg_gb300.tensor_data import IN, OUT, BlockTensorData, Index

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    c.set_gemm_form(1)
    yield c
    c.close()


def dense(a, dirs):
    idx = [Index.make([((0,), d)], s) for d, s in zip(a.shape, dirs)]
    return BlockTensorData(idx, {(0,) * a.ndim: a}, a.dtype.type)


def product(ctx, a, b):
    x = api.DeviceTensor.from_data(ctx, dense(a, (IN, OUT)))
    y = api.DeviceTensor.from_data(ctx, dense(b, (IN, OUT)))
    return api.contract(ctx, x, y, [1], [0]).to_data().blocks[0, 0]


def check(c, a, b):
    wide = np.clongdouble if np.iscomplexobj(a) else np.longdouble
    # long double has 64 bits on x86 and 113 on Arm: either is enough
    ref = a.astype(wide) @ b.astype(wide)
    parts = (lambda x: np.maximum(np.abs(x.real), np.abs(x.imag))) if np.iscomplexobj(a) else np.abs
    k = a.shape[1] * (2 if np.iscomplexobj(a) else 1)
    bound = 2.0 ** -53 * np.abs(ref) + k * 2.0 ** -57 * (
        parts(a).max(1)[:, None] * parts(b).max(0)[None, :])
    assert np.all(np.abs(c - ref) <= bound * (2 if np.iscomplexobj(a) else 1))


SIZES = [(1, 1, 1), (1, 300, 17), (129, 65, 16), (64, 128, 255), (127, 63, 256), (130, 257, 257),
         (66, 5, 513), (200, 190, 1031)]


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("cplx", [False, True])
def test_tile_edges(ctx, m, n, k, cplx):
    rng = np.random.default_rng(m + 7 * n + 13 * k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if cplx:
        a, b = a + 1j * rng.standard_normal((m, k)), b + 1j * rng.standard_normal((k, n))
    check(product(ctx, a, b), a, b)


@pytest.mark.parametrize("k", [376, 384, 400, 2047, 2305, 5001])
def test_k_parts(ctx, k):
    """Few tiles of a long contraction: split over K parts of at least 256."""
    rng = np.random.default_rng(k)
    a, b = rng.standard_normal((130, k)), rng.standard_normal((k, 33))
    check(product(ctx, a, b), a, b)


@pytest.mark.parametrize("kind", ["ones", "graded", "scaled", "zero_rows", "powers"])
def test_values(ctx, kind):
    rng = np.random.default_rng(5)
    m, n, k = 150, 140, 300
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if kind == "ones":  # every digit product of one sign: the largest exact sums
        a, b = np.full((m, k), 1 - 2.0 ** -53), np.full((k, n), -1 + 2.0 ** -53)
    elif kind == "graded":
        a, b = a * 10.0 ** -np.linspace(0, 12, k), b * 10.0 ** -np.linspace(0, 9, k)[:, None]
    elif kind == "scaled":
        a, b = a * 2.0 ** rng.integers(-300, 300, (m, 1)), b * 2.0 ** rng.integers(-100, 100, (1, n))
    elif kind == "zero_rows":
        a[3], b[:, 7] = 0.0, 0.0
    else:
        a, b = np.exp2(rng.integers(-40, 40, (m, k)).astype(float)), -np.exp2(
            rng.integers(-3, 3, (k, n)).astype(float))
    check(product(ctx, a, b), a, b)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e200, 1e-200])
def test_out_of_range_operands_take_the_fp64_form(ctx, bad):
    """Non-finite values and lines beyond the sliced range: the FP64 kernels'
    result, bit for bit."""
    rng = np.random.default_rng(6)
    a, b = rng.standard_normal((140, 90)), rng.standard_normal((90, 70))
    a[17] = bad if abs(bad) < 1 else a[17]
    a[17, 3] = bad
    got = product(ctx, a, b)
    ctx.set_gemm_form(0)
    try:
        want = product(ctx, a, b)
    finally:
        ctx.set_gemm_form(1)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
def test_block_sparse_forms_agree(ctx, dtype):
    """Every contraction of a two-site product and of both environment updates,
    in either form (the oracle tests cover the FP64 one): merged groups, absent
    blocks, strided axes."""
    mpo, pb = M.hubbard_cylinder_mpo(3, 2, t=1.0, U=8.0, dtype=dtype)
    mps = M.random_canonical_mps([pb] * 6, (5, 1), 60, 2, seed=3, dtype=dtype)
    out = {}
    for form in (0, 1):
        ctx.set_gemm_form(form)
        ten = [[api.DeviceTensor.from_data(ctx, t) for t in x] for x in (mps, mpo)]
        L, R = (api.DeviceTensor.from_data(ctx, api.trivial_env_data(mps[i], mpo[i], s))
                for i, s in ((0, "l"), (5, "r")))
        for i in (0, 1):
            L = api.update_site_lenvs(ctx, L, ten[0][i], ten[1][i])
            R = api.update_site_renvs(ctx, R, ten[0][5 - i], ten[1][5 - i])
        w1, w2 = (api.DeviceTensor.from_data(ctx, mpo[i]) for i in (2, 3))
        psi = api.contract(ctx, api.DeviceTensor.from_data(ctx, mps[2]),
                           api.DeviceTensor.from_data(ctx, mps[3]), [2], [0])
        hp = api.eff_ham_mul_two_site_state(ctx, [L, w1, w2, R], psi)
        out[form] = [t.to_data() for t in (L, R, psi, hp)]
    ctx.set_gemm_form(1)
    for x, y in zip(out[0], out[1]):
        assert sorted(x.blocks) == sorted(y.blocks)
        scale = max(np.abs(v).max() for v in x.blocks.values())
        for k in x.blocks:
            assert np.abs(x.blocks[k] - y.blocks[k]).max() <= 1e-13 * scale


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
def test_scales_from_the_mpo_step(ctx, dtype):
    """The product on a plan, where the MPO step finds the scales of the last
    GEMM's operand: against the FP64 form, and linear in the state bit for bit
    under powers of two (scales left over from a larger state would show)."""
    mpo, pb = M.hubbard_cylinder_mpo(3, 2, t=1.0, U=8.0, dtype=dtype)
    mps = M.random_canonical_mps([pb] * 6, (5, 1), 60, 2, seed=3, dtype=dtype)
    out = {}
    for form in (0, 1):
        ctx.set_gemm_form(form)
        ten = [[api.DeviceTensor.from_data(ctx, t) for t in x] for x in (mps, mpo)]
        L, R = (api.DeviceTensor.from_data(ctx, api.trivial_env_data(mps[i], mpo[i], s))
                for i, s in ((0, "l"), (5, "r")))
        for i in (0, 1):
            L = api.update_site_lenvs(ctx, L, ten[0][i], ten[1][i])
            R = api.update_site_renvs(ctx, R, ten[0][5 - i], ten[1][5 - i])
        psi = api.contract(ctx, ten[0][2], ten[0][3], [2], [0])
        plan = api.MatvecPlan(ctx, [L, ten[1][2], ten[1][3], R], psi)
        for p in (0, -40, 7):
            data = psi.to_data()
            data.blocks = {k: v * 2.0 ** p for k, v in data.blocks.items()}
            x = plan.embed(api.DeviceTensor.from_data(ctx, data))
            y = plan.embed(psi)
            plan.apply(x, y)
            out[form, p] = y.to_data().blocks
    ctx.set_gemm_form(1)
    scale = max(np.abs(v).max() for v in out[0, 0].values())
    for k, v in out[1, 0].items():
        assert np.abs(v - out[0, 0][k]).max() <= 1e-13 * scale
        for p in (-40, 7):
            assert np.array_equal(out[1, p][k], v * 2.0 ** p)
