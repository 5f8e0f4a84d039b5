"""The sliced FP64 GEMM at the ends of its range and on the calls that reach it in
other ways than a plain contraction."""
import numpy as np
import pytest

from test_gpu_slice import ctx, product  # noqa: F401
from ultradmrg_gb300 import api

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
