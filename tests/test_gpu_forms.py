"""What the choice of a form must not change: results that a mixed Krylov run
amplifies keep one summation order whatever the cost rule takes elsewhere."""
import json
import os

import numpy as np
import pytest

from ultradmrg_gb300 import _lib, api
from ultradmrg_gb300 import models as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ultradmrg_gb300 import build
    build.build()
    c = api.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def problem(ctx):
    """Centre bond of a Hubbard cylinder, large enough that the cost rule slices."""
    mpo, pb = M.hubbard_cylinder_mpo(4, 4, t=1.0, U=8.0, builder="reference")
    mps = M.random_mps([pb] * 16, (14, 0), 400, seed=5, sigma=2.0)
    L, R = api.build_envs(ctx, mpo, mps, 7)
    ten = [api.DeviceTensor.from_data(ctx, t) for t in (mps[7], mps[8], mpo[7], mpo[8])]
    psi = api.contract(ctx, ten[0], ten[1], [2], [0])
    return [L, ten[2], ten[3], R], psi, ten[:2]


def in_form(ctx, form, fn):
    old = ctx.gemm_form()
    ctx.set_gemm_form(form)
    try:
        return fn()
    finally:
        ctx.set_gemm_form(old)


def test_mixed_anchor_keeps_its_order(ctx, problem):
    """The double-word anchor under the cost rule is the FMA form's, bit for bit,
    at a size where the rule slices the plain product."""
    eff, psi, _ = problem

    def products(precision, anchor):
        plan = api.MatvecPlan(ctx, eff, psi, precision=precision)
        x, y = plan.embed(psi), plan.embed(psi)
        (plan.apply_anchor if anchor else plan.apply)(x, y)
        return y.download_packed()

    rule, fma = (in_form(ctx, f, lambda: products(api.PREC_MIXED, True)) for f in (-1, 0))
    assert np.array_equal(rule, fma)
    rule, fma = (in_form(ctx, f, lambda: products(api.PREC_FP64, False)) for f in (-1, 0))
    assert not np.array_equal(rule, fma)  # (the rule does slice here)


def test_mixed_solve_keeps_its_order(ctx, problem):
    """So a whole mixed solve does not depend on the rule."""
    eff, psi, _ = problem

    def solve():
        r = api.lanczos_solver(ctx, eff, psi, 1e-9, 100, precision=api.PREC_MIXED)
        return r.gs_eng, r.gs_vec.download_packed()

    (e0, v0), (e1, v1) = (in_form(ctx, f, solve) for f in (-1, 0))
    assert e0 == e1 and np.array_equal(v0, v1)


# ---- small sectors of the SVD ---------------------------------------------------

def exact_gram(n, rank):
    """Z D Z^T of small integers and powers of two: exact in FP64, its smallest
    eigenvalues up to 2^-32 of the largest."""
    rng = np.random.default_rng(100 * n + rank)
    z = rng.integers(-64, 65, (n, rank)) * 2.0 ** -np.sort(rng.integers(0, 17, rank))
    return z @ z.T


def sym_eig(ctx, mats):
    ns = np.array([m.shape[0] for m in mats], np.int32)
    flat = np.concatenate([m.ravel() for m in mats])
    lam, vec = np.zeros(int(ns.sum())), np.zeros(flat.size)
    ptr = lambda a, t: a.ctypes.data_as(t)  # noqa: E731
    _lib.call("udmrg_selftest_sym_eig", ctx.h, len(mats), ptr(ns, _lib.c_int32_p),
              ptr(flat, _lib.c_double_p), ptr(ns, _lib.c_int32_p), ptr(lam, _lib.c_double_p),
              ptr(vec, _lib.c_double_p))
    cut = np.cumsum(ns)[:-1]
    return [(w, v.reshape(len(w), -1)) for w, v in
            zip(np.split(lam, cut), np.split(vec, np.cumsum(ns.astype(int) ** 2)[:-1]))]


def test_small_sectors_keep_their_order(ctx):
    """Up to 32 rows the eigenvalues are the one-CTA reduction's bit for bit
    (recorded from it), and so is, up to the rounding of the projection itself,
    the space of the leading vectors.  The lowest of these eigenvalues lie 2^-32
    below the largest: another order of any sum in the reduction turns the space
    by about 2^-53 2^32."""
    path = os.path.join(os.path.dirname(__file__), "golden", "sym_eig_ordered.json")
    gold = json.load(open(path))
    sizes = [tuple(map(int, k.split())) for k in gold]
    for (n, rank), (lam, z), g in zip(sizes, sym_eig(ctx, [exact_gram(*s) for s in sizes]),
                                      gold.values()):
        assert np.array_equal(lam, [float.fromhex(v) for v in g["lam"]]), n
        z, x = z[:, :rank], np.arange(1, n + 1) / n
        px = np.array([float.fromhex(v) for v in g["px"]])
        assert np.abs(z @ (z.T @ x) - px).max() <= 1e-13 * np.linalg.norm(x), n


# ---- environments ---------------------------------------------------------------

def _chain():
    mpo, pb = M.hubbard_cylinder_mpo(4, 4, t=1.0, U=8.0, builder="reference")
    return mpo, M.random_mps([pb] * 16, (14, 0), 250, seed=6, sigma=2.0)


def test_build_envs_keeps_a_chosen_form(ctx):
    """build_envs: FMAs under the rule, the caller's form where one is set (the
    context's own updates, one by one)."""
    mpo, mps = _chain()

    def built():
        return [t.download_packed() for t in api.build_envs(ctx, mpo, mps, 7, normalize=False)]

    def grown():
        out = []
        for side, sites, grow in (("l", range(7), api.update_site_lenvs),
                                  ("r", range(15, 8, -1), api.update_site_renvs)):
            end = 0 if side == "l" else 15
            e = api.DeviceTensor.from_data(ctx, api.trivial_env_data(mps[end], mpo[end], side))
            for i in sites:
                e = grow(ctx, e, *(api.DeviceTensor.from_data(ctx, t) for t in (mps[i], mpo[i])))
            out.append(e.download_packed())
        return out

    for form, like in ((-1, 0), (0, 0), (1, 1)):
        for x, y in zip(in_form(ctx, form, built), in_form(ctx, like, grown)):
            assert np.array_equal(x, y), form


def test_mixed_solve_from_either_environments(ctx):
    """A mixed solve from environments of FMAs and of slices: Ritz values that move
    less than 1e-10 in their last step, so the energies agree to a hundred such
    steps."""
    mpo, mps = _chain()
    ten = [api.DeviceTensor.from_data(ctx, t) for t in (mps[7], mps[8], mpo[7], mpo[8])]
    psi = in_form(ctx, 0, lambda: api.contract(ctx, ten[0], ten[1], [2], [0]))
    e = []
    for form in (0, 1):
        L, R = in_form(ctx, form, lambda: api.build_envs(ctx, mpo, mps, 7, normalize=False))
        e.append(api.lanczos_solver(ctx, [L, ten[2], ten[3], R], psi, 1e-10, 100,
                                    precision=api.PREC_MIXED).gs_eng)
    assert abs(e[0] - e[1]) <= 1e-8
