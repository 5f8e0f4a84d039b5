"""The work that users of this framework have it do, as cases that can be timed.

A case is one call (or the few calls that belong together) of the two-site
DMRG / TDVP update: the effective-Hamiltonian product on a plan, a whole
Lanczos or Krylov-exponential solve, an environment grown by one site, a
truncated SVD, and one whole local update.  The problems are those of the
benchmark configurations (Fermi-Hubbard cylinder of width 4 at 1/8 doping with
U(1)xU(1), the S = 1/2 Heisenberg chain and the two-leg ladder under TDVP with
U(1)), over their range of bond dimensions, in both element types and both
matvec forms.  Chains are cut to the length at which the centre bond still
reaches the asked bond dimension: the two-site problem there has the sectors
and MPO channels of the long chain.

States and environments: MPS tensors are random isometries with the sector
sizes of ``models.bond_sectors``, the environments are grown from them, and
two-site states have a Schmidt spectrum that decays over five decades.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ultradmrg_gb300 import api, models as M
from ultradmrg_gb300.tensor_data import BlockTensorData

PREC = {"fp64": api.PREC_FP64, "mixed": api.PREC_MIXED}
SITES = {"hubbard": 16, "heisenberg": 20, "ladder": 22}
LANCZOS = (1e-9, 100)  # tolerance and Krylov limit of the ground-state configurations
EXPMV = (1e-10, 20)    # of the time evolution
TAU_HALF = 0.025       # half of its time step
TRUNC = 1e-8

# case fields: op, model, D, and form (matvec) or side (environment, update)


def listed():
    return [
        # the smallest product: early sweeps and short chains, launch latency
        dict(name="heff_mixed_heis_d64", op="heff", model="heisenberg", D=64, form="mixed"),
        # the product inside the ground-state solver while a sweep schedule grows D
        dict(name="heff_mixed_hub_d701", op="heff", model="hubbard", D=701, form="mixed"),
        # ... and at the headline size
        dict(name="heff_mixed_hub_d2000", op="heff", model="hubbard", D=2000, form="mixed"),
        # the product inside the time evolution (complex128)
        dict(name="heff_mixed_ladder_d512", op="heff", model="ladder", D=512, form="mixed"),
        # the plain double-precision product
        dict(name="heff_fp64_hub_d1000", op="heff", model="hubbard", D=1000, form="fp64"),
        # a whole ground-state solve, double precision
        dict(name="lanczos_fp64_heis_d256", op="lanczos", model="heisenberg", D=256, form="fp64"),
        # a whole Krylov exponential of the time evolution, double precision
        dict(name="expmv_fp64_ladder_d512", op="expmv", model="ladder", D=512, form="fp64"),
        # environments grown to the right and to the left
        dict(name="env_l_hub_d2000", op="env", model="hubbard", D=2000, side="l"),
        dict(name="env_r_ladder_d333", op="env", model="ladder", D=333, side="r"),
        # truncated SVDs: a ground-state update (right move), a time step (left move)
        dict(name="svd_r_hub_d2000", op="svd", model="hubbard", D=2000, side="r"),
        dict(name="svd_l_ladder_d511", op="svd", model="ladder", D=511, side="l"),
        # one whole local update of the headline sweep
        dict(name="update_mixed_hub_d2000", op="update", model="hubbard", D=2000, form="mixed",
             side="r"),
    ]


def draw(rng):
    op = rng.choice(["heff", "heff", "lanczos", "expmv", "env", "svd", "update"])
    model = rng.choice(["hubbard", "heisenberg"] if op in ("lanczos", "update")
                       else ["ladder"] if op == "expmv"
                       else ["hubbard", "heisenberg", "ladder"])
    form = rng.choice(["fp64", "mixed"])
    top = {"hubbard": 2000, "heisenberg": 400, "ladder": 512}[model]
    if op in ("lanczos", "update") and form == "fp64":
        top = min(top, 400)  # a double-precision solve at 2000 costs more than any listed case
    D = int(round(math.exp(rng.uniform(math.log(48), math.log(top)))))
    case = dict(op=op, model=model, D=D)
    if op in ("heff", "lanczos", "expmv", "update"):
        case["form"] = form
    if op in ("env", "svd", "update"):
        case["side"] = rng.choice(["l", "r"])
    return case


# ---- the problem of a case ------------------------------------------------------

_ctx = []
_mpos = {}


def _context():
    if not _ctx:
        _ctx.append(api.Context(0))
    return _ctx[0]


def _model(model):
    """(MPO, physical index, divergence, element type): independent of seed and D."""
    if model not in _mpos:
        n = SITES[model]
        if model == "hubbard":
            mpo, pb = M.hubbard_cylinder_mpo(n // 4, 4, t=1.0, U=8.0, builder="reference")
            _mpos[model] = mpo, pb, (n - n // 8, 0), np.float64
        elif model == "heisenberg":
            mpo, pb = M.heisenberg_chain_mpo(n, builder="reference")
            _mpos[model] = mpo, pb, (0,), np.float64
        else:
            mpo, pb = M.heisenberg_chain_mpo(n, dtype=np.complex128,
                                             pairs=M.heisenberg_ladder_pairs(n // 2, 2),
                                             builder="reference")
            _mpos[model] = mpo, pb, (0,), np.complex128
    return _mpos[model]


def _isometry(A, left):
    """Block tensor A made a left (right) isometry: QR per sector of its open bond."""
    ax = 2 if left else 0
    groups = {}
    for k in sorted(A.blocks):
        groups.setdefault(k[ax], []).append(k)
    for keys in groups.values():
        if left:
            m = np.concatenate([A.blocks[k].reshape(-1, A.blocks[k].shape[2]) for k in keys], 0)
        else:
            m = np.concatenate([A.blocks[k].reshape(A.blocks[k].shape[0], -1) for k in keys], 1).T
        q = torch.linalg.qr(torch.from_numpy(np.ascontiguousarray(m)).cuda())[0].cpu().numpy()
        full = np.zeros_like(m)
        full[:, :q.shape[1]] = q
        full = full if left else full.T
        off = 0
        for k in keys:
            shp = A.blocks[k].shape
            if left:
                A.blocks[k] = full[off:off + shp[0] * shp[1]].reshape(shp)
                off += shp[0] * shp[1]
            else:
                A.blocks[k] = np.ascontiguousarray(full[:, off:off + shp[1] * shp[2]]).reshape(shp)
                off += shp[1] * shp[2]


def _decay(dims, decades):
    return [10.0 ** (-decades * np.arange(d) / max(d, 1)) * (d / max(dims)) for d in dims]


def _problem(case, seed, envs=True, centre=None):
    """Host tensors of the two-site problem at the centre bond."""
    mpo, pb, div, dtype = _model(case["model"])
    n = len(mpo)
    l = n // 2 - 1
    mps = M.random_mps([pb] * n, div, case["D"], seed=seed, dtype=dtype, sigma=2.0)
    for i in range(n):
        if envs or i in (l, l + 1):
            _isometry(mps[i], i <= l)
    # the Schmidt weights of the centre bond, on its right tensor
    w = _decay(mps[l].indexes[2].dims, 5.0)
    for k in mps[l + 1].blocks:
        mps[l + 1].blocks[k] = mps[l + 1].blocks[k] * w[k[0]][:, None, None]
    nrm = mps[l + 1].norm()
    for k in mps[l + 1].blocks:
        mps[l + 1].blocks[k] = mps[l + 1].blocks[k] / nrm
    return mpo, mps, l


def _two_site_state(mps_l, mps_r, seed):
    """A unit two-site state on every block the symmetry allows, graded over the
    two outer bonds as a solver's ground state is (its singular values decay
    over five decades)."""
    idx = [mps_l.indexes[0], mps_l.indexes[1], mps_r.indexes[1], mps_r.indexes[2]]
    div = tuple(x + y for x, y in zip(mps_l.div(), mps_r.div()))
    rng = np.random.default_rng(1000 + seed)
    psi = BlockTensorData(idx, {}, mps_l.dtype)
    wa, wb = _decay(idx[0].dims, 2.5), _decay(idx[3].dims, 2.5)
    for a in range(idx[0].nsec):
        for s in range(idx[1].nsec):
            for t in range(idx[2].nsec):
                for b in range(idx[3].nsec):
                    if psi.block_qn_sum((a, s, t, b)) != div:
                        continue
                    x = rng.standard_normal(psi.block_shape((a, s, t, b)))
                    if psi.dtype == np.complex128:
                        x = x + 1j * rng.standard_normal(x.shape)
                    psi.blocks[a, s, t, b] = (x * wa[a][:, None, None, None] * wb[b]).astype(psi.dtype)
    nrm = psi.norm()
    for k in psi.blocks:
        psi.blocks[k] = psi.blocks[k] / nrm
    return psi


def prepare(case, seed):
    ctx = _context()
    put = lambda t: api.DeviceTensor.from_data(ctx, t)  # noqa: E731
    op = case["op"]
    mpo, mps, l = _problem(case, seed, envs=op != "svd")
    st = dict(case=case, ctx=ctx)
    if op == "svd":
        psi = _two_site_state(mps[l], mps[l + 1], seed)
        st.update(psi=put(psi), size=psi.size(), ldiv=tuple(mps[l].div()))
        return st
    L, R = api.build_envs(ctx, mpo, mps, l)
    if op == "env":
        site = l if case["side"] == "l" else l + 1
        st.update(env=L if case["side"] == "l" else R, mps=put(mps[site]), mpo=put(mpo[site]))
        return st
    st["eff"] = [L, put(mpo[l]), put(mpo[l + 1]), R]
    if op == "update":
        st.update(mps_l=put(mps[l]), mps_r=put(mps[l + 1]), size=int(_size(_structure(case)[2])))
        return st
    st["psi"] = put(_two_site_state(mps[l], mps[l + 1], seed))
    if op == "heff":
        st["plan"] = api.MatvecPlan(ctx, st["eff"], st["psi"], precision=PREC[case["form"]])
        st["x"] = st["plan"].embed(st["psi"])
        st["y"] = st["plan"].embed(st["psi"])
    return st


class _DeviceArray:
    """A device tensor's packed buffer for ``torch.as_tensor`` (no copy)."""

    def __init__(self, t):
        inf = t.info()
        self.owner = t
        self.__cuda_array_interface__ = dict(
            shape=(inf["size"],), typestr="<c16" if inf["dtype"] == api.C128 else "<f8",
            data=(t.device_ptr(), False), version=2)


def _view(t):
    return torch.as_tensor(_DeviceArray(t), device="cuda")


def _split(ctx, u, vt, size):
    # the factors of an SVD are fixed up to a sign (a rotation, a phase) of each
    # singular pair; the two-site state they make is not.  It has the blocks of
    # the kept sectors, so its length follows the data: zeros up to that of all
    # sectors
    state = api.contract(ctx, u, vt, [2], [0])
    ctx.sync()  # torch reads it on a stream of its own
    return _padded(_view(state), size)


def _padded(x, size):
    return torch.nn.functional.pad(x, (0, size - x.numel()))


def _values(s):
    """The singular values on the diagonals of s's blocks."""
    x = _view(s)
    return x[x > 0]


def run(state):
    case, ctx = state["case"], state["ctx"]
    op = case["op"]
    if op == "heff":
        state["plan"].apply(state["x"], state["y"])
        return _view(state["y"])
    if op == "lanczos":
        r = api.lanczos_solver(ctx, state["eff"], state["psi"], *LANCZOS,
                               precision=PREC[case["form"]])
        return [r.gs_eng, _view(r.gs_vec)]
    if op == "expmv":
        _, v = api.lanczos_expmv_solver(ctx, state["eff"], state["psi"], TAU_HALF, *EXPMV,
                                        precision=PREC[case["form"]])
        return _view(v)
    if op == "env":
        grow = api.update_site_lenvs if case["side"] == "l" else api.update_site_renvs
        return _view(grow(ctx, state["env"], state["mps"], state["mpo"]))
    if op == "svd":
        mode = api.SVD_SPLIT_LEFT if case["side"] == "r" else api.SVD_SPLIT_RIGHT
        u, s, vt, err, D = api.svd(ctx, state["psi"], 2, state["ldiv"], TRUNC, 1, case["D"], mode)
        return [_split(ctx, u, vt, state["size"]), _values(s), err, D]
    L, w1, w2, R = state["eff"]
    p = api.FiniteVMPSSweepParams(1, 1, case["D"], TRUNC, *LANCZOS, precision=PREC[case["form"]])
    a, b, env, log = api.two_site_update(ctx, L, R, state["mps_l"], state["mps_r"], w1, w2, p,
                                         case["side"])
    # the grown environment, in the new bond's basis: through the one-site
    # product of the new centre tensor, put back into the two-site space
    if case["side"] == "r":
        c = api.eff_ham_mul_single_site_state(ctx, [env, w2, R], b)
        c = api.contract(ctx, a, c, [2], [0])
    else:
        c = api.eff_ham_mul_single_site_state(ctx, [L, w1, env], a)
        c = api.contract(ctx, c, b, [2], [0])
    size = state["size"]
    return [_split(ctx, a, b, size), _padded(_view(c), size), log["e0"], log["trunc_err"], log["D"]]


# ---- plain block-sparse contraction (torch, 64 bits) ------------------------------

def _contract(A, B, ca, cb, fa, fb):
    """Blocks {key: tensor} of A and B contracted over axes ca, cb; the output's
    axes are fa of A, then fb of B.  Blocks that are shapes give their flops."""
    by = {}
    for kb in B:
        by.setdefault(tuple(kb[i] for i in cb), []).append(kb)
    out, flops = {}, 0.0
    for ka, x in A.items():
        for kb in by.get(tuple(ka[i] for i in ca), ()):
            y = B[kb]
            ko = tuple(ka[i] for i in fa) + tuple(kb[i] for i in fb)
            if isinstance(x, tuple):
                out[ko] = tuple(x[i] for i in fa) + tuple(y[i] for i in fb)
                flops += 2.0 * math.prod(x) * math.prod(y[i] for i in fb)
                continue
            z = torch.tensordot(x, y, (ca, cb))
            # tensordot leaves the free axes in ascending order
            ra, rb = sorted(fa), sorted(fb)
            z = z.permute([ra.index(i) for i in fa] + [len(ra) + rb.index(i) for i in fb])
            out[ko] = out[ko] + z if ko in out else z
    return out, flops


def _dag(A):
    return {k: x.conj() if not isinstance(x, tuple) else x for k, x in A.items()}


def _heff(L, W1, W2, R, psi):
    t, f1 = _contract(L, psi, [2], [0], [0, 1], [1, 2, 3])       # a' w s1 s2 b
    t, _ = _contract(t, W1, [1, 2], [0, 1], [3, 4, 0], [2, 3])   # s2 b a' s1' w1
    t, _ = _contract(t, W2, [4, 0], [0, 1], [1, 2, 3], [2, 3])   # b a' s1' s2' w2
    t, f2 = _contract(t, R, [4, 0], [1, 2], [1, 2, 3], [0])      # a' s1' s2' b'
    return t, f1 + f2


def _env(side, E, A, W):
    if side == "l":
        t, f1 = _contract(E, A, [2], [0], [0, 1], [1, 2])                # a' w s b
        t, _ = _contract(t, W, [1, 2], [0, 1], [3, 0], [2, 3])           # b a' s' w'
        t, f2 = _contract(_dag(A), t, [0, 1], [1, 2], [2], [3, 0])       # b' w' b
    else:
        t, f1 = _contract(_dag(A), E, [2], [0], [0, 1], [1, 2])          # a' s' w b
        t, _ = _contract(t, W, [1, 2], [2, 3], [3, 0], [0, 1])           # b a' w0 s
        t, f2 = _contract(t, A, [3, 0], [1, 2], [1, 2], [0])             # a' w0 a
    return t, f1 + f2


def _blocks(t):
    d = t.to_data() if isinstance(t, api.DeviceTensor) else t
    return {k: torch.from_numpy(np.ascontiguousarray(b)).cuda() for k, b in d.blocks.items()}


def _pack(blocks, like=None):
    """One flat tensor, blocks in the order of their keys (those of `like`, zeros
    where there is none)."""
    return torch.cat([(blocks[k] if k in blocks else torch.zeros_like(like[k])).reshape(-1)
                      for k in sorted(like if like is not None else blocks)])


def _sectors(psi, div_l):
    """Bond sectors of a two-site tensor: {QN: (row keys, column keys)}."""
    secs = {}
    for k in psi.sorted_keys():
        q = tuple(d - sum(psi.indexes[i].qns[k[i]][c] * psi.indexes[i].dir for i in (0, 1))
                  for c, d in enumerate(div_l))
        rows, cols = secs.setdefault(q, (set(), set()))
        rows.add(k[:2])
        cols.add(k[2:])
    return {q: (sorted(secs[q][0]), sorted(secs[q][1])) for q in sorted(secs)}


def _svd_exact(psi, div_l, D):
    found, vals = [], []
    for rows, cols in _sectors(psi, div_l).values():
        m = np.concatenate([np.concatenate([psi.blocks[r + c].reshape(
            math.prod(psi.block_shape(r + c)[:2]), -1) for c in cols], 1) for r in rows], 0)
        found.append((rows, cols, np.linalg.svd(m, full_matrices=False)))
        vals.append(found[-1][2][1])
    flat = sorted(((s, q, i) for q, v in enumerate(vals) for i, s in enumerate(v)),
                  key=lambda x: (-x[0], x[1], x[2]))
    w = np.array([s * s for s, _, _ in flat])
    tail = np.concatenate([np.cumsum(w[::-1])[::-1], [0.0]])
    kept = next((k for k in range(1, min(D, len(flat)) + 1) if tail[k] / tail[0] <= TRUNC),
                min(D, len(flat)))
    count = [0] * len(vals)
    for _, q, _ in flat[:kept]:
        count[q] += 1
    state, sv = {}, []
    for (rows, cols, (u, s, vt)), k in zip(found, count):
        if k == 0:
            continue
        m = (u[:, :k] * s[:k]) @ vt[:k]
        sv.append(s[:k])
        r0 = 0
        for r in rows:
            nr = math.prod(psi.block_shape(r + cols[0])[:2])
            c0 = 0
            for c in cols:
                nc = math.prod(psi.block_shape(rows[0] + c)[2:])
                state[r + c] = torch.from_numpy(np.ascontiguousarray(m[r0:r0 + nr, c0:c0 + nc]))
                c0 += nc
            r0 += nr
    return [_padded(_pack(state), psi.size()), np.concatenate(sv), float(tail[kept] / tail[0]),
            kept]


def _krylov(eff, psi, like, stop):
    """Three-term Lanczos from psi: (basis, diagonal, off-diagonal, stop's value)."""
    shapes = {k: v.shape for k, v in like.items()}

    def apply(v):
        out, off = {}, 0
        for k in sorted(shapes):
            n = math.prod(shapes[k])
            out[k] = v[off:off + n].reshape(shapes[k])
            off += n
        return _pack(_heff(*eff, out)[0], like)

    v = _pack(psi, like)
    basis, a, b = [v / torch.linalg.vector_norm(v)], [], []
    while True:
        g = apply(basis[-1])
        a.append(float(torch.vdot(basis[-1], g).real))
        g = g - a[-1] * basis[-1] - (b[-1] * basis[-2] if b else 0)
        got = stop(a, b)
        if got is not None:
            return basis, got
        b.append(float(torch.linalg.vector_norm(g)))
        basis.append(g / b[-1])


def _tridiagonal(a, b):
    return np.linalg.eigh(np.diag(a) + np.diag(b, 1) + np.diag(b, -1))


def exact(case, seed):
    op = case["op"]
    if op == "update" or (op in ("lanczos", "expmv") and
                          (case["model"] == "hubbard" or case.get("form") == "mixed")):
        return None  # minutes in this form, or another algorithm in 64 bits
    if op == "svd":
        _, mps, l = _problem(case, seed, envs=False)
        return _svd_exact(_two_site_state(mps[l], mps[l + 1], seed), mps[l].div(), case["D"])
    st = prepare(case, seed)
    if op == "env":
        return _pack(_env(case["side"], _blocks(st["env"]), _blocks(st["mps"]),
                          _blocks(st["mpo"]))[0])
    eff, psi = [_blocks(t) for t in st["eff"]], _blocks(st["psi"])
    if op == "heff":
        return _pack(_heff(*eff, psi)[0], psi)
    if op == "lanczos":
        last = []

        def energy(a, b):
            e = _tridiagonal(a, b)[0][0]
            done = (last and last[-1] - e < LANCZOS[0]) or len(a) == LANCZOS[1]
            last.append(e)
            return e if done else None

        return [float(_krylov(eff, psi, psi, energy)[1]), None]  # the vector's sign is free
    last = [np.zeros(1, complex)]

    def coefficients(a, b):
        w, z = _tridiagonal(a, b)
        c = z @ (np.exp(-1j * TAU_HALF * w) * z[0])
        far = np.linalg.norm(c - np.pad(last[0], (0, len(c) - len(last[0]))))
        last[0] = c
        return c if len(a) > 1 and (far < EXPMV[0] or len(a) == EXPMV[1]) else None

    basis, c = _krylov(eff, psi, psi, coefficients)
    return sum(complex(x) * v for x, v in zip(c, basis))


# ---- what a pass cannot do without -------------------------------------------------

def _shapes(t):
    return {k: t.block_shape(k) for k in t.blocks}


def _size(shapes):
    return float(sum(math.prod(s) for s in shapes.values()))


def _allowed(idx, div):
    """Shapes of every block that the symmetry allows on these indexes."""
    t = BlockTensorData(idx, {}, np.float64)
    keys = [()]
    for ind in idx:
        keys = [k + (s,) for k in keys for s in range(ind.nsec)]
    return {k: t.block_shape(k) for k in keys if t.block_qn_sum(k) == div}


_structs = {}


def _structure(case):
    """Shapes of the two-site problem's tensors (no data)."""
    key = case["model"], case["D"]
    if key not in _structs:
        mpo, pb, div, dtype = _model(case["model"])
        n = len(mpo)
        l = n // 2 - 1
        mps = M.random_mps([pb] * n, div, case["D"], seed=0, dtype=dtype, sigma=2.0)
        zero = tuple(0 for _ in div)
        A, B = mps[l], mps[l + 1]
        L = _allowed([A.indexes[0], mpo[l].indexes[0].inverse(), A.indexes[0].inverse()], zero)
        R = _allowed([B.indexes[2], mpo[l + 1].indexes[3].inverse(), B.indexes[2].inverse()], zero)
        psi = _allowed([A.indexes[0], A.indexes[1], B.indexes[1], B.indexes[2]],
                       tuple(x + y for x, y in zip(A.div(), B.div())))
        _structs[key] = (L, R, psi, _shapes(A), _shapes(B), _shapes(mpo[l]), _shapes(mpo[l + 1]),
                         A.div(), 4.0 if dtype == np.complex128 else 1.0,
                         16 if dtype == np.complex128 else 8, A, B)
    return _structs[key]


def work(case):
    """Flops of the large contractions and of the factorisations; bytes of the
    inputs and outputs.  Solves are counted with the Krylov steps that they take
    at least (a state near convergence: ten)."""
    L, R, psi, A, B, W1, W2, ldiv, cf, es, ta, tb = _structure(case)
    op = case["op"]
    heff = cf * (_contract(L, psi, [2], [0], [0, 1], [1, 2, 3])[1] +
                 _contract(psi, R, [3], [2], [0, 1, 2], [0, 1])[1])
    heff_bytes = es * (_size(L) + _size(R) + 2 * _size(psi))
    if op == "env":
        E, T, W = (L, A, W1) if case["side"] == "l" else (R, B, W2)
        out, f = _env(case["side"], E, T, W)
        return {"bytes": es * (_size(E) + _size(T) + _size(out)), "flops": cf * f}
    secs = {}
    for k, s in psi.items():
        q = tuple(ta.indexes[0].qns[k[0]][c] * ta.indexes[0].dir +
                  ta.indexes[1].qns[k[1]][c] * ta.indexes[1].dir for c in range(len(ldiv)))
        rows, cols = secs.setdefault(q, ({}, {}))
        rows[k[:2]], cols[k[2:]] = s[0] * s[1], s[2] * s[3]
    svd = cf * sum(4.0 * m * n * min(m, n) for m, n in
                   ((sum(r.values()), sum(c.values())) for r, c in secs.values()))
    if op == "svd":
        return {"bytes": es * 2 * _size(psi), "flops": svd}
    if op == "heff":
        return {"bytes": heff_bytes, "flops": heff}
    if op in ("lanczos", "expmv"):
        return {"bytes": heff_bytes, "flops": 10 * heff}
    E, T, W = (L, A, W1) if case["side"] == "r" else (R, B, W2)
    env = cf * _env("l" if case["side"] == "r" else "r", E, T, W)[1]
    return {"bytes": heff_bytes, "flops": 10 * heff + svd + env}
