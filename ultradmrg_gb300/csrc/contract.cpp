// Contraction planner: block matching by quantum numbers -> grouped GEMM.
#include <algorithm>
#include <map>

#include "gemm.hpp"

namespace udmrg {

GemmPlan::~GemmPlan() {
  if (ctx) ctx->free(d_block);
}

void GemmPlan::upload() {
  UploadBatch up(*ctx);
  const size_t os = up.add(segs), op = up.add(probs);
  size_t ot[kNumCfg];
  for (int c = 0; c < kNumCfg; ++c) ot[c] = up.add(tiles[c]);
  ctx->free(d_block);
  d_block = up.commit();
  d_segs = (GSeg *)(d_block + os);
  d_probs = (GProb *)(d_block + op);
  for (int c = 0; c < kNumCfg; ++c) d_tiles[c] = (GTile *)(d_block + ot[c]);
  if (sl && !sl->d_block) sl->upload();
}

static const int kCfgBM[kNumCfg] = {64, 256, 16, 32};
static const int kCfgBN[kNumCfg] = {64, 16, 256, 32};

void cyclic_axes(int ra, int rb, int a_start, int b_start, int n, std::vector<int> &ca,
                 std::vector<int> &cb, std::vector<int> &fa, std::vector<int> &fb) {
  ca.clear();
  cb.clear();
  fa.clear();
  fb.clear();
  for (int i = 0; i < n; ++i) {
    ca.push_back((a_start + i) % ra);
    cb.push_back((b_start + i) % rb);
  }
  for (int i = 0; i < ra - n; ++i) fa.push_back((a_start + n + i) % ra);
  for (int i = 0; i < rb - n; ++i) fb.push_back((b_start + n + i) % rb);
}

namespace {

struct SubDim {
  int64_t ext;
  int64_t sa, sb;  // strides in operand A / B (unused one = 0)
};

constexpr int kMaxRank = 8;

// Row-major strides of a block with the given sector ids.
void block_strides(const BTensor &T, int64_t b, int64_t *st) {
  const int r = T.rank();
  st[r - 1] = 1;
  for (int i = r - 2; i >= 0; --i) st[i] = st[i + 1] * T.dim_of(b, i + 1);
}

// Sector-id tuples packed 16 bits per axis, first axis in the highest bits,
// so integer order is the lexicographic order of the tuples.
using Key128 = unsigned __int128;

struct Match {
  Key128 okey;
  int64_t a, b;
};

// The tile configuration with the least padded work.  Policy 1 charges 32 x 32
// tiles (four outputs per thread) twice their padded work, so they are taken
// only where the larger tiles would pad more than twice as much.
int tile_cfg(int64_t M, int64_t N, int policy, double *padded = nullptr) {
  int best = 0;
  double bestw = 1e300;
  for (int c = 0; c < kNumCfg; ++c) {
    double w = (double)((M + kCfgBM[c] - 1) / kCfgBM[c] * kCfgBM[c]) *
               (double)((N + kCfgBN[c] - 1) / kCfgBN[c] * kCfgBN[c]);
    if (policy == 1 && c == kCfg32x32) w *= 2.0;
    if (w < bestw * 0.999) {
      bestw = w;
      best = c;
    }
  }
  if (padded) *padded = bestw;
  return best;
}

void add_tiles(GemmPlan &g, int32_t pid, int64_t M, int64_t N, int policy) {
  const int best = tile_cfg(M, N, policy);
  for (int64_t m0 = 0; m0 < M; m0 += kCfgBM[best])
    for (int64_t n0 = 0; n0 < N; n0 += kCfgBN[best])
      g.tiles[best].push_back({pid, (int32_t)m0, (int32_t)n0, 0});
}

}  // namespace

static void tile_all(GemmPlan &g);

namespace {

// One tile configuration for all problems: 64 x 64, or the one whose padded work
// is less by a quarter or more (32 x 32 charged twice: four outputs per thread).
int one_cfg(const GemmPlan &g) {
  double w[kNumCfg] = {0, 0, 0, 0};
  for (const GProb &p : g.probs) {
    double k = 0;
    for (int s = 0; s < p.nseg; ++s) k += g.segs[p.seg0 + s].K;
    for (int c = 0; c < kNumCfg; ++c)
      w[c] += k * (double)(((int64_t)p.M + kCfgBM[c] - 1) / kCfgBM[c] * kCfgBM[c]) *
              (double)(((int64_t)p.N + kCfgBN[c] - 1) / kCfgBN[c] * kCfgBN[c]);
  }
  w[kCfg32x32] *= 2.0;
  int best = kCfg64x64;
  for (int c = 1; c < kNumCfg; ++c)
    if (w[c] < (best == kCfg64x64 ? 0.75 * w[best] : w[best])) best = c;
  return best;
}

// Whether a tile holds entries on or above the diagonal.
bool reaches_diagonal(int cfg, int32_t m0, int32_t n0) { return m0 <= n0 + kCfgBN[cfg] - 1; }

constexpr int64_t up8(int64_t x) { return (x + 7) & ~(int64_t)7; }

// Estimated time of a plan's FP64 tiles: multiply-adds of the padded tiles
// (half of them for an upper triangle) at 0.5e12 per second (80% of the FP64
// pipe), four per complex one.
double fp64_seconds(const GemmPlan &g, bool cplx, bool upper) {
  double macs = 0;
  for (const GProb &p : g.probs) {
    double k = 0, area = 0;
    for (int s = 0; s < p.nseg; ++s) k += (double)((g.segs[p.seg0 + s].K + 15) / 16 * 16);
    tile_cfg(p.M, p.N, 0, &area);
    macs += k * area;
  }
  return 4e-6 + macs * (cplx ? 4.0 : 1.0) * (upper ? 0.5 : 1.0) / 0.5e12;
}

// Below this estimate the sliced form's three launches and its passes over
// the operands hardly pay (96^3: 43 us in FP64, 36 sliced; 64^3 takes 35), and
// its tables are not built.
constexpr double kSliceMin = 50e-6;

// Shorter contractions stay on the FMAs: their K fills less than half of one
// step, and cutting the large operand into digits costs what the products
// save.  FP64 / sliced form, device time: 40000 x 8 x 8 (rows, columns, K)
// 48 / 43 us, 40000 x 20 x 20 89 / 49, 40000 x 64 x 16 103 / 64; T1 with an MPO
// tensor, Hubbard D = 500 870 / 321 us, complex ladder D = 300 464 / 193.
constexpr double kSliceMinK = 8;
double mean_k(const GemmPlan &g) {  // mean summed K, weighted with the work
  double w = 0, wk = 0;
  for (const GProb &p : g.probs) {
    double k = 0;
    for (int s = 0; s < p.nseg; ++s) k += g.segs[p.seg0 + s].K;
    w += k * p.M * p.N;
    wk += k * k * p.M * p.N;
  }
  return w > 0 ? wk / w : 0.0;
}

// Sub-dimensions (extent, stride in doubles) of a block over some axes,
// row-major, merged where contiguous; false: more than four remain.
bool op_dims(const BTensor &T, int64_t b, const int64_t *st, const std::vector<int> &axes, int es,
             int32_t *ext, int64_t *str, int32_t *n) {
  int m = 0;
  int64_t e[kMaxRank], s[kMaxRank];
  for (int ax : axes) {
    const int64_t d = T.dim_of(b, ax);
    if (d == 1) continue;
    if (m > 0 && s[m - 1] == d * st[ax] * es) {
      e[m - 1] *= d;
      s[m - 1] = st[ax] * es;
    } else {
      e[m] = d;
      s[m++] = st[ax] * es;
    }
  }
  if (m > 4) return false;
  for (int i = 0; i < m; ++i) {
    ext[i] = (int32_t)e[i];
    str[i] = s[i];
  }
  *n = m;
  return true;
}

// The ops of one operand block (or strided matrix): `base` real; complex data
// [re | im] along K for operand A, rows (re, im) interleaved for operand B:
// [[re, -im], [im, re]], so that the real product is the interleaved complex
// one.  kh: K columns of the real half.
void add_ops(SlicePlan &sp, int group, SlOp base, bool cplx, int32_t kh) {
  if (!cplx) {
    base.rstep = 1;
    sp.add_op(group, base);
    return;
  }
  auto part = [&](int im, int32_t r0, int32_t rstep, int32_t k0, int neg) {
    SlOp o = base;
    o.src_off = base.src_off + im;
    o.r0 = base.r0 * rstep + r0;
    o.rstep = rstep;
    o.k0 = base.k0 + k0;
    o.neg = neg;
    sp.add_op(group, o);
  };
  if (base.src == 0) {
    part(0, 0, 1, 0, 0);
    part(1, 0, 1, kh, 0);
  } else {
    part(0, 0, 2, 0, 0);
    part(1, 0, 2, kh, 1);
    part(1, 1, 2, 0, 0);
    part(0, 1, 2, kh, 0);
  }
}

// Lines of C's rows (blk, m) and columns (blk, n, block width; two per complex
// column).
void push_rows(std::vector<SlLine> &v, int blk, int64_t M) {
  const size_t n0 = v.size();
  v.resize(n0 + M);
  for (int64_t m = 0; m < M; ++m) v[n0 + m] = {blk, (int32_t)m, 0, 0};
}
void push_cols(std::vector<SlLine> &v, int blk, int64_t N, int es) {
  const size_t n0 = v.size();
  v.resize(n0 + N * es);
  for (int64_t n = 0; n < N * es; ++n) v[n0 + n] = {blk, (int32_t)n, (int32_t)(N * es), 0};
}

// The sliced form of gemm_add_simple's problems: one group each.
std::unique_ptr<SlicePlan> slice_simple(const GemmPlan &g, bool cplx, bool upper) {
  auto sp = std::make_unique<SlicePlan>();
  sp->ctx = g.ctx;
  const int es = cplx ? 2 : 1;
  for (const GProb &p : g.probs) {
    const GSeg &s = g.segs[p.seg0];
    const int64_t kh = up8(s.K);
    std::vector<SlLine> rows, cols;
    push_rows(rows, 0, p.M);
    push_cols(cols, 0, p.N, es);
    const int id = sp->add_group({p.M, (int64_t)p.N * es, kh * es}, rows, cols, {p.c_off * es},
                                 upper);
    for (int side = 0; side < 2; ++side) {
      SlOp o{};
      o.src = side;
      o.src_off = (side ? s.b_off : s.a_off) * es;
      o.rows = side ? p.N : p.M;
      o.cols = s.K;
      o.nr = o.nk = 1;
      o.re[0] = o.rows;
      o.ke[0] = o.cols;
      o.rs[0] = (side ? s.b_ns[0] : s.a_ms[0]) * es;
      o.ks[0] = (side ? s.b_ks[0] : s.a_ks[0]) * es;
      if (o.cols) add_ops(*sp, id, o, cplx, (int32_t)kh);
    }
  }
  sp->finalize();
  return sp;
}

// The sliced form of a block contraction: blocks that share contracted
// sectors, directly or through others, form one dense group (with abelian
// charges: one quantum-number flow), its rows the A blocks' free sectors, its
// columns the B blocks', its K their common contracted sectors, each padded
// to a multiple of 8.  matches sorted by (output key, a, b); output o's block
// starts at coff[o].
std::unique_ptr<SlicePlan> slice_contract(const BTensor &A, const BTensor &B,
                                          const std::vector<int> &ca, const std::vector<int> &cb,
                                          const std::vector<int> &fa, const std::vector<int> &fb,
                                          const std::vector<Match> &matches,
                                          const std::vector<size_t> &mstart,
                                          const std::vector<int64_t> &coff) {
  const bool cplx = A.dtype == kC128;
  const int es = cplx ? 2 : 1;
  auto key_of = [](const BTensor &T, int64_t b, const std::vector<int> &axes) {
    Key128 k = 0;
    for (int ax : axes) k = (k << 16) | (Key128)T.key(b)[ax];
    return k;
  };
  // ids of the contracted keys, A's and B's free keys (ascending keys), over
  // the blocks that have a partner
  std::vector<char> ahit(A.nblocks(), 0), bhit(B.nblocks(), 0);
  for (const Match &m : matches) ahit[m.a] = bhit[m.b] = 1;
  struct Ids {
    std::vector<Key128> keys;
    void close() {
      std::sort(keys.begin(), keys.end());
      keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
    }
    int at(Key128 k) const {
      return (int)(std::lower_bound(keys.begin(), keys.end(), k) - keys.begin());
    }
    int n() const { return (int)keys.size(); }
  } kk, ki, kj;
  for (int64_t a = 0; a < A.nblocks(); ++a)
    if (ahit[a]) {
      kk.keys.push_back(key_of(A, a, ca));
      ki.keys.push_back(key_of(A, a, fa));
    }
  for (int64_t b = 0; b < B.nblocks(); ++b)
    if (bhit[b]) kj.keys.push_back(key_of(B, b, fb));
  kk.close();
  ki.close();
  kj.close();
  std::vector<int> a_k(A.nblocks()), a_i(A.nblocks()), b_k(B.nblocks()), b_j(B.nblocks());
  // connected components over the contracted keys
  const int nodes = kk.n() + ki.n() + kj.n();
  std::vector<int> root(nodes);
  for (int i = 0; i < nodes; ++i) root[i] = i;
  auto find = [&](int x) {
    while (root[x] != x) x = root[x] = root[root[x]];
    return x;
  };
  for (int64_t a = 0; a < A.nblocks(); ++a)
    if (ahit[a]) {
      a_k[a] = kk.at(key_of(A, a, ca));
      a_i[a] = ki.at(key_of(A, a, fa));
      root[find(a_k[a])] = find(kk.n() + a_i[a]);
    }
  for (int64_t b = 0; b < B.nblocks(); ++b)
    if (bhit[b]) {
      b_k[b] = kk.at(key_of(B, b, cb));
      b_j[b] = kj.at(key_of(B, b, fb));
      root[find(b_k[b])] = find(kk.n() + ki.n() + b_j[b]);
    }
  // members of each component with their sizes and offsets
  std::vector<int64_t> ksz(kk.n(), 0), isz(ki.n(), 0), jsz(kj.n(), 0);
  auto prod = [](const BTensor &T, int64_t b, const std::vector<int> &axes) {
    int64_t p = 1;
    for (int ax : axes) p *= T.dim_of(b, ax);
    return p;
  };
  for (int64_t a = 0; a < A.nblocks(); ++a)
    if (ahit[a]) {
      ksz[a_k[a]] = prod(A, a, ca);
      isz[a_i[a]] = prod(A, a, fa);
    }
  for (int64_t b = 0; b < B.nblocks(); ++b)
    if (bhit[b]) jsz[b_j[b]] = prod(B, b, fb);
  std::vector<int> comp(nodes, -1);  // component of a root
  int nc = 0;
  auto comp_of = [&](int node) {
    const int r = find(node);
    if (comp[r] < 0) comp[r] = nc++;
    return comp[r];
  };
  struct Comp {
    std::vector<SlLine> rows, cols;
    int64_t M = 0, N = 0, K = 0;
    int ni = 0, nj = 0, nk = 0;
    int64_t na = 0, nb = 0;
    std::vector<int64_t> blocks;
    int id = 0;
  };
  std::vector<Comp> cs;
  auto at = [&](int c) -> Comp & {
    if ((int)cs.size() <= c) cs.resize(c + 1);
    return cs[c];
  };
  std::vector<int64_t> k0(kk.n()), r0(ki.n()), c0(kj.n());
  std::vector<int> iloc(ki.n()), jloc(kj.n());
  for (int k = 0; k < kk.n(); ++k) {
    Comp &c = at(comp_of(k));
    k0[k] = c.K;
    c.K += up8(ksz[k]);
    c.nk++;
  }
  for (int i = 0; i < ki.n(); ++i) {
    Comp &c = at(comp_of(kk.n() + i));
    r0[i] = c.M;
    iloc[i] = c.ni++;
    push_rows(c.rows, iloc[i], isz[i]);
    c.M += isz[i];
  }
  for (int j = 0; j < kj.n(); ++j) {
    Comp &c = at(comp_of(kk.n() + ki.n() + j));
    c0[j] = c.N;
    jloc[j] = c.nj++;
    push_cols(c.cols, jloc[j], jsz[j], es);
    c.N += jsz[j];
  }
  for (Comp &c : cs) {
    if (c.M >= (1 << 30) || c.N >= (1 << 29) || c.K >= (1 << 29)) return nullptr;
    c.blocks.assign((size_t)c.ni * c.nj, -1);
  }
  for (size_t o = 0; o + 1 < mstart.size(); ++o) {
    const Match &m = matches[mstart[o]];
    Comp &c = cs[comp_of(kk.n() + a_i[m.a])];
    c.blocks[(size_t)iloc[a_i[m.a]] * c.nj + jloc[b_j[m.b]]] = coff[o] * es;
  }
  auto sp = std::make_unique<SlicePlan>();
  sp->ctx = A.ctx;
  for (Comp &c : cs)
    c.id = sp->add_group({c.M, c.N * es, c.K * es}, c.rows, c.cols, c.blocks, false);
  int64_t st[kMaxRank];
  for (int side = 0; side < 2; ++side) {
    const BTensor &T = side ? B : A;
    for (int64_t b = 0; b < T.nblocks(); ++b) {
      if (!(side ? bhit : ahit)[b]) continue;
      const int k = side ? b_k[b] : a_k[b];
      Comp &c = cs[comp_of(k)];
      (side ? c.nb : c.na)++;
      SlOp o{};
      o.src = side;
      o.src_off = T.offs[b] * es;
      o.rows = (int32_t)(side ? jsz[b_j[b]] : isz[a_i[b]]);
      o.cols = (int32_t)ksz[k];
      o.r0 = (int32_t)(side ? c0[b_j[b]] : r0[a_i[b]]);
      o.k0 = (int32_t)k0[k];
      block_strides(T, b, st);
      if (!op_dims(T, b, st, side ? fb : fa, es, o.re, o.rs, &o.nr) ||
          !op_dims(T, b, st, side ? cb : ca, es, o.ke, o.ks, &o.nk))
        return nullptr;
      add_ops(*sp, c.id, o, cplx, (int32_t)c.K);
    }
  }
  for (const Comp &c : cs)  // sub-matrices without a block
    if (c.na != (int64_t)c.ni * c.nk || c.nb != (int64_t)c.nj * c.nk) sp->holes = true;
  sp->finalize();
  return sp;
}

// The form rule: the sliced plan where its estimate is below the FP64 tiles'.
// Both are sums over padded work, so ragged sectors, short K and narrow blocks
// (the MPO tensors' few channels) stay on the FMAs.
template <typename Build>
std::unique_ptr<SlicePlan> slice_worth(GemmPlan &g, bool cplx, bool upper, Build build) {
  const int form = g.ctx ? g.ctx->gemm_form : 0;
  if (form == 0 || g.probs.empty()) return nullptr;
  double t64 = 0.0;
  if (form < 0) {
    if (mean_k(g) < kSliceMinK) return nullptr;
    t64 = fp64_seconds(g, cplx, upper);
    if (t64 < kSliceMin) return nullptr;
  }
  auto sp = build();
  if (sp && form < 0 && sp->seconds() >= t64) sp.reset();
  if (sp) {  // the FP64 tiles of operands outside its range: one launch
    const int cfg = one_cfg(g);
    for (size_t p = 0; p < g.probs.size(); ++p)
      for (int32_t m = 0; m < g.probs[p].M; m += kCfgBM[cfg])
        for (int32_t n = 0; n < g.probs[p].N; n += kCfgBN[cfg])
          if (!upper || reaches_diagonal(cfg, m, n))
            g.tiles[cfg].push_back({(int32_t)p, m, n, 0});
  }
  return sp;
}

}  // namespace

static std::unique_ptr<ContractPlan> plan_impl(const BTensor &A, const BTensor &B,
                                               const std::vector<int> &ca,
                                               const std::vector<int> &cb,
                                               const std::vector<int> &fa,
                                               const std::vector<int> &fb, const BTensor *dst,
                                               std::vector<int64_t> *missing, bool upload,
                                               const std::vector<int> &seg_axes = {}) {
  UDMRG_REQUIRE(ca.size() == cb.size(), "contract: axis lists differ in length");
  UDMRG_REQUIRE(A.dtype == B.dtype, "contract: operands must have the same element type");
  UDMRG_REQUIRE(fa.size() + ca.size() == (size_t)A.rank(), "contract: bad A axes");
  UDMRG_REQUIRE(fb.size() + cb.size() == (size_t)B.rank(), "contract: bad B axes");
  for (size_t i = 0; i < ca.size(); ++i) {
    const Index &ia = A.idx[ca[i]], &ib = B.idx[cb[i]];
    UDMRG_REQUIRE(ia.same_space(ib) && ia.dir == -ib.dir,
                  "contract: contracted indexes do not match (sectors or directions)");
  }
  auto plan = std::make_unique<ContractPlan>();
  plan->gemm.ctx = A.ctx;
  auto out = std::make_unique<BTensor>();
  out->ctx = A.ctx;
  out->dtype = A.dtype;
  out->nq = A.nq;
  for (int i : fa) out->idx.push_back(A.idx[i]);
  for (int i : fb) out->idx.push_back(B.idx[i]);
  const int ro = out->rank();
  UDMRG_REQUIRE(ro > 0, "contract: full contractions to a scalar are not supported here");

  UDMRG_REQUIRE(A.rank() <= kMaxRank && B.rank() <= kMaxRank && ro <= kMaxRank,
                "contract: tensors of rank above 8 are not supported");
  for (const BTensor *T : {&A, &B})
    for (const Index &ix : T->idx)
      UDMRG_REQUIRE(ix.nsec() < 65536, "contract: more than 65535 sectors on one index");
  // B blocks sorted by their contracted sector ids
  std::vector<std::pair<uint64_t, int64_t>> bk(B.nblocks());
  for (int64_t b = 0; b < B.nblocks(); ++b) {
    uint64_t k = 0;
    for (int ax : cb) k = (k << 16) | (uint64_t)B.key(b)[ax];
    bk[b] = {k, b};
  }
  std::sort(bk.begin(), bk.end());
  // matching pairs with their output keys, sorted by (output key, a, b)
  std::vector<Match> matches;
  for (int64_t a = 0; a < A.nblocks(); ++a) {
    uint64_t k = 0;
    for (int ax : ca) k = (k << 16) | (uint64_t)A.key(a)[ax];
    auto it = std::lower_bound(bk.begin(), bk.end(), std::make_pair(k, (int64_t)-1));
    Key128 ka = 0;
    for (int ax : fa) ka = (ka << 16) | (Key128)A.key(a)[ax];
    for (; it != bk.end() && it->first == k; ++it) {
      Key128 ok = ka;
      for (int ax : fb) ok = (ok << 16) | (Key128)B.key(it->second)[ax];
      matches.push_back({ok, a, it->second});
    }
  }
  auto before = [](const Match &x, const Match &y) {
    if (x.okey != y.okey) return x.okey < y.okey;
    if (x.a != y.a) return x.a < y.a;
    return x.b < y.b;
  };
  if (seg_axes.empty())
    std::sort(matches.begin(), matches.end(), before);
  else
    std::sort(matches.begin(), matches.end(), [&](const Match &x, const Match &y) {
      if (x.okey == y.okey)
        for (int ax : seg_axes)
          if (A.key(x.a)[ax] != A.key(y.a)[ax]) return A.key(x.a)[ax] < A.key(y.a)[ax];
      return before(x, y);
    });
  // output blocks = distinct keys; [mstart[o], mstart[o + 1]) are their matches
  std::vector<int32_t> flat;
  std::vector<size_t> mstart;
  for (size_t i = 0; i < matches.size(); ++i) {
    if (i > 0 && matches[i].okey == matches[i - 1].okey) continue;
    mstart.push_back(i);
    flat.resize(flat.size() + ro);
    Key128 ok = matches[i].okey;
    for (int j = ro - 1; j >= 0; --j) {
      flat[flat.size() - ro + j] = (int32_t)(uint32_t)(ok & 0xFFFF);
      ok >>= 16;
    }
  }
  mstart.push_back(matches.size());
  const size_t nout = mstart.size() - 1;
  out->set_blocks(flat);  // sorted and unique by construction

  const BTensor *C = out.get();
  if (dst) {
    UDMRG_REQUIRE(dst->rank() == ro, "contract-into: rank mismatch");
    for (int i = 0; i < ro; ++i)
      UDMRG_REQUIRE(dst->idx[i] == out->idx[i], "contract-into: index mismatch");
    C = dst;
  }
  // destination block of every output block
  std::vector<int64_t> dest(nout);
  {
    std::vector<int32_t> okey(ro);
    std::vector<char> hit(dst ? dst->nblocks() : 0, 0);
    for (size_t o = 0; o < nout; ++o) {
      if (!dst) {
        dest[o] = (int64_t)o;
        continue;
      }
      std::copy(flat.begin() + o * ro, flat.begin() + (o + 1) * ro, okey.begin());
      const int64_t id = dst->find(okey);
      UDMRG_REQUIRE(id >= 0, "contract-into: produced block absent from destination");
      dest[o] = id;
      hit[id] = 1;
    }
    if (dst && missing) {
      missing->clear();
      for (int64_t i = 0; i < dst->nblocks(); ++i)
        if (!hit[i]) missing->push_back(i);
    }
  }

  GemmPlan &g = plan->gemm;
  int64_t sa[kMaxRank], sb[kMaxRank];
  const double cplx = A.dtype == kC128 ? 4.0 : 1.0;
  const int nmi = (int)fa.size(), nni = (int)fb.size();
  // merged groups of free axes: (extent, index of the last original axis),
  // extent-1 groups dropped
  auto groups = [](const int64_t *ext, int n, const char *mg, int64_t *gext, int *glast) {
    int ng = 0;
    int64_t ce = 1;
    int cl = -1;
    for (int i = 0; i < n; ++i) {
      if (i > 0 && mg[i - 1]) {
        ce *= ext[i];
        cl = i;
      } else {
        if (cl >= 0 && ce != 1) {
          gext[ng] = ce;
          glast[ng++] = cl;
        }
        ce = ext[i];
        cl = i;
      }
    }
    if (cl >= 0 && ce != 1) {
      gext[ng] = ce;
      glast[ng++] = cl;
    }
    return ng;
  };
  for (size_t o = 0; o < nout; ++o) {
    const int32_t *okey = flat.data() + o * ro;
    const size_t m0 = mstart[o], m1 = mstart[o + 1];
    GProb p{};
    p.c_off = C->offs[dest[o]];
    // M / N sub-dims (extents are the output block's sector dims)
    int64_t mext[kMaxRank], next[kMaxRank];
    for (int i = 0; i < nmi; ++i) mext[i] = A.idx[fa[i]].dims[okey[i]];
    for (int i = 0; i < nni; ++i) next[i] = B.idx[fb[i]].dims[okey[nmi + i]];
    // merge decisions valid for all segments
    char mmerge[kMaxRank], nmerge[kMaxRank];
    for (int i = 0; i < kMaxRank; ++i) mmerge[i] = nmerge[i] = 1;
    for (size_t q = m0; q < m1; ++q) {
      block_strides(A, matches[q].a, sa);
      block_strides(B, matches[q].b, sb);
      for (int i = 0; i + 1 < nmi; ++i)
        if (sa[fa[i]] != mext[i + 1] * sa[fa[i + 1]]) mmerge[i] = 0;
      for (int i = 0; i + 1 < nni; ++i)
        if (sb[fb[i]] != next[i + 1] * sb[fb[i + 1]]) nmerge[i] = 0;
    }
    int64_t mgx[kMaxRank], ngx[kMaxRank];
    int mgl[kMaxRank], ngl[kMaxRank];
    const int nmg = groups(mext, nmi, mmerge, mgx, mgl);
    const int nng = groups(next, nni, nmerge, ngx, ngl);
    UDMRG_REQUIRE(nmg <= kMaxSub && nng <= kMaxSub, "contract: too many non-mergeable free axes");
    int64_t M = 1, N = 1;
    for (int i = 0; i < nmi; ++i) M *= mext[i];
    for (int i = 0; i < nni; ++i) N *= next[i];
    UDMRG_REQUIRE(M < (1ll << 31) && N < (1ll << 31), "contract: block too large");
    p.M = (int32_t)M;
    p.N = (int32_t)N;
    p.nm = nmg;
    p.nn = nng;
    for (int j = 0; j < nmg; ++j) p.m_ext[j] = (int32_t)mgx[j];
    for (int j = 0; j < nng; ++j) p.n_ext[j] = (int32_t)ngx[j];
    p.seg0 = (int32_t)g.segs.size();
    p.nseg = (int32_t)(m1 - m0);
    double kflops = 0;
    for (size_t q = m0; q < m1; ++q) {
      const int64_t pa = matches[q].a, pb = matches[q].b;
      block_strides(A, pa, sa);
      block_strides(B, pb, sb);
      GSeg sg{};
      sg.a_off = A.offs[pa];
      sg.b_off = B.offs[pb];
      for (int j = 0; j < nmg; ++j) sg.a_ms[j] = sa[fa[mgl[j]]];
      for (int j = 0; j < nng; ++j) sg.b_ns[j] = sb[fb[ngl[j]]];
      // K sub-dims merged where both operands allow it; unit dims dropped
      SubDim kd[kMaxRank];
      int nk = 0;
      for (size_t i = 0; i < ca.size(); ++i) {
        SubDim d{A.dim_of(pa, ca[i]), sa[ca[i]], sb[cb[i]]};
        if (nk > 0 && kd[nk - 1].sa == d.ext * d.sa && kd[nk - 1].sb == d.ext * d.sb) {
          kd[nk - 1].ext *= d.ext;
          kd[nk - 1].sa = d.sa;
          kd[nk - 1].sb = d.sb;
        } else if (d.ext != 1) {
          kd[nk++] = d;
        }
      }
      int nk2 = 0;
      for (int i = 0; i < nk; ++i)
        if (kd[i].ext != 1) kd[nk2++] = kd[i];
      UDMRG_REQUIRE(nk2 <= kMaxSub, "contract: too many contracted sub-dims");
      int64_t K = 1;
      for (int i = 0; i < nk2; ++i) K *= kd[i].ext;
      sg.nk = nk2;
      sg.K = (int32_t)K;
      for (int j = 0; j < nk2; ++j) {
        sg.k_ext[j] = (int32_t)kd[j].ext;
        sg.a_ks[j] = kd[j].sa;
        sg.b_ks[j] = kd[j].sb;
      }
      kflops += (double)K;
      g.segs.push_back(sg);
    }
    g.flops += 2.0 * cplx * (double)M * (double)N * kflops;
    g.probs.push_back(p);
  }
  if (!ca.empty()) {
    std::vector<int64_t> coff(nout);
    for (size_t o = 0; o < nout; ++o) coff[o] = C->offs[dest[o]];
    g.sl = slice_worth(g, A.dtype == kC128, false, [&] {
      return slice_contract(A, B, ca, cb, fa, fb, matches, mstart, coff);
    });
  }
  if (!g.sl) tile_all(g);
  if (upload) g.upload();
  plan->out = std::move(out);
  return plan;
}

void gemm_add_simple(GemmPlan &g, int64_t c_off, int64_t M, int64_t N, int64_t K, int64_t a_off,
                     int64_t a_ms, int64_t a_ks, int64_t b_off, int64_t b_ks, int64_t b_ns,
                     bool cplx) {
  if (M == 0 || N == 0) return;
  UDMRG_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "gemm: too large");
  GProb p{};
  p.c_off = c_off;
  p.M = (int32_t)M;
  p.N = (int32_t)N;
  p.nm = 1;
  p.nn = 1;
  p.m_ext[0] = (int32_t)M;
  p.n_ext[0] = (int32_t)N;
  p.seg0 = (int32_t)g.segs.size();
  p.nseg = 1;
  GSeg s{};
  s.a_off = a_off;
  s.b_off = b_off;
  s.a_ms[0] = a_ms;
  s.b_ns[0] = b_ns;
  s.nk = K > 0 ? 1 : 0;
  s.K = (int32_t)K;
  s.k_ext[0] = (int32_t)K;
  s.a_ks[0] = a_ks;
  s.b_ks[0] = b_ks;
  g.segs.push_back(s);
  g.flops += 2.0 * (cplx ? 4.0 : 1.0) * (double)M * (double)N * (double)K;
  g.probs.push_back(p);
}

// Every problem's tiles under the plan's policy.
static void tile_all(GemmPlan &g) {
  for (auto &t : g.tiles) t.clear();
  for (size_t p = 0; p < g.probs.size(); ++p)
    add_tiles(g, (int32_t)p, g.probs[p].M, g.probs[p].N, g.policy);
  // largest K first for load balance
  std::vector<int64_t> ktot(g.probs.size(), 0);
  for (size_t i = 0; i < g.probs.size(); ++i)
    for (int s = 0; s < g.probs[i].nseg; ++s) ktot[i] += g.segs[g.probs[i].seg0 + s].K;
  for (int c = 0; c < kNumCfg; ++c)
    std::stable_sort(g.tiles[c].begin(), g.tiles[c].end(), [&](const GTile &x, const GTile &y) {
      return ktot[x.prob] > ktot[y.prob];
    });
}

void gemm_finalize(GemmPlan &g, bool cplx, bool upper, bool adds) {
  if (!adds) g.sl = slice_worth(g, cplx, upper, [&] { return slice_simple(g, cplx, upper); });
  if (!g.sl) {
    tile_all(g);
    if (upper)
      for (int c = 0; c < kNumCfg; ++c) {
        auto &t = g.tiles[c];
        t.erase(std::remove_if(
                    t.begin(), t.end(),
                    [&](const GTile &x) { return !reaches_diagonal(c, x.m0, x.n0); }),
                t.end());
      }
  }
  g.upload();
}

void gemm_upload(GemmPlan &g) { g.upload(); }

void gemm_retile(GemmPlan &g, int policy) {
  if (policy == g.policy) return;
  g.policy = policy;
  tile_all(g);
  g.upload();
}

TensorPtr contract_struct(const BTensor &A, const BTensor &B, const std::vector<int> &ca,
                          const std::vector<int> &cb, const std::vector<int> &fa,
                          const std::vector<int> &fb) {
  UDMRG_REQUIRE(ca.size() == cb.size(), "contract: axis lists differ in length");
  UDMRG_REQUIRE(fa.size() + ca.size() == (size_t)A.rank(), "contract: bad A axes");
  UDMRG_REQUIRE(fb.size() + cb.size() == (size_t)B.rank(), "contract: bad B axes");
  auto out = std::make_unique<BTensor>();
  out->ctx = A.ctx;
  out->dtype = A.dtype;
  out->nq = A.nq;
  for (int i : fa) out->idx.push_back(A.idx[i]);
  for (int i : fb) out->idx.push_back(B.idx[i]);
  const int ro = out->rank();
  UDMRG_REQUIRE(ro > 0 && ro <= kMaxRank, "contract: output rank");
  for (const BTensor *T : {&A, &B})
    for (const Index &ix : T->idx)
      UDMRG_REQUIRE(ix.nsec() < 65536, "contract: more than 65535 sectors on one index");
  // B's distinct (contracted key, free key) pairs, grouped by contracted key
  std::vector<std::pair<uint64_t, Key128>> bk;
  bk.reserve(B.nblocks());
  for (int64_t b = 0; b < B.nblocks(); ++b) {
    uint64_t k = 0;
    for (int ax : cb) k = (k << 16) | (uint64_t)B.key(b)[ax];
    Key128 f = 0;
    for (int ax : fb) f = (f << 16) | (Key128)B.key(b)[ax];
    bk.push_back({k, f});
  }
  std::sort(bk.begin(), bk.end());
  bk.erase(std::unique(bk.begin(), bk.end()), bk.end());
  std::vector<Key128> keys;
  for (int64_t a = 0; a < A.nblocks(); ++a) {
    uint64_t k = 0;
    for (int ax : ca) k = (k << 16) | (uint64_t)A.key(a)[ax];
    Key128 ka = 0;
    for (int ax : fa) ka = (ka << 16) | (Key128)A.key(a)[ax];
    if (!fb.empty()) ka = fa.empty() ? 0 : ka << (16 * fb.size());
    auto it = std::lower_bound(bk.begin(), bk.end(), std::make_pair(k, (Key128)0));
    for (; it != bk.end() && it->first == k; ++it) keys.push_back(ka | it->second);
  }
  std::sort(keys.begin(), keys.end());
  keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
  std::vector<int32_t> flat(keys.size() * ro);
  for (size_t o = 0; o < keys.size(); ++o) {
    Key128 ok = keys[o];
    for (int j = ro - 1; j >= 0; --j) {
      flat[o * ro + j] = (int32_t)(uint32_t)(ok & 0xFFFF);
      ok >>= 16;
    }
  }
  out->set_blocks(flat);
  return out;
}

std::unique_ptr<ContractPlan> plan_contract(const BTensor &A, const BTensor &B,
                                            const std::vector<int> &ca, const std::vector<int> &cb,
                                            const std::vector<int> &fa,
                                            const std::vector<int> &fb, bool upload) {
  return plan_impl(A, B, ca, cb, fa, fb, nullptr, nullptr, upload);
}

std::unique_ptr<ContractPlan> plan_contract_into(const BTensor &A, const BTensor &B,
                                                 const std::vector<int> &ca,
                                                 const std::vector<int> &cb,
                                                 const std::vector<int> &fa,
                                                 const std::vector<int> &fb, const BTensor &dst,
                                                 std::vector<int64_t> *missing, bool upload,
                                                 const std::vector<int> &seg_axes) {
  return plan_impl(A, B, ca, cb, fa, fb, &dst, missing, upload, seg_axes);
}

std::unique_ptr<ContractPlan> plan_contract_axes(const BTensor &A, const BTensor &B,
                                                 const std::vector<int> &ca,
                                                 const std::vector<int> &cb, bool upload) {
  std::vector<int> fa, fb;
  for (int i = 0; i < A.rank(); ++i)
    if (std::find(ca.begin(), ca.end(), i) == ca.end()) fa.push_back(i);
  for (int i = 0; i < B.rank(); ++i)
    if (std::find(cb.begin(), cb.end(), i) == cb.end()) fb.push_back(i);
  return plan_contract(A, B, ca, cb, fa, fb, upload);
}

std::unique_ptr<ContractPlan> plan_contract_cyclic(const BTensor &A, const BTensor &B, int a_start,
                                                   int b_start, int n, bool upload) {
  std::vector<int> ca, cb, fa, fb;
  cyclic_axes(A.rank(), B.rank(), a_start, b_start, n, ca, cb, fa, fb);
  return plan_contract(A, B, ca, cb, fa, fb, upload);
}

TensorPtr run_contract(Ctx &ctx, const ContractPlan &plan, const BTensor &A, const BTensor &B,
                       bool dw) {
  auto out = plan.out->clone_struct();
  out->alloc_data();
  (dw ? run_gemm_dw : run_gemm)(ctx, plan.gemm, A.dtype, A.data, B.data, out->data, 1.0, 0.0);
  return out;
}

}  // namespace udmrg
