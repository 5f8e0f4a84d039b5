#include "mpo_step.hpp"

#include <algorithm>

namespace udmrg {

std::vector<double> mpo_data(Ctx &ctx, const BTensor &t, bool *real) {
  const int es = elem_doubles(t.dtype);
  std::vector<double> h(t.size() * es);
  if (t.size())
    UDMRG_CHECK_CUDA(cudaMemcpyAsync(h.data(), t.data, h.size() * sizeof(double),
                                     cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  *real = true;
  if (es == 1) return h;
  std::vector<double> r(t.size());
  for (int64_t i = 0; i < t.size(); ++i) {
    if (h[2 * i + 1] != 0.0) *real = false;
    r[i] = h[2 * i];
  }
  return r;
}

FusedMpo::FusedMpo(Ctx &ctx, const BTensor &w1, const BTensor &w2) : W1(w1), W2(w2) {
  bool r1 = true, r2 = true;
  w1h = mpo_data(ctx, W1, &r1);
  w2h = mpo_data(ctx, W2, &r2);
  real = r1 && r2;
  for (int64_t b = 0; b < W1.nblocks(); ++b) w1_by_s1o[W1.key(b)[2]].push_back(b);
  for (int64_t b = 0; b < W2.nblocks(); ++b)
    w2_by[{W2.key(b)[0], W2.key(b)[2], W2.key(b)[3]}].push_back(b);
}

const std::vector<FusedMpo::Entry> &FusedMpo::get(int32_t S1p, int32_t S2p, int32_t W2s) {
  const std::array<int32_t, 3> ck = {S1p, S2p, W2s};
  auto cit = cache.find(ck);
  if (cit != cache.end()) return cit->second;
  const int64_t ds1p = W1.idx[2].dims[S1p], ds2p = W2.idx[2].dims[S2p];
  const int64_t dw2 = W2.idx[3].dims[W2s];
  const int64_t nout = ds1p * ds2p * dw2;
  std::map<std::array<int32_t, 3>, std::vector<double>> acc;  // (W, S1, S2) -> coef
  auto it1 = w1_by_s1o.find(S1p);
  if (it1 != w1_by_s1o.end()) {
    for (int64_t b1 : it1->second) {
      const int32_t Ws = W1.key(b1)[0], S1 = W1.key(b1)[1], Wr = W1.key(b1)[3];
      auto it2 = w2_by.find({Wr, S2p, W2s});
      if (it2 == w2_by.end()) continue;
      for (int64_t b2 : it2->second) {
        const int32_t S2 = W2.key(b2)[1];
        const int64_t dw = W1.idx[0].dims[Ws], ds1 = W1.idx[1].dims[S1];
        const int64_t dwr = W1.idx[3].dims[Wr], ds2 = W2.idx[1].dims[S2];
        const int64_t nin = dw * ds1 * ds2;
        auto &c = acc[{Ws, S1, S2}];
        if (c.empty()) c.assign(nin * nout, 0.0);
        // W1(w, s1, s1', wr) W2(wr, s2, s2', w2), blocks row-major
        const double *w1 = w1h.data() + W1.offs[b1];
        const double *w2 = w2h.data() + W2.offs[b2];
        for (int64_t w = 0; w < dw; ++w)
          for (int64_t s1 = 0; s1 < ds1; ++s1)
            for (int64_t s2 = 0; s2 < ds2; ++s2)
              for (int64_t s1o = 0; s1o < ds1p; ++s1o)
                for (int64_t s2o = 0; s2o < ds2p; ++s2o)
                  for (int64_t w2i = 0; w2i < dw2; ++w2i) {
                    double v = 0;
                    for (int64_t wr = 0; wr < dwr; ++wr)
                      v += w1[((w * ds1 + s1) * ds1p + s1o) * dwr + wr] *
                           w2[((wr * ds2 + s2) * ds2p + s2o) * dw2 + w2i];
                    const int64_t ic = (w * ds1 + s1) * ds2 + s2;
                    const int64_t oc = (s1o * ds2p + s2o) * dw2 + w2i;
                    c[ic * nout + oc] += v;
                  }
      }
    }
  }
  std::vector<Entry> entries;
  for (auto &kv : acc) {
    bool nz = false;
    for (double v : kv.second) nz |= (v != 0.0);
    if (nz) entries.push_back({kv.first, std::move(kv.second)});
  }
  return cache.emplace(ck, std::move(entries)).first->second;
}

MpoStep64::~MpoStep64() {
  if (!ctx) return;
  ctx->free(d_block);
}

namespace {

// Couplings and writes of one task: a warp walks them in turn, so long runs leave
// the chip with few warps and an uneven end; short ones read inputs that a
// neighbouring run has in L1 again.  The step of Hubbard 4x8, D = 500 / 1000 /
// 2000 in runs of 24: 29 / 66 / 210 us, 48: 31 / 70 / 212, 96: 44 / 82 / 226,
// whole pairs: 50 / 89 / 236.
constexpr int32_t kMpoRun = 24;

// One (a, b) sector pair under construction: its channels and couplings.
struct PairMap {
  struct In {
    int64_t base, astride;
  };
  struct Nz {
    int32_t o, i;
    double v;
  };
  std::vector<In> ins;
  std::vector<MpoOut64> outs;
  std::vector<Nz> nz, sorted;
  std::vector<int32_t> start, at;
  std::vector<std::pair<int64_t, int32_t>> in_first;  // input block -> its first channel
  void clear() {
    ins.clear();
    outs.clear();
    nz.clear();
    in_first.clear();
  }
  // first channel of input block b, appended with `n` channels of `db` columns
  // from offset off if it is new
  int32_t input(int64_t b, int64_t off, int64_t n, int64_t db) {
    for (const auto &f : in_first)
      if (f.first == b) return f.second;
    const int32_t c0 = (int32_t)ins.size();
    in_first.push_back({b, c0});
    for (int64_t c = 0; c < n; ++c) ins.push_back({off + c * db, n * db});
    return c0;
  }
};

// Appends the pair in CSR form (couplings of one (o, i) summed, by ascending i).
void push_pair(MpoStep64 &p, PairMap &m, int64_t da, int64_t db, int es) {
  MpoPair64 pr{};
  pr.out0 = (int32_t)p.outs.size();
  pr.nout = (int32_t)m.outs.size();
  pr.row0 = (int32_t)(p.rowptr.size() - 1);
  pr.da = (int32_t)da;
  pr.db = (int32_t)(db * es);
  for (MpoOut64 o : m.outs) p.outs.push_back({o.base * es, o.astride * es, -1, 0, 0});
  // couplings by output channel (counting sort, stable), then by input
  m.start.assign(pr.nout + 1, 0);
  for (const PairMap::Nz &z : m.nz) m.start[z.o + 1]++;
  for (int o = 0; o < pr.nout; ++o) m.start[o + 1] += m.start[o];
  m.sorted.resize(m.nz.size());
  m.at.assign(m.start.begin(), m.start.end() - 1);
  for (const PairMap::Nz &z : m.nz) m.sorted[m.at[z.o]++] = z;
  const size_t n0 = p.nz.size();
  for (int o = 0; o < pr.nout; ++o) {
    auto b = m.sorted.begin() + m.start[o], e = m.sorted.begin() + m.start[o + 1];
    auto less = [](const PairMap::Nz &x, const PairMap::Nz &y) { return x.i < y.i; };
    if (!std::is_sorted(b, e, less)) std::stable_sort(b, e, less);
    for (auto q = b; q != e;) {
      double v = 0.0;
      const int i = q->i;
      for (; q != e && q->i == i; ++q) v += q->v;
      if (v == 0.0) continue;
      UDMRG_REQUIRE(m.ins[i].astride * es < (1ll << 31), "MPO step: block too large");
      p.nz.push_back({m.ins[i].base * es, v, (int32_t)(m.ins[i].astride * es), 0});
    }
    p.rowptr.push_back((int32_t)p.nz.size());
  }
  p.flops += 2.0 * (double)(p.nz.size() - n0) * pr.da * pr.db;
  // (a task counts to 64 past its first entry in 32 bits)
  UDMRG_REQUIRE((int64_t)pr.da * db * es < (1ll << 31) - 64, "MPO step: block too large");
  // runs of output channels of at most kMpoRun couplings and writes (one channel at least)
  for (int32_t o0 = 0, o1; o0 < pr.nout; o0 = o1) {
    const int32_t *row = p.rowptr.data() + pr.row0;
    for (o1 = o0 + 1; o1 < pr.nout && row[o1 + 1] - row[o0] + (o1 + 1 - o0) <= kMpoRun; ++o1) {
    }
    for (int64_t u = 0; u < (int64_t)pr.da * pr.db; u += 64)
      p.tasks.push_back({(int32_t)p.pairs.size(), (int32_t)u, o0, o1});
  }
  p.pairs.push_back(pr);
}

// Blocks with the sectors of their first and last axes, grouped by them
// (ascending; block order within a pair).
struct Ends {
  int32_t a, b;
  int64_t blk;
};
std::vector<Ends> by_ends(const BTensor &t) {
  std::vector<Ends> v(t.nblocks());
  for (int64_t b = 0; b < t.nblocks(); ++b) v[b] = {t.key(b)[0], t.key(b)[t.rank() - 1], b};
  std::sort(v.begin(), v.end(), [](const Ends &x, const Ends &y) {
    return x.a != y.a ? x.a < y.a : x.b != y.b ? x.b < y.b : x.blk < y.blk;
  });
  return v;
}

// Block of t with the given sector ids (blocks are sorted), or -1.
int64_t find_block(const BTensor &t, const int32_t *k) {
  const int r = t.rank();
  int64_t lo = 0, hi = t.nblocks();
  while (lo < hi) {
    const int64_t mid = (lo + hi) / 2;
    if (std::lexicographical_compare(t.key(mid), t.key(mid) + r, k, k + r))
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < t.nblocks() && std::equal(k, k + r, t.key(lo)) ? lo : -1;
}

}  // namespace

std::unique_ptr<MpoStep64> build_mpo_step64(FusedMpo &fm, const BTensor &T1, const BTensor &T3) {
  UDMRG_REQUIRE(T1.rank() == 5 && T3.rank() == 5, "MPO step: rank-5 intermediates expected");
  auto p = std::make_unique<MpoStep64>();
  const int es = elem_doubles(T1.dtype);
  p->rowptr.push_back(0);
  const std::vector<Ends> ends = by_ends(T3);
  PairMap m;
  for (size_t g = 0; g < ends.size();) {
    const int32_t Ap = ends[g].a, Bs = ends[g].b;
    const int64_t da = T3.idx[0].dims[Ap], db = T3.idx[4].dims[Bs];
    m.clear();
    for (; g < ends.size() && ends[g].a == Ap && ends[g].b == Bs; ++g) {
      const int64_t ob = ends[g].blk;
      const int32_t *k = T3.key(ob);
      const int64_t nout =
          T3.idx[1].dims[k[1]] * T3.idx[2].dims[k[2]] * T3.idx[3].dims[k[3]];
      UDMRG_REQUIRE(nout * db * es < (1ll << 31), "MPO step: block too large");
      const int32_t ofirst = (int32_t)m.outs.size();
      for (int64_t c = 0; c < nout; ++c)
        m.outs.push_back({T3.offs[ob] + c * db, (int32_t)(nout * db), -1, 0, 0});
      for (const FusedMpo::Entry &e : fm.get(k[1], k[2], k[3])) {
        const int32_t tk[5] = {Ap, e.src[0], e.src[1], e.src[2], Bs};
        const int64_t tb = find_block(T1, tk);
        if (tb < 0) continue;
        const int64_t nin = T1.idx[1].dims[e.src[0]] * T1.idx[2].dims[e.src[1]] *
                            T1.idx[3].dims[e.src[2]];
        const int32_t ifirst = m.input(tb, T1.offs[tb], nin, db);
        for (int64_t ic = 0; ic < nin; ++ic)
          for (int64_t oc = 0; oc < nout; ++oc) {
            const double v = e.coef[ic * nout + oc];
            if (v != 0.0) m.nz.push_back({(int32_t)(ofirst + oc), (int32_t)(ifirst + ic), v});
          }
      }
    }
    push_pair(*p, m, da, db, es);
  }
  return p;
}

std::unique_ptr<MpoStep64> build_mpo_map(const BTensor &T, const BTensor &W,
                                         const std::vector<double> &wh, int x1, int x2,
                                         const BTensor &out) {
  UDMRG_REQUIRE(T.rank() == 4 && out.rank() == 4 && W.rank() == 4, "MPO map: rank-4 tensors");
  auto p = std::make_unique<MpoStep64>();
  const int es = elem_doubles(T.dtype);
  int y[2], ny = 0;
  for (int ax = 0; ax < 4; ++ax)
    if (ax != x1 && ax != x2) y[ny++] = ax;
  // W's blocks by their output sectors, with the nonzeros of each
  struct WNz {
    int32_t i, o;
    double v;
  };
  struct WBlk {
    int32_t y1, y2, k1, k2;
    int64_t nin;
    std::vector<WNz> nz;
  };
  std::vector<WBlk> wb;
  for (int64_t b = 0; b < W.nblocks(); ++b) {
    const int32_t *kw = W.key(b);
    const int64_t e1 = W.idx[x1].dims[kw[x1]], e2 = W.idx[x2].dims[kw[x2]];
    const int64_t d1 = W.idx[y[0]].dims[kw[y[0]]], d2 = W.idx[y[1]].dims[kw[y[1]]];
    int64_t st[4];
    st[3] = 1;
    for (int ax = 2; ax >= 0; --ax) st[ax] = st[ax + 1] * W.idx[ax + 1].dims[kw[ax + 1]];
    WBlk w{kw[y[0]], kw[y[1]], kw[x1], kw[x2], e1 * e2, {}};
    for (int64_t i1 = 0; i1 < e1; ++i1)
      for (int64_t i2 = 0; i2 < e2; ++i2)
        for (int64_t o1 = 0; o1 < d1; ++o1)
          for (int64_t o2 = 0; o2 < d2; ++o2) {
            const double v =
                wh[W.offs[b] + i1 * st[x1] + i2 * st[x2] + o1 * st[y[0]] + o2 * st[y[1]]];
            if (v != 0.0) w.nz.push_back({(int32_t)(i1 * e2 + i2), (int32_t)(o1 * d2 + o2), v});
          }
    wb.push_back(std::move(w));
  }
  std::stable_sort(wb.begin(), wb.end(), [](const WBlk &u, const WBlk &v) {
    return u.y1 != v.y1 ? u.y1 < v.y1 : u.y2 < v.y2;
  });
  p->rowptr.push_back(0);
  const std::vector<Ends> ends = by_ends(out);
  PairMap m;
  for (size_t g = 0; g < ends.size();) {
    const int32_t Ap = ends[g].a, Bs = ends[g].b;
    const int64_t da = out.idx[0].dims[Ap], db = out.idx[3].dims[Bs];
    m.clear();
    for (; g < ends.size() && ends[g].a == Ap && ends[g].b == Bs; ++g) {
      const int64_t ob = ends[g].blk;
      const int32_t *k = out.key(ob);
      const int64_t d1 = out.idx[1].dims[k[1]], d2 = out.idx[2].dims[k[2]];
      UDMRG_REQUIRE(d1 * d2 * db * es < (1ll << 31), "MPO step: block too large");
      const int32_t ofirst = (int32_t)m.outs.size();
      for (int64_t c = 0; c < d1 * d2; ++c)
        m.outs.push_back({out.offs[ob] + c * db, (int32_t)(d1 * d2 * db), -1, 0, 0});
      auto it = std::lower_bound(wb.begin(), wb.end(), std::make_pair(k[1], k[2]),
                                 [](const WBlk &u, const std::pair<int32_t, int32_t> &q) {
                                   return u.y1 != q.first ? u.y1 < q.first : u.y2 < q.second;
                                 });
      for (; it != wb.end() && it->y1 == k[1] && it->y2 == k[2]; ++it) {
        const int32_t tk[4] = {Ap, it->k1, it->k2, Bs};
        const int64_t tb = find_block(T, tk);
        if (tb < 0) continue;
        const int32_t ifirst = m.input(tb, T.offs[tb], it->nin, db);
        for (const WNz &z : it->nz) m.nz.push_back({ofirst + z.o, ifirst + z.i, z.v});
      }
    }
    push_pair(*p, m, da, db, es);
  }
  return p;
}

bool link_scales(MpoStep64 &p, SlicePlan *next) {
  if (!next) return false;
  struct Block {
    int64_t off, end, row;  // source range, doubles per row
    int64_t line;
    int32_t rstep;
  };
  std::vector<Block> blocks;
  for (const SlOp &o : next->ops) {
    if (o.src != 0) continue;
    if (o.nr > 1 || o.nk > 1 || o.rows_fast) return false;
    const int64_t es = o.nk ? o.ks[0] : 1;
    if (es > 2) return false;
    const int64_t off = o.src_off / es * es;  // (of the imaginary parts: their block's)
    const int64_t row = o.nr ? o.rs[0] : o.cols * es;
    if (row != o.cols * es) return false;
    blocks.push_back({off, off + o.rows * row, row, o.sc0 + o.r0, o.rstep});
  }
  std::sort(blocks.begin(), blocks.end(),
            [](const Block &x, const Block &y) { return x.off < y.off; });
  for (const MpoPair64 &pr : p.pairs)
    for (int32_t c = pr.out0; c < pr.out0 + pr.nout; ++c) {
      MpoOut64 &o = p.outs[c];
      auto it = std::upper_bound(blocks.begin(), blocks.end(), o.base,
                                 [](int64_t v, const Block &b) { return v < b.off; });
      if (it == blocks.begin() || o.base >= (it - 1)->end) continue;  // not contracted
      const Block &b = *(it - 1);
      const int64_t in_row = (o.base - b.off) % b.row;
      if (in_row + pr.db > b.row || o.astride % b.row != 0 ||
          o.base + (int64_t)(pr.da - 1) * o.astride >= b.end) {
        for (MpoOut64 &q : p.outs) q.line = -1;
        return false;
      }
      o.line = (int32_t)(b.line + (o.base - b.off) / b.row * b.rstep);
      o.step = (int32_t)(o.astride / b.row * b.rstep);
    }
  next->prescaled = true;
  return true;
}

void upload_mpo_step64(Ctx &ctx, MpoStep64 &m) {
  m.ctx = &ctx;
  UploadBatch up(ctx);
  const size_t o0 = up.add(m.pairs), o1 = up.add(m.outs), o2 = up.add(m.rowptr), o3 = up.add(m.nz),
               o4 = up.add(m.tasks);
  m.d_block = up.commit();
  m.d_pairs = (MpoPair64 *)(m.d_block + o0);
  m.d_outs = (MpoOut64 *)(m.d_block + o1);
  m.d_rowptr = (int32_t *)(m.d_block + o2);
  m.d_nz = (MpoNz64 *)(m.d_block + o3);
  m.d_tasks = (MpoTask64 *)(m.d_block + o4);
}

}  // namespace udmrg
