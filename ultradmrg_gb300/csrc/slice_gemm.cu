// Digit-sliced FP64-accurate grouped GEMM (see slice_gemm.hpp): scale pass,
// digit pack, tcgen05 GEMM.
#include "slice_gemm.hpp"

#include <algorithm>

#include "tc_roles.cuh"

namespace udmrg {

namespace {

constexpr int kPackThreads = 256, kPackWarps = kPackThreads / 32;
constexpr int kPackRows = 8, kPackCols = 128;  // item of the warps with contiguous columns
// Biased exponents of the sliced range.  Two lines from its lower end have sums in
// units of 2^-1018: no result is below the normal range.
constexpr int kLoExp = 1023 - 476, kHiExp = 1023 + 476;
static_assert(2 * (kLoExp - 1022) - 68 >= -1022, "sliced GEMM: sl_round makes no denormals");
static_assert(2 * (kHiExp - 1022) + 30 <= 1023, "sliced GEMM: sums of 2^30 products stay finite");

__device__ __forceinline__ int64_t sl_off(int64_t i, const int32_t *ext, const int64_t *str, int n) {
  int64_t off = 0;
  for (int j = n - 1; j > 0; --j) {
    const int32_t e = ext[j];
    const int32_t q = (int32_t)i / e;
    off += (int64_t)((int32_t)i - q * e) * str[j];
    i = q;
  }
  return n > 0 ? off + i * str[0] : 0;
}

// Offsets of the tile's 32 rows and 64 columns (one division chain each, by
// 96 threads); -1 past the op's edge.
__device__ __forceinline__ void tile_offsets(const SlOp &op, const SlItem &it, int64_t *roff,
                                             int64_t *koff) {
  const int t = threadIdx.x;
  if (t < 32) {
    const int r = it.r0 + t;
    roff[t] = r < op.rows ? op.src_off + sl_off(r, op.re, op.rs, op.nr) : -1;
  } else if (t < 96) {
    const int k = it.k0 + t - 32;
    koff[t - 32] = k < op.cols ? sl_off(k, op.ke, op.ks, op.nk) : -1;
  }
}

// scale[line] = max over the line's elements of tc::abs_high: its exponent bounds
// the line.  HBM bound: 8 B per element, read once.  The first nbk blocks take
// the items with contiguous columns (or every second double: complex parts), a
// warp 8 rows at a time with sixteen loads per lane in flight; the others an
// item of 32 rows x 64 columns per block, lanes along the contiguous direction.
__global__ void __launch_bounds__(kPackThreads)
    slice_scale_kernel(const SlOp *__restrict__ ops, const SlItem *__restrict__ items_k, int nk,
                       int nbk, const SlItem *__restrict__ items_t, int nt,
                       const double *__restrict__ a, const double *__restrict__ b,
                       int *__restrict__ scale) {
  __shared__ int64_t roff[32], koff[64];
  __shared__ int mx[32];
  const int tid = threadIdx.x;
  tc::pdl_launch_dependents();
  if (blockIdx.x < nbk) {
    const int lane = tid & 31;
    for (int w = blockIdx.x * kPackWarps + (tid >> 5); w < nk; w += nbk * kPackWarps) {
      const SlItem it = items_k[w];
      const SlOp &op = ops[it.op];
      const int es = op.nk ? (int)op.ks[0] : 1, nr = min(kPackRows, op.rows - it.r0);
      const int n = min(op.cols - it.k0, it.width);
      const double *src = (op.src ? b : a) + op.src_off + (int64_t)it.k0 * es;
      const long long off = lane < nr ? sl_off(it.r0 + lane, op.re, op.rs, op.nr) : 0;
      int best = 0;  // of row it.r0 + lane
#pragma unroll
      for (int r0 = 0; r0 < kPackRows; r0 += 4) {
        double x[4][kPackCols / 32];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const long long o = __shfl_sync(0xffffffffu, off, r0 + r);
#pragma unroll
          for (int c = 0; c < kPackCols / 32; ++c) {
            const int k = lane + 32 * c;
            x[r][c] = r0 + r < nr && k < n ? __ldg(src + o + (int64_t)k * es) : 0.0;
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          int v = 0;
#pragma unroll
          for (int c = 0; c < kPackCols / 32; ++c) v = max(v, tc::abs_high(x[r][c]));
          v = __reduce_max_sync(0xffffffffu, v);
          if (lane == r0 + r) best = v;
        }
      }
      if (best)
        atomicMax(scale + 2 + op.sc0 + op.r0 + (int64_t)(it.r0 + lane) * op.rstep, best);
    }
    return;
  }
  for (int w = blockIdx.x - nbk; w < nt; w += gridDim.x - nbk) {
    const SlItem it = items_t[w];
    const SlOp &op = ops[it.op];
    const double *src = op.src ? b : a;
    const bool rows_fast = op.rows_fast != 0;
    __syncthreads();
    tile_offsets(op, it, roff, koff);
    if (tid < 32) mx[tid] = 0;
    __syncthreads();
    int best[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = tid + q * kPackThreads;
      const int r = rows_fast ? e & 31 : e >> 6, k = rows_fast ? e >> 5 : e & 63;
      best[q] = roff[r] >= 0 && koff[k] >= 0 ? tc::abs_high(__ldg(src + roff[r] + koff[k])) : 0;
    }
    if (rows_fast) {  // a thread's eight elements share its row
      int v = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) v = max(v, best[q]);
      if (v) atomicMax(&mx[tid & 31], v);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int v = __reduce_max_sync(0xffffffffu, best[q]);
        if ((tid & 31) == 0 && v) atomicMax(&mx[(tid + q * kPackThreads) >> 6], v);
      }
    }
    __syncthreads();
    if (tid < 32 && mx[tid]) {
      atomicMax(scale + 2 + op.sc0 + op.r0 + (int64_t)(it.r0 + tid) * op.rstep, mx[tid]);
    }
  }
}

// x 2^(62 - e) rounded to an integer, e the line's exponent (|x| < 2^e), plus
// 128 in each of its seven lower base-256 digits: byte d of the result is the
// digit's value + 128 (balanced digits, -128 .. 127), its top byte the signed
// leading digit (-64 .. 64).  Integer instructions only.
__device__ __forceinline__ int64_t slice_bits(double x, int be, bool neg) {
  const uint64_t d = (uint64_t)__double_as_longlong(x);
  const int s = be - (int)((d >> 52) & 0x7FF);  // 0 for the line's largest binade
  const uint64_t m = (d & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  int64_t v = 0;
  if (s <= 9)
    v = (int64_t)(m << (9 - s));
  else if (s < 64)
    v = (int64_t)((m + (1ull << (s - 10))) >> (s - 9));
  if (((d >> 63) != 0) != neg) v = -v;
  return v + 0x80808080808080ll;
}

// Eight consecutive columns of one row into their eight 16-byte plane segments: a
// byte of slice_bits becomes a float by the 2^23 + byte pattern (one byte
// permute and one FP32 add per digit), two floats' upper halves a BF16 pair.
__device__ __forceinline__ void store_digits(const double (&x)[8], int be, bool neg, uint8_t *o,
                                             int64_t plane) {
  uint32_t p[kSlDigits][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float f[2][kSlDigits];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int64_t v = slice_bits(x[2 * j + t], be, neg);
      const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
      f[t][0] = __uint_as_float(0x4B000000u + 128u + (uint32_t)((int32_t)hi >> 24));
      f[t][1] = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7652));
      f[t][2] = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7651));
      f[t][3] = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7650));
      f[t][4] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7653));
      f[t][5] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7652));
      f[t][6] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7651));
      f[t][7] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7650));
    }
#pragma unroll
    for (int d = 0; d < kSlDigits; ++d)
      p[d][j] = __byte_perm(__float_as_uint(f[0][d] - 8388736.0f),
                            __float_as_uint(f[1][d] - 8388736.0f), 0x7632);
  }
#pragma unroll
  for (int d = 0; d < kSlDigits; ++d)
    *(uint4 *)(o + d * plane) = make_uint4(p[d][0], p[d][1], p[d][2], p[d][3]);
}

// Image address of row `row`, K step and column follow; be: the row's biased
// exponent (0x7FF for a line of zeros: every digit zero).  A line whose largest
// element is non-finite or outside the sliced range raises the flag.
__device__ __forceinline__ uint8_t *image_row(const SlOp &op, int row, int *scale, uint8_t *img,
                                              int &be) {
  const int sc = scale[2 + op.sc0 + row];
  be = sc == 0 ? 0x7FF : sc >> 20;
  if (sc != 0 && (be < kLoExp || be > kHiExp)) atomicExch(scale, 1);
  const int64_t plane = (int64_t)op.tr * kSlK * 2;
  return img + op.img_off + (int64_t)(row >> (op.tr == kSlU ? 7 : 6)) * op.kc * kSlDigits * plane;
}

// Digits of the operands into their images.  HBM bound: 8 B read and 16 B
// written per element.  Ops start at columns that are multiples of 8; the columns
// from an op's edge to the next one are written as zeros.
//
// The first nbk blocks take the items with contiguous columns (or every second
// double), without shared memory: a warp takes 8 rows x 32 columns at a time, lane =
// (column group, row): eight loads of its row's 64 bytes (consecutive lanes' rows
// share no sectors, but each sector is used whole over the eight), then the
// plane segments of eight rows fill 128 contiguous bytes.  The other blocks'
// items are 32 rows x 64 columns, staged in shared memory along the source's
// contiguous direction; then a thread cuts one row's 8 consecutive columns, and
// the 32 rows of a warp fill 512 contiguous bytes per plane.
__global__ void __launch_bounds__(kPackThreads)
    slice_pack_kernel(const SlOp *__restrict__ ops, const SlItem *__restrict__ items_k, int nk,
                      int nbk, const SlItem *__restrict__ items_t, int nt,
                      const double *__restrict__ a, const double *__restrict__ b,
                      int *__restrict__ scale, uint8_t *__restrict__ img) {
  __shared__ int64_t roff[32], koff[64];
  __shared__ double tile[64][33];
  const int tid = threadIdx.x;
  tc::pdl_launch_dependents();
  tc::pdl_wait();  // the scales
  if (blockIdx.x < nbk) {
    const int lane = tid & 31, r = lane % kPackRows, g = lane / kPackRows;
    for (int w = blockIdx.x * kPackWarps + (tid >> 5); w < nk; w += nbk * kPackWarps) {
      const SlItem it = items_k[w];
      const SlOp &op = ops[it.op];
      const int rs = it.r0 + r;
      if (rs >= op.rows) continue;
      const double *src = (op.src ? b : a) + op.src_off + sl_off(rs, op.re, op.rs, op.nr);
      const int es = op.nk ? (int)op.ks[0] : 1, row = op.r0 + rs * op.rstep;
      int be;
      uint8_t *orow = image_row(op, row, scale, img, be);
      const int64_t plane = (int64_t)op.tr * kSlK * 2;
      const int rin = row & (op.tr - 1), end = min(op.cols, it.k0 + it.width);
      const bool neg = op.neg != 0;
      for (int ks = it.k0 + g * 8; ks < end; ks += 32) {
        const int n = min(8, op.cols - ks), col = op.k0 + ks;
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = j < n ? __ldg(src + (int64_t)(ks + j) * es) : 0.0;
        store_digits(x, be, neg, orow + (int64_t)(col >> 4) * kSlDigits * plane +
                                     canon_off(rin, col & 15, op.tr), plane);
      }
    }
    return;
  }
  for (int w = blockIdx.x - nbk; w < nt; w += gridDim.x - nbk) {
    const SlItem it = items_t[w];
    const SlOp &op = ops[it.op];
    const double *src = op.src ? b : a;
    const bool rows_fast = op.rows_fast != 0;
    __syncthreads();
    tile_offsets(op, it, roff, koff);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = tid + q * kPackThreads;
      const int r = rows_fast ? e & 31 : e >> 6, k = rows_fast ? e >> 5 : e & 63;
      tile[k][r] = roff[r] >= 0 && koff[k] >= 0 ? __ldg(src + roff[r] + koff[k]) : 0.0;
    }
    __syncthreads();
    const int r = tid & 31, g = tid >> 5;
    const int rs = it.r0 + r, ks = it.k0 + g * 8;
    if (rs >= op.rows || ks >= op.cols) continue;
    const int row = op.r0 + rs * op.rstep, col = op.k0 + ks;
    int be;
    uint8_t *orow = image_row(op, row, scale, img, be);
    const int64_t plane = (int64_t)op.tr * kSlK * 2;
    double x[8];  // (zeros past the op's columns)
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = tile[g * 8 + j][r];
    store_digits(x, be, op.neg != 0,
                 orow + (int64_t)(col >> 4) * kSlDigits * plane +
                     canon_off(row & (op.tr - 1), col & 15, op.tr), plane);
  }
}

// ---- the GEMM ----
//
// Warp-specialised persistent kernel over the tile list: warp 0 stages the two
// operands' K steps by bulk copies (four stages of 48 KB), warp 1 issues 36
// tcgen05.mma (M 128, N 64, K 16) per step into eight 64-column accumulators
// (all 512 TMEM columns), warps 2 .. 17 drain them after every kSlChunk steps.
// An epilogue thread owns 16 outputs of one lane; it adds the levels into a
// 96-bit integer per output and frees the accumulators before it rounds and
// stores, so the next chunk's products overlap the rounding.  Every wait is
// bounded.
//
// Bound by the draining: the accumulators take all of TMEM, so the tensor core
// waits while they are read, and the 64-bit integer sums cost more issue slots
// than the 36 products of a step.  Sixteen warps of 16 outputs (three registers
// each: no spills at the 96 registers that 576 threads leave) against eight of
// 32: Hubbard 4x8, D = 1000, effective Hamiltonian 549 -> 402 us together with
// the K parts and the direct pack of contiguous columns.
constexpr int kSlParts = 4;  // epilogue warps per lane quarter
constexpr int kSlCols = kSlV / kSlParts;
constexpr int kSlThreads = 64 + 128 * kSlParts;
constexpr int kSlStages = 4;
constexpr int kSlStageBytes = (int)(kSlUnitU + kSlUnitV);
constexpr int kSlBarOffset = kSlStages * kSlStageBytes + kPadBytes;
constexpr int kSlSmem = kSlBarOffset + 1024;
static_assert(kSlSmem <= 227 * 1024, "sliced GEMM: shared memory budget");
static_assert(kSlLevels * kSlV == 512, "sliced GEMM: the accumulators fill TMEM");

struct SlBars {
  uint64_t full[kSlStages], empty[kSlStages], tfull, tempty, fin;
  uint32_t tmem;
  volatile int abort;
};

__device__ __forceinline__ void sl_fail(SlBars *b, int *flags) {
  atomicExch(flags + 1, 1);
  b->abort = 1;
}

// 32 lanes x 32 bit, 2 consecutive columns per thread
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(taddr)
               : "memory");
}

// A sum of level products in units of 2^-68: hi 2^32 + lo, hi signed.
struct SlSum {
  int64_t hi;
  uint32_t lo;
};
__device__ __forceinline__ void sl_add(SlSum &s, int64_t hi, int64_t lo) {  // + hi 2^32 + lo
  lo += s.lo;
  s.hi += hi + (lo >> 32);
  s.lo = (uint32_t)lo;
}

// s 2^(e - 68) rounded to nearest FP64; |hi| < 2^62, e within twice the sliced
// range (the result is zero or normal)
__device__ __forceinline__ double sl_round(const SlSum &s, int e) {
  const int64_t hi = s.hi;
  uint32_t w0 = s.lo;
  const bool neg = hi < 0;
  uint64_t h = (uint64_t)hi;
  if (neg) {
    h = ~h + (w0 == 0 ? 1 : 0);
    w0 = 0u - w0;
  }
  uint32_t w2 = (uint32_t)(h >> 32), w1 = (uint32_t)h;
  int ex = 1023 + 95 - 68 + e;
  if (w2 == 0) {
    w2 = w1;
    w1 = w0;
    w0 = 0;
    ex -= 32;
    if (w2 == 0) {
      w2 = w1;
      w1 = 0;
      ex -= 32;
    }
  }
  if (w2 == 0) return 0.0;
  const int c = __clz(w2);
  ex -= c;
  const uint32_t m1 = __funnelshift_l(w1, w2, c), m0 = __funnelshift_l(w0, w1, c);
  const uint64_t m = ((uint64_t)m1 << 32) | m0;
  uint64_t r = ((uint64_t)ex << 52) + ((m >> 11) & 0xFFFFFFFFFFFFFull) + ((m >> 10) & 1);
  r |= (uint64_t)neg << 63;
  return __longlong_as_double((long long)r);
}

__global__ void __launch_bounds__(kSlThreads, 1)
    slice_gemm_kernel(const SlTile *__restrict__ tiles, int ntiles,
                      const SlGroup *__restrict__ groups, const SlLine *__restrict__ lines,
                      const int64_t *__restrict__ cblk, const int *scale,
                      const uint8_t *__restrict__ img, double *__restrict__ C, int *flags,
                      longlong2 *__restrict__ scratch, int *__restrict__ arrived) {
  extern __shared__ __align__(1024) uint8_t smem[];
  SlBars *b = (SlBars *)(smem + kSlBarOffset);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kSlStages; ++s) {
      tc::mbar_init(&b->full[s], 1);
      tc::mbar_init(&b->empty[s], 1);
    }
    tc::mbar_init(&b->tfull, 1);
    tc::mbar_init(&b->tempty, 4 * kSlParts);  // one arrival per epilogue warp
    tc::mbar_init(&b->fin, 1);
    b->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    tc::tmem_alloc(&b->tmem, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = b->tmem;
  tc::pdl_wait();  // the images and scales
  if (scale[0]) {  // the sliced form does not apply (uniform over the grid)
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
    return;
  }

  if (warp == 0) {
    if (lane == 0) {
      uint32_t G = 0;
      for (int i = 0, t; (t = tc::snake_tile(i)) < ntiles && !b->abort; ++i) {
        const SlTile tile = tiles[t];
        const SlGroup g = groups[tile.group];
        const uint8_t *u = img + g.u_img + (int64_t)tile.ut * g.kc * kSlUnitU;
        const uint8_t *v = img + g.v_img + (int64_t)tile.vt * g.kc * kSlUnitV;
        const int c0 = tile.part * g.kpart, c1 = min(g.kc, c0 + g.kpart);
        for (int c = c0; c < c1; ++c, ++G) {
          const uint32_t s = G % kSlStages;
          if (G >= kSlStages && !wait_phase(&b->empty[s], ((G / kSlStages) - 1) & 1)) {
            sl_fail(b, flags);
            break;
          }
          uint8_t *st = smem + s * kSlStageBytes;
          tc::mbar_expect_tx(&b->full[s], (uint32_t)kSlStageBytes);
          tc::bulk_g2s(st, u + (int64_t)c * kSlUnitU, (uint32_t)kSlUnitU, &b->full[s]);
          tc::bulk_g2s(st + kSlUnitU, v + (int64_t)c * kSlUnitV, (uint32_t)kSlUnitV, &b->full[s]);
        }
      }
      // no copy is in flight when the block ends
      for (uint32_t k = G < kSlStages ? 0 : G - kSlStages; k < G; ++k)
        if (!wait_phase(&b->full[k % kSlStages], (k / kSlStages) & 1)) sl_fail(b, flags);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(kSlU, kSlV);
      uint32_t G = 0, n = 0;  // K steps, chunks so far
      bool ok = true;
      for (int i = 0, t; (t = tc::snake_tile(i)) < ntiles && ok && !b->abort; ++i) {
        const SlGroup &g = groups[tiles[t].group];
        const int kc = min(g.kpart, g.kc - tiles[t].part * g.kpart);
        for (int c = 0; c < kc && ok; ++c, ++G) {
          const bool first = c % kSlChunk == 0;
          if (first) {
            if (n > 0 && !wait_phase(&b->tempty, (n - 1) & 1)) {
              ok = false;
              break;
            }
            ++n;
          }
          const uint32_t s = G % kSlStages;
          if (!wait_phase(&b->full[s], (G / kSlStages) & 1)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint32_t su = tc::smem_u32(smem + s * kSlStageBytes);
          const uint32_t sv = su + (uint32_t)kSlUnitU;
          constexpr uint32_t planeU = kSlU * kSlK * 2, planeV = kSlV * kSlK * 2;
#pragma unroll
          for (int u = 0; u < kSlDigits; ++u) {
            const uint64_t ad =
                tc::make_desc(su + u * planeU, (kSlU / 8) * 128, 128);
#pragma unroll
            for (int j = 0; j < kSlDigits; ++j) {
              if (u + j >= kSlLevels) break;
              const uint64_t bd =
                  tc::make_desc(sv + j * planeV, (kSlV / 8) * 128, 128);
              // digit pair (0, l) is the first product of level l
              const uint32_t d = tmem + (u + j) * kSlV, acc = first && u == 0 ? 0u : 1u;
              // U plane u stays in the collector over its products
              if (u + 1 == kSlDigits)
                tc::mma_bf16(d, ad, bd, idesc, acc);
              else if (j == 0)
                tc::mma_bf16_a<tc::kCollectFill>(d, ad, bd, idesc, acc);
              else if (u + j + 1 == kSlLevels)
                tc::mma_bf16_a<tc::kCollectLast>(d, ad, bd, idesc, acc);
              else
                tc::mma_bf16_a<tc::kCollectUse>(d, ad, bd, idesc, acc);
            }
          }
          tc::mma_commit(&b->empty[s]);
          if (c % kSlChunk == kSlChunk - 1 || c == kc - 1) tc::mma_commit(&b->tfull);
        }
      }
      if (!ok) sl_fail(b, flags);
      tc::mma_commit(&b->fin);  // every MMA of this CTA has completed
      if (!wait_phase(&b->fin, 0)) sl_fail(b, flags);
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;  // lane quarter, column part
    uint32_t n = 0;  // chunks so far
    for (int i = 0, t; (t = tc::snake_tile(i)) < ntiles; ++i) {
      const SlTile tile = tiles[t];
      const SlGroup g = groups[tile.group];
      // the lane's own line, and lane j's register line j
      const int64_t ui = (int64_t)tile.ut * kSlU + q * 32 + lane;
      const bool uok = ui < g.nu;
      const SlLine ul = uok ? lines[g.u0 + ui] : SlLine{0, 0, 0, 0};
      const int64_t vi = (int64_t)tile.vt * kSlV + part * kSlCols + lane;
      const bool vok = lane < kSlCols && vi < g.nv;
      const SlLine vl = vok ? lines[g.v0 + vi] : SlLine{-1, 0, 0, 0};
      // a line without nonzero elements has scale 0: its sums are zero
      const int ue = (uok ? scale[2 + g.u0 + ui] >> 20 : 0) - 1022;
      const int ve = (vok ? scale[2 + g.v0 + vi] >> 20 : 0) - 1022;
      SlSum sum[kSlCols];
#pragma unroll
      for (int j = 0; j < kSlCols; ++j) sum[j] = SlSum{0, 0};
      bool ok = true;
      // pieces entirely past the result's edge are neither read nor rounded
      const bool live = tile.ut * kSlU + q * 32 < g.nu &&
                        tile.vt * kSlV + part * kSlCols < g.nv;
      const int kc = min(g.kpart, g.kc - tile.part * g.kpart);
      for (int c0 = 0; c0 < kc; c0 += kSlChunk, ++n) {
        if (b->abort || !wait_phase(&b->tfull, n & 1)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + part * kSlCols;
        if (live)
#pragma unroll
        for (int cb = 0; cb < kSlCols / 2; ++cb) {
          uint32_t r[kSlLevels][2];
#pragma unroll
          for (int l = 0; l < kSlLevels; ++l) tmem_ld2(base + l * kSlV + cb * 2, r[l]);
          tc::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            int v[kSlLevels];
#pragma unroll
            for (int l = 0; l < kSlLevels; ++l) v[l] = __float2int_rn(__uint_as_float(r[l][j]));
            sl_add(sum[cb * 2 + j],
                   (int64_t)v[0] * (1 << 24) + (int64_t)v[1] * (1 << 16) +
                       (int64_t)v[2] * (1 << 8) + (int64_t)v[3],
                   (int64_t)v[4] * (1 << 24) + (int64_t)v[5] * (1 << 16) +
                       (int64_t)v[6] * (1 << 8) + (int64_t)v[7]);
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&b->tempty);
      }
      if (!ok) {
        if (lane == 0) sl_fail(b, flags);
        break;
      }
      if (!live) continue;
      if (tile.part0 >= 0) {
        // the integer sums of this K part; the warp that arrives last for its
        // piece of the tile adds the others' (exact, so the order is free)
        const int w = q * kSlParts + part;
        auto slot = [&](int p) {
          return scratch + ((int64_t)(tile.part0 + p) * kSlU * kSlV + w * (32 * kSlCols) + lane);
        };
        longlong2 *mine = slot(tile.part);
#pragma unroll
        for (int j = 0; j < kSlCols; ++j) __stcg(mine + 32 * j, make_longlong2(sum[j].hi, sum[j].lo));
        __threadfence();
        __syncwarp();
        int before = 0;
        if (lane == 0) before = atomicAdd(arrived + (int64_t)tile.part0 * 16 + w, 1);
        if (__shfl_sync(0xffffffffu, before, 0) != g.parts - 1) continue;
        __threadfence();
        for (int p = 0; p < g.parts; ++p) {
          if (p == tile.part) continue;
          const longlong2 *o = slot(p);
#pragma unroll
          for (int j = 0; j < kSlCols; ++j) {
            const longlong2 x = __ldcg(o + 32 * j);
            sl_add(sum[j], x.x, x.y);
          }
        }
      }
      // within a block consecutive register lines are a fixed stride apart
      int64_t at = -1;
      int blk = -1;
      const int64_t step = g.lanes_n ? ul.w : 1;
#pragma unroll
      for (int j = 0; j < kSlCols; ++j) {
        const double x = sl_round(sum[j], ue + __shfl_sync(0xffffffffu, ve, j));
        const int bj = __shfl_sync(0xffffffffu, vl.blk, j);
        at += step;
        if (bj != blk) {  // warp-uniform
          blk = bj;
          const int loc = __shfl_sync(0xffffffffu, vl.loc, j);
          const int w = __shfl_sync(0xffffffffu, vl.w, j);
          const int64_t cb =
              bj < 0 || !uok ? -1
                             : cblk[g.cb0 + (g.lanes_n ? (int64_t)bj * g.ncb + ul.blk
                                                       : (int64_t)ul.blk * g.ncb + bj)];
          at = cb < 0 ? INT64_MIN / 2
                      : cb + (g.lanes_n ? (int64_t)loc * ul.w + ul.loc : (int64_t)ul.loc * w + loc);
        }
        if (at >= 0) C[at] = x;
      }
    }
  }
  tc::pdl_launch_dependents();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

}  // namespace

SlicePlan::~SlicePlan() {
  if (!ctx) return;
  ctx->free(d_block);
  ctx->free(img);
}

int SlicePlan::add_group(const Dims &d, const std::vector<SlLine> &rows,
                         const std::vector<SlLine> &cols, const std::vector<int64_t> &blocks,
                         bool upper) {
  auto tiles_of = [](int64_t n, int t) { return (n + t - 1) / t; };
  SlGroup g{};
  // the side of 128-row tiles: the one that pads less, C's columns on a tie
  // (consecutive lanes then store consecutive elements)
  const int64_t wn = tiles_of(d.N, kSlU) * kSlU * tiles_of(d.M, kSlV) * kSlV;
  const int64_t wm = tiles_of(d.M, kSlU) * kSlU * tiles_of(d.N, kSlV) * kSlV;
  g.lanes_n = wn <= wm ? 1 : 0;
  g.nu = (int32_t)(g.lanes_n ? d.N : d.M);
  g.nv = (int32_t)(g.lanes_n ? d.M : d.N);
  g.kc = (int32_t)((d.K + kSlK - 1) / kSlK);
  g.u0 = (int64_t)lines.size();
  const std::vector<SlLine> &u = g.lanes_n ? cols : rows, &v = g.lanes_n ? rows : cols;
  lines.insert(lines.end(), u.begin(), u.end());
  g.v0 = (int64_t)lines.size();
  lines.insert(lines.end(), v.begin(), v.end());
  g.cb0 = (int64_t)cblk.size();
  int32_t ncb = 0;
  for (const SlLine &l : cols) ncb = std::max(ncb, l.blk + 1);
  g.ncb = ncb;
  cblk.insert(cblk.end(), blocks.begin(), blocks.end());
  g.upper = upper ? 1 : 0;
  const int64_t ut = tiles_of(g.nu, kSlU), vt = tiles_of(g.nv, kSlV);
  g.u_img = img_bytes;
  img_bytes += ut * g.kc * kSlUnitU;
  g.v_img = img_bytes;
  img_bytes += vt * g.kc * kSlUnitV;
  const int32_t id = (int32_t)groups.size();
  if (d.K % kSlK) holes = true;
  groups.push_back(g);
  return id;
}

void SlicePlan::add_op(int group, SlOp op) {
  const SlGroup &g = groups[group];
  const bool is_u = (op.src == 1) == (g.lanes_n == 1);  // operand B holds C's columns
  op.img_off = is_u ? g.u_img : g.v_img;
  op.sc0 = is_u ? g.u0 : g.v0;
  op.tr = is_u ? kSlU : kSlV;
  op.kc = g.kc;
  // lanes walk the source's contiguous direction
  const bool rf = op.nr > 0 && op.re[op.nr - 1] > 1 && (op.nk == 0 || op.ke[op.nk - 1] == 1 ||
                                                        op.rs[op.nr - 1] < op.ks[op.nk - 1]);
  op.rows_fast = rf ? 1 : 0;
  ops.push_back(op);
}

void SlicePlan::finalize() {
  items_k.clear();
  items_t.clear();
  // fewer columns per item where the items of a warp's full width would leave
  // SMs without work
  auto by_cols = [](const SlOp &op) {
    return !op.rows_fast && op.nk <= 1 && (op.nk == 0 || op.ks[0] <= 2);
  };
  int64_t wide = 0;
  for (const SlOp &op : ops)
    if (by_cols(op))
      wide += (int64_t)((op.rows + kPackRows - 1) / kPackRows) *
              ((op.cols + kPackCols - 1) / kPackCols);
  const int width = wide < 4 * kPackWarps * ctx->num_sms ? 32 : kPackCols;
  for (int src = 0; src < 2; ++src) {
    for (size_t o = 0; o < ops.size(); ++o) {
      const SlOp &op = ops[o];
      if (op.src != src) continue;
      if (by_cols(op)) {
        for (int32_t r = 0; r < op.rows; r += kPackRows)
          for (int32_t k = 0; k < op.cols; k += width)
            items_k.push_back({(int32_t)o, r, k, width});
      } else {
        for (int32_t r = 0; r < op.rows; r += 32)
          for (int32_t k = 0; k < op.cols; k += 64) items_t.push_back({(int32_t)o, r, k, 64});
      }
    }
    if (src == 0) {
      first_k = (int)items_k.size();
      first_t = (int)items_t.size();
    }
  }
  // K parts: a unit of work is at most about a third of one SM's share of the
  // K steps, so that few large tiles (long contractions with small results)
  // still fill the chip; parts cost 16 B per output and part of L2 traffic.
  // Last stage of the effective Hamiltonian without parts / halves / thirds /
  // sixths: ladder D = 300 174 / 105 / 106 / 106 us, D = 512 299 / 205 / 197 /
  // 221 us, Hubbard D = 1000 209 / 184 / 201 / 201 us.
  auto of_group = [&](auto &&fn) {
    for (size_t id = 0; id < groups.size(); ++id) {
      const SlGroup &g = groups[id];
      const int es = std::max(1, g.lanes_n ? g.nu / std::max(g.nv, 1) : g.nv / std::max(g.nu, 1));
      for (int32_t i = 0; i * kSlU < g.nu; ++i)
        for (int32_t j = 0; j * kSlV < g.nv; ++j) {
          if (g.upper) {  // rows m, columns n: drop tiles with every n < m
            const int n1 = (g.lanes_n ? i * kSlU + kSlU - 1 : j * kSlV + kSlV - 1) / es;
            if ((g.lanes_n ? j * kSlV : i * kSlU) > n1) continue;
          }
          fn((int32_t)id, i, j);
        }
    }
  };
  double steps = 0;
  of_group([&](int32_t id, int32_t, int32_t) { steps += groups[id].kc; });
  const int unit = std::max<int>(
      kSlChunk, ((int)(steps / ctx->num_sms / 3) + kSlChunk - 1) / kSlChunk * kSlChunk);
  for (SlGroup &g : groups) {
    g.parts = std::max(1, std::min(8, (g.kc + unit / 2) / unit));
    const int per = (g.kc + g.parts - 1) / g.parts;
    g.kpart = std::max(kSlChunk, (per + kSlChunk - 1) / kSlChunk * kSlChunk);
    g.parts = std::max(1, (g.kc + g.kpart - 1) / g.kpart);
  }
  tiles.clear();
  slots = 0;
  of_group([&](int32_t id, int32_t i, int32_t j) {
    const int32_t p0 = groups[id].parts > 1 ? (int32_t)slots : -1;
    for (int32_t p = 0; p < groups[id].parts; ++p) tiles.push_back({id, i, j, p, p0, 0});
    if (p0 >= 0) slots += groups[id].parts;
  });
  // most K steps first (longest processing time first over the persistent grid)
  auto cost = [&](const SlTile &t) {
    const SlGroup &g = groups[t.group];
    return std::min(g.kpart, g.kc - t.part * g.kpart);
  };
  std::vector<int> count;
  for (const SlTile &t : tiles) {
    const int c = cost(t);
    if ((int)count.size() <= c) count.resize(c + 1, 0);
    count[c]++;
  }
  std::vector<int> at(count.size(), 0);
  for (int c = (int)count.size() - 1, sum = 0; c >= 0; sum += count[c], --c) at[c] = sum;
  std::vector<SlTile> sorted(tiles.size());
  for (const SlTile &t : tiles) sorted[at[cost(t)]++] = t;
  tiles.swap(sorted);
}

void SlicePlan::upload() {
  UploadBatch up(*ctx);
  const size_t o0 = up.add(ops), o1 = up.add(items_k), o1t = up.add(items_t),
               o2 = up.add(groups), o3 = up.add(tiles),
               o4 = up.add(lines), o5 = up.add(cblk),
               o6 = up.reserve(nscale() * sizeof(int)),
               o7 = up.reserve(slots * kSlU * kSlV * sizeof(longlong2));
  d_block = up.commit();
  d_ops = (SlOp *)(d_block + o0);
  d_items_k = (SlItem *)(d_block + o1);
  d_items_t = (SlItem *)(d_block + o1t);
  d_groups = (SlGroup *)(d_block + o2);
  d_tiles = (SlTile *)(d_block + o3);
  d_lines = (SlLine *)(d_block + o4);
  d_cblk = (int64_t *)(d_block + o5);
  scale = (int *)(d_block + o6);
  scratch = (longlong2 *)(d_block + o7);
  img = (uint8_t *)ctx->alloc(std::max<int64_t>(img_bytes, 1));
  if (holes) UDMRG_CHECK_CUDA(cudaMemsetAsync(img, 0, img_bytes, ctx->stream));
}

double SlicePlan::seconds() const {
  double steps = 0, elems = 0;
  for (const SlTile &t : tiles) steps += std::min(groups[t.group].kpart, groups[t.group].kc) + 2.0;
  for (const SlOp &o : ops) elems += (double)o.rows * o.cols;
  return 30e-6 + steps * 0.7e-6 / ctx->num_sms + elems * 30.0 / 3e12;
}

void SlicePlan::clear_scales() const {
  UDMRG_CHECK_CUDA(cudaMemsetAsync(scale, 0, nscale() * sizeof(int), ctx->stream));
}

void run_slice(Ctx &ctx, const SlicePlan &p, const double *a, const double *b, double *c) {
  if (p.tiles.empty()) return;
  if (!p.prescaled) p.clear_scales();
  const int nk = (int)p.items_k.size(), nx = (int)p.items_t.size();
  const int k0 = p.prescaled ? p.first_k : 0, t0 = p.prescaled ? p.first_t : 0;
  auto k_blocks = [&](int n) {
    return std::min((n + kPackWarps - 1) / kPackWarps, 16 * ctx.num_sms);
  };
  auto grid = [&](int n, int m) { return k_blocks(n) + std::min(m, 8 * ctx.num_sms); };
  if (grid(nk - k0, nx - t0)) {
    slice_scale_kernel<<<grid(nk - k0, nx - t0), kPackThreads, 0, ctx.stream>>>(
        p.d_ops, p.d_items_k + k0, nk - k0, k_blocks(nk - k0), p.d_items_t + t0, nx - t0, a, b,
        p.scale);
    UDMRG_CHECK_CUDA(cudaGetLastError());
    ctx.launches++;
  }
  if (grid(nk, nx)) {
    UDMRG_CHECK_CUDA(tc::launch_pdl(slice_pack_kernel, dim3(grid(nk, nx)), dim3(kPackThreads), 0,
                                    ctx.stream, p.d_ops, p.d_items_k, nk, k_blocks(nk),
                                    p.d_items_t, nx, a, b, p.scale, p.img));
    ctx.launches++;
  }
  ctx.allow_smem((const void *)slice_gemm_kernel, kSlSmem);
  const int nt = (int)p.tiles.size();
  UDMRG_CHECK_CUDA(tc::launch_pdl(slice_gemm_kernel, dim3(std::min(nt, ctx.num_sms)),
                                  dim3(kSlThreads), kSlSmem, ctx.stream, p.d_tiles, nt,
                                  p.d_groups, p.d_lines, p.d_cblk, p.scale, p.img, c, p.scale,
                                  p.scratch, p.scale + 2 + p.lines.size()));
  ctx.launches++;
}

}  // namespace udmrg
