// FP64-accurate grouped GEMM on the tcgen05 tensor cores by digit slicing (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59
// (2012) 95, with exact integer slices).
//
// This GPU multiplies FP64 at two FMAs per clock and SM; its BF16 tensor rate
// is about 1500 times that.  Every row of either operand is scaled by a power
// of two to |x| < 1 and cut into eight signed digits of 8 bits (the leading one
// of 6: 62 bits below the row's power of two), each exact in BF16.  The products
// of digit s of one operand and digit t of the other have weight
// 2^-(12 + 8 (s + t)); those with s + t <= 7 (36 of the 64 pairs) are summed in
// FP32 TMEM accumulators, one per level s + t.  The sums of levels 0 .. 4 are
// integers of at most 2^24 for 256-deep K, so they are exact.  The epilogue
// adds the eight levels of an output in 64-bit integers (over all 256-deep K
// chunks) and rounds once to FP64, without an FP64 instruction.
//
// Error: one FP64 rounding of the result, and per product of the two lines' scales
// 2^-62 for the operands' last digits and 2^-59.2 for the dropped pairs (seven of
// level 8, below 2^14 each): K 2^-57 rowmax colmax, since a scale is at most twice
// its line's maximum.  Sums of levels 5 .. 7 can reach 1.75 2^24, where FP32 has
// units of two; only where nearly all digits of a 256-deep run agree in sign and
// size, and then by at most four units of level 5 (2^-50 of the scales) per
// product.
// The bound is to the lines' maxima, not to the terms of the sum as that of FP64
// FMAs: elements more than 2^9 below their line's maximum keep fewer than 53
// bits, so a small term that meets no large one (a product with an identity, an
// output of graded lines whose large parts meet zeros) is not correct to its own
// last bit.  In norm the form is the more accurate one: 1.0e-16 against the
// FMAs' 7.5e-16 for an effective-Hamiltonian product (Heisenberg, D = 308, in
// extended precision).
//
// The GEMMs of a block contraction are merged into one dense GEMM per set of
// blocks that share contracted sectors (a quantum-number flow); sub-matrices
// that no block fills stay zero in the operand images.
#pragma once

#include <memory>

#include "btensor.hpp"

namespace udmrg {

constexpr int kSlDigits = 8;
constexpr int kSlLevels = 8;
constexpr int kSlU = 128;  // image rows of a U tile (UMMA M, TMEM lanes)
constexpr int kSlV = 64;   // image rows of a V tile (UMMA N)
constexpr int kSlK = 16;   // K per step (one MMA per digit pair)
constexpr int kSlChunk = 16;  // K steps per accumulation: 256-deep sums stay exact
constexpr int64_t kSlUnitU = (int64_t)kSlDigits * kSlU * kSlK * 2;
constexpr int64_t kSlUnitV = (int64_t)kSlDigits * kSlV * kSlK * 2;

// One sub-matrix of an operand: element (r, k), r and k decomposed row-major
// over their sub-dimension extents, at src[src_off + sum r_j rs[j] + sum k_j
// ks[j]] (doubles), lands at image row r0 + r * rstep, column k0 + k.
struct SlOp {
  int64_t src_off;
  int64_t rs[4], ks[4];
  int32_t re[4], ke[4];
  int32_t nr, nk;
  int32_t rows, cols;
  int64_t img_off;  // byte offset of the operand's image in its group
  int64_t sc0;      // scale entry of image row 0
  int32_t r0, k0, rstep, kc;  // k0: a multiple of 8; kc: K steps of the image
  int32_t tr;       // rows per image tile (kSlU or kSlV)
  int32_t src;      // 0: operand A, 1: operand B
  int32_t neg;      // negated values
  int32_t rows_fast;  // rows are the contiguous direction of the source
};
struct SlItem {  // work item of the scale and pack kernels: rows from r0, width columns from k0
  int32_t op, r0, k0, width;
};

// Output address of (lane line u, register line v): with lanes along C's
// columns base[v.blk][u.blk] + v.loc * u.w + u.loc, with lanes along C's rows
// base[u.blk][v.blk] + u.loc * v.w + v.loc; base < 0: the block is absent.
struct SlLine {
  int32_t blk, loc, w, pad;
};
struct SlGroup {
  int64_t u_img, v_img;  // byte offsets of the images
  int64_t u0, v0;        // first line (and scale) of the U / V side
  int64_t cb0;           // first entry of the group's block table
  int32_t nu, nv;        // lines of the U / V side
  int32_t kc;            // K steps
  int32_t ncb;           // columns of the block table (C column blocks)
  int32_t lanes_n;       // lanes along C's columns
  int32_t upper;         // square: entries below the diagonal are not needed
  int32_t parts, kpart;  // K parts of a tile, K steps of each (a multiple of kSlChunk)
};
// One K part of an output tile.  Tiles of several parts leave their integer
// sums at part0 in the scratch; the part that arrives last adds them up.
struct SlTile {
  int32_t group, ut, vt, part;
  int32_t part0, pad;  // first of the tile's slots in the scratch (-1: one part)
};

struct SlicePlan {
  Ctx *ctx = nullptr;
  std::vector<SlOp> ops;
  // of ops with contiguous columns, of the others; the first operand's first
  std::vector<SlItem> items_k, items_t;
  int first_k = 0, first_t = 0;  // the first operand's
  std::vector<SlGroup> groups;
  std::vector<SlTile> tiles;
  std::vector<SlLine> lines;
  std::vector<int64_t> cblk;
  int64_t slots = 0;  // scratch slots (one per part of a tile with several)
  int64_t img_bytes = 0;
  bool prescaled = false;  // the first operand's scales are found by its producer
  bool holes = false;  // image entries no op writes
  uint8_t *d_block = nullptr;  // the tables and scale
  SlOp *d_ops = nullptr;
  SlItem *d_items_k = nullptr, *d_items_t = nullptr;
  SlGroup *d_groups = nullptr;
  SlTile *d_tiles = nullptr;
  SlLine *d_lines = nullptr;
  int64_t *d_cblk = nullptr;
  uint8_t *img = nullptr;
  // flags[0]: an operand is out of the sliced range (non-finite, or a row
  // maximum outside 2^-476 .. 2^476), flags[1]: a bounded wait ran out; then
  // one scale entry per line, then the arrival counters of the scratch slots
  int *scale = nullptr;
  longlong2 *scratch = nullptr;
  SlicePlan() = default;
  SlicePlan(const SlicePlan &) = delete;
  SlicePlan &operator=(const SlicePlan &) = delete;
  ~SlicePlan();

  // Adds a dense group C(M x N) = A(M x K) B(K x N) (doubles; K may hold a
  // complex embedding); the caller then adds the ops of both operands with
  // add_op and the lines.  Returns the group's id.
  struct Dims {
    int64_t M, N, K;
  };
  int add_group(const Dims &d, const std::vector<SlLine> &rows, const std::vector<SlLine> &cols,
                const std::vector<int64_t> &blocks, bool upper);
  // op: strides, extents, rows, cols, src, r0, k0, rstep, neg set by the caller
  void add_op(int group, SlOp op);
  double seconds() const;  // the cost model's estimate
  void finalize();         // items, K parts and tile order (host)
  void upload();           // device tables and workspaces
  void clear_scales() const;  // device: flags, scales, counters to zero
  size_t nscale() const { return 2 + lines.size() + 16 * (size_t)slots; }
};

// C = A B for every group; sets the plan's flags where the sliced form does
// not apply (the caller's FP64 kernels then run, gated on them).
void run_slice(Ctx &ctx, const SlicePlan &p, const double *a, const double *b, double *c);

}  // namespace udmrg
