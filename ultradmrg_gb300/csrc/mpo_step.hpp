// The MPO step of the two-site matvec, T3 = (W1 W2) T1, as a sparse channel
// map on CUDA cores.
//
// In the four-step contraction of eff_ham_mul_two_site_state
// (lanczos_vmps_solver_impl.h:268-272) the two middle steps contract T1 with
// the MPO tensors, whose sector dimensions are a few elements: as GEMMs their
// K and N are tiny and the tiles are mostly padding.  Here the two MPO
// tensors are first contracted over their shared bond (FusedMpo, per target
// sector triple), then every (A', B) sector pair of T1/T3 becomes one small
// dense channel map: out[o](a', b) = sum_i C[o][i] in[i](a', b), applied per
// (a', b) by one warp for 64 of them.  The single MPO tensor of an environment
// update and of the one-site product is such a map too.
#pragma once

#include <array>
#include <map>

#include "btensor.hpp"
#include "slice_gemm.hpp"

namespace udmrg {

// W1 (w, s1, s1', wr) and W2 (wr, s2, s2', w2) contracted over wr, by the
// output sector triple (S1', S2', W2): the contributing input sectors
// (W, S1, S2) with their dense coefficient matrices coef[ic * nout + oc],
// ic = (w ds1 + s1) ds2 + s2, oc = (s1' ds2' + s2') dw2 + w2.  Host side;
// zero matrices are dropped.  real: every imaginary part of complex MPO tensors
// is zero (an MPO promoted to complex with its state); only then may get be called.
struct FusedMpo {
  struct Entry {
    std::array<int32_t, 3> src;  // (W, S1, S2)
    std::vector<double> coef;
  };
  const BTensor &W1, &W2;
  std::vector<double> w1h, w2h;
  bool real = true;
  std::map<int32_t, std::vector<int64_t>> w1_by_s1o;
  std::map<std::array<int32_t, 3>, std::vector<int64_t>> w2_by;  // (wr, s2', w2)
  std::map<std::array<int32_t, 3>, std::vector<Entry>> cache;
  FusedMpo(Ctx &ctx, const BTensor &W1, const BTensor &W2);
  const std::vector<Entry> &get(int32_t S1p, int32_t S2p, int32_t W2s);
};

// FP64 form: T1 (A', W, S1, S2, B) to T3 (A', S1', S2', W2, B), both row-major
// block tensors with b contiguous, so reads, writes and the next step's K runs
// are contiguous.  The coefficients are real; complex data are moved as twice
// as many reals.  Offsets and strides in doubles.
struct MpoNz64 {
  int64_t base;  // input channel at (a' = 0, b = 0)
  double v;
  int32_t astride, pad;  // doubles between consecutive a'
};
struct MpoOut64 {
  int64_t base;
  int32_t astride;
  int32_t line, step, pad;  // scale entry at a' = 0 (-1: none), entries between a'
};
struct MpoPair64 {
  int32_t out0, nout;
  int32_t row0, da, db, pad;  // row0: first CSR row of the pair; db in doubles
};
struct MpoTask64 {  // 64 consecutive (a', b) entries of a pair, channels o0 .. o1 - 1
  int32_t pair, u0, o0, o1;
};

struct MpoStep64 {
  Ctx *ctx = nullptr;
  std::vector<MpoPair64> pairs;
  std::vector<MpoOut64> outs;
  std::vector<int32_t> rowptr;
  std::vector<MpoNz64> nz;
  std::vector<MpoTask64> tasks;
  uint8_t *d_block = nullptr;
  MpoPair64 *d_pairs = nullptr;
  MpoOut64 *d_outs = nullptr;
  int32_t *d_rowptr = nullptr;
  MpoNz64 *d_nz = nullptr;
  MpoTask64 *d_tasks = nullptr;
  double flops = 0;  // 2 per nonzero coupling and (a', b) entry
  ~MpoStep64();
};

// The tables (host only: safe on a host thread with its own FusedMpo), for the
// block structures of the two outer steps' intermediates.  Every T3 entry is
// written (zero where no coupling reaches it).
std::unique_ptr<MpoStep64> build_mpo_step64(FusedMpo &fm, const BTensor &T1, const BTensor &T3);
// One MPO tensor W (data wh, real): T (a, x1, x2, b) to out (a, y1, y2, b) over
// W's axes x1, x2; y1, y2 are W's two others in ascending order.
std::unique_ptr<MpoStep64> build_mpo_map(const BTensor &T, const BTensor &W,
                                         const std::vector<double> &wh, int x1, int x2,
                                         const BTensor &out);
// Host copy of an MPO tensor's real parts; *real = no nonzero imaginary part.
std::vector<double> mpo_data(Ctx &ctx, const BTensor &w, bool *real);
void upload_mpo_step64(Ctx &ctx, MpoStep64 &p);
// Lets the step find the scales of T3, the next sliced GEMM's first operand: its
// scale pass need not read T3 again.  Before upload_mpo_step64; true where every
// channel's row of b lies within one line of the operand (its rows of b are K
// runs); p then runs with next, before it.
bool link_scales(MpoStep64 &p, SlicePlan *next);
void run_mpo_step64(Ctx &ctx, const MpoStep64 &p, const double *t1, double *t3,
                    const SlicePlan *next = nullptr);

}  // namespace udmrg
