// MPO step of the mixed-precision matvec: T3 = (W1 W2) T1 on CUDA cores,
// grouped by (A', B) sector pair.  A thread owns one unit (pair, a', 8-wide
// chunk of b): for each output channel of the pair it accumulates the
// coefficient-weighted input chunks (two 16-byte loads of FP32 T1 per
// nonzero, read straight from global memory: an input channel serves ~1.25
// outputs, the second use hits L1), splits the eight sums into three BF16
// planes and writes each plane with one 16-byte store into the step-3 tile
// image.  A warp takes 32 consecutive units of one pair, so the CSR walk over
// the pair's nonzeros is warp-uniform (broadcast metadata loads, no
// divergence).  The pair's nonzero records, channel ends and image targets
// are loaded 32 at a time, one per lane, and shuffled out; nonzeros are
// processed four at a time with their eight loads in flight.  Padded b columns (up to a multiple of 8) read and
// write zeros.  HBM bound: T1 read once (FP32), T3 written once (3 x BF16).
#include <cuda_bf16.h>

#include <climits>

#include "mpo_step.hpp"
#include "sg_matvec.hpp"
#include "tc_roles.cuh"

namespace udmrg {

namespace {

__device__ __forceinline__ int canon(int r, int k, int tr) {
  return (((k >> 3) * (tr >> 3) + (r >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1);
}

constexpr int kMpoWarps = 8;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kNzBatch = 4;  // nonzeros whose loads are in flight together

__global__ void __launch_bounds__(32 * kMpoWarps, 2)
    mpo_chunk_kernel(const MpoTask *__restrict__ tasks, int ntasks,
                     const MpoPair *__restrict__ pairs, const MpoOut *__restrict__ outs,
                     const int32_t *__restrict__ rowptr, const MpoNzRec *__restrict__ nzr,
                     const float *__restrict__ t1, uint8_t *__restrict__ img) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int64_t plane = (int64_t)kTcBM * kTcBK * 2;
  tc::pdl_wait();  // T1 from the L.psi GEMM
  for (int t = blockIdx.x * kMpoWarps + warp; t < ntasks; t += gridDim.x * kMpoWarps) {
    const MpoTask tk = tasks[t];
    MpoPair pr = pairs[tk.pair];
    pr.out0 += tk.o0;  // the task's output channels
    pr.row0 += tk.o0;
    pr.nout = tk.nout;
    const int nch = pr.dbp >> 3;
    const int u = tk.u0 + lane;
    const bool valid = u < pr.da * nch;
    const int a = valid ? u / nch : 0;
    const int c8 = valid ? (u - a * nch) * 8 : 0;
    const int kbeg = __ldg(rowptr + pr.row0), kend = __ldg(rowptr + pr.row0 + pr.nout);
    // Output channels [ob, ob + 32): lane l holds channel ob + l's end in the
    // nonzero list and its image target (loaded together, read by shuffles).
    int ob = 0;
    const bool has = lane < pr.nout;
    int endv = has ? __ldg(rowptr + pr.row0 + 1 + lane) : INT_MAX;
    MpoOut outv = has ? outs[pr.out0 + lane] : MpoOut{0, 0, 0, 0, 0};
    int o = 0;
    int next = __shfl_sync(kFull, endv, 0);  // end of output channel o's nonzeros
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    // write channel o's sums, then move to channel o + 1 (warp-uniform)
    auto finish = [&]() {
      const int sl = o - ob;
      const long long off0 = __shfl_sync(kFull, (long long)outv.img_off, sl);
      const int row0 = __shfl_sync(kFull, outv.row0, sl);
      const int rstride = __shfl_sync(kFull, outv.rstride, sl);
      const int col0 = __shfl_sync(kFull, outv.col0, sl);
      const int kc = __shfl_sync(kFull, outv.kc, sl);
      if (valid) {
        const int row = row0 + a * rstride;
        const int col = col0 + c8;
        const int64_t off = off0 + ((int64_t)(row >> 7) * kc + (col >> 6)) * 3 * plane +
                            canon(row & 127, col & 63, kTcBM);
        uint4 h, m, l;
        split8(acc, h, m, l);
        *(uint4 *)(img + off) = h;
        *(uint4 *)(img + off + plane) = m;
        *(uint4 *)(img + off + 2 * plane) = l;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      if (++o - ob == 32) {
        ob += 32;
        const bool h2 = ob + lane < pr.nout;
        endv = h2 ? __ldg(rowptr + pr.row0 + 1 + ob + lane) : INT_MAX;
        outv = h2 ? outs[pr.out0 + ob + lane] : MpoOut{0, 0, 0, 0, 0};
      }
      next = __shfl_sync(kFull, endv, o - ob);
    };
    // Nonzeros 32 at a time, one record per lane (shuffled out), eight
    // nonzeros' sixteen 16-byte loads in flight together.
    for (int kb = kbeg; kb < kend; kb += 32) {
      const int nb = min(32, kend - kb);
      MpoNzRec mine{0, 0, 0.f};
      if (lane < nb) mine = nzr[kb + lane];
      for (int q0 = 0; q0 < nb; q0 += kNzBatch) {
        float4 x[kNzBatch][2];
        float v[kNzBatch];
#pragma unroll
        for (int q = 0; q < kNzBatch; ++q) {
          const int sl = q0 + q;
          const long long base = __shfl_sync(kFull, (long long)mine.base, sl);
          const int astride = __shfl_sync(kFull, mine.astride, sl);
          v[q] = __shfl_sync(kFull, mine.v, sl);
          x[q][0] = x[q][1] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (sl < nb && valid) {
            const float4 *src = (const float4 *)(t1 + base + (int64_t)a * astride + c8);
            x[q][0] = __ldg(src);
            x[q][1] = __ldg(src + 1);
          }
        }
#pragma unroll
        for (int q = 0; q < kNzBatch; ++q) {
          if (q0 + q >= nb) break;
          while (kb + q0 + q >= next) finish();  // output channel o is complete
          acc[0] = fmaf(v[q], x[q][0].x, acc[0]);
          acc[1] = fmaf(v[q], x[q][0].y, acc[1]);
          acc[2] = fmaf(v[q], x[q][0].z, acc[2]);
          acc[3] = fmaf(v[q], x[q][0].w, acc[3]);
          acc[4] = fmaf(v[q], x[q][1].x, acc[4]);
          acc[5] = fmaf(v[q], x[q][1].y, acc[5]);
          acc[6] = fmaf(v[q], x[q][1].z, acc[6]);
          acc[7] = fmaf(v[q], x[q][1].w, acc[7]);
        }
      }
    }
    while (o < pr.nout) finish();  // the last channel and channels without nonzeros
  }
  tc::pdl_launch_dependents();
}

// FP64 form.  A warp takes 64 consecutive (a', b) entries of one pair, two per
// lane, and walks a run of the pair's couplings (32 records held one per lane,
// handed out by shuffles; the loads of four couplings' two entries in flight).
// 8 B read per T1 entry and written per T3 entry, both in contiguous runs of db;
// bound by the latency of the loads (Hubbard 4x8, D = 1000: 66 us, 2.2 TB/s).
// With scale, the maxima of T3's rows too: one per a' and channel where the
// task spans at most four a', else over runs of lanes of one a' (against a
// pass of its own over T3: 44 us).
__global__ void __launch_bounds__(256)
    mpo_map64_kernel(const MpoTask64 *__restrict__ tasks, int ntasks,
                     const MpoPair64 *__restrict__ pairs, const MpoOut64 *__restrict__ outs,
                     const int32_t *__restrict__ rowptr, const MpoNz64 *__restrict__ nz,
                     const double *__restrict__ t1, double *__restrict__ t3,
                     int *__restrict__ scale) {
  constexpr int kB = 4;  // couplings whose loads are in flight together
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  tc::pdl_wait();  // T1 from the L.psi GEMM
  for (int t = blockIdx.x * 8 + warp; t < ntasks; t += gridDim.x * 8) {
    const MpoTask64 tk = tasks[t];
    const MpoPair64 pr = pairs[tk.pair];
    const int u0 = tk.u0 + lane, u1 = u0 + 32, n = pr.da * pr.db;
    const bool v0 = u0 < n, v1 = u1 < n;
    const int a0 = v0 ? u0 / pr.db : 0, b0 = v0 ? u0 - a0 * pr.db : 0;
    const int a1 = v1 ? u1 / pr.db : 0, b1 = v1 ? u1 - a1 * pr.db : 0;
    const int kbeg = __ldg(rowptr + pr.row0 + tk.o0), kend = __ldg(rowptr + pr.row0 + tk.o1);
    // scales: few a' over the task, or runs of lanes of one a' (bit i of run:
    // lane + 2^i belongs to the lane's run; bit 5: first of its run)
    const int alo = tk.u0 / pr.db, na = (min(tk.u0 + 64, n) - 1) / pr.db - alo + 1;
    uint32_t run0 = 0, run1 = 0;
    if (scale && na > 4) {
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const int d = 1 << i;
        const int p = __shfl_down_sync(kFull, a0, d), q = __shfl_down_sync(kFull, a1, d);
        run0 |= (lane + d < 32 && p == a0) << i;
        run1 |= (lane + d < 32 && q == a1) << i;
      }
      const int p = __shfl_up_sync(kFull, a0, 1), q = __shfl_up_sync(kFull, a1, 1);
      run0 |= (lane == 0 || p != a0) << 5;
      run1 |= (lane == 0 || q != a1) << 5;
    }
    auto run_max = [&](int v, uint32_t run, int *at) {
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const int w = __shfl_down_sync(kFull, v, 1 << i);
        if (run >> i & 1) v = max(v, w);
      }
      if ((run >> 5 & 1) && v) atomicMax(at, v);
    };
    int o = tk.o0;
    int next = __ldg(rowptr + pr.row0 + o + 1);  // end of output channel o's couplings
    double s0 = 0.0, s1 = 0.0;
    auto finish = [&]() {  // warp-uniform: write channel o, move to o + 1
      const MpoOut64 ot = outs[pr.out0 + o];
      if (v0) t3[ot.base + (int64_t)a0 * ot.astride + b0] = s0;
      if (v1) t3[ot.base + (int64_t)a1 * ot.astride + b1] = s1;
      if (scale && ot.line >= 0) {
        const int h0 = v0 ? tc::abs_high(s0) : 0, h1 = v1 ? tc::abs_high(s1) : 0;
        int *at = scale + 2 + ot.line;
        if (na <= 4) {
          int best = 0;  // of a' = alo + lane
          for (int i = 0; i < na; ++i) {
            const int v = __reduce_max_sync(
                kFull, max(a0 == alo + i ? h0 : 0, a1 == alo + i ? h1 : 0));
            if (lane == i) best = v;
          }
          if (best) atomicMax(at + (int64_t)(alo + lane) * ot.step, best);
        } else {
          run_max(h0, run0, at + (int64_t)a0 * ot.step);
          run_max(h1, run1, at + (int64_t)a1 * ot.step);
        }
      }
      s0 = s1 = 0.0;
      if (++o < tk.o1) next = __ldg(rowptr + pr.row0 + 1 + o);
    };
    for (int kb = kbeg; kb < kend; kb += 32) {
      const int nb = min(32, kend - kb);
      MpoNz64 mine{0, 0.0, 0, 0};
      if (lane < nb) mine = nz[kb + lane];
      for (int q0 = 0; q0 < nb; q0 += kB) {
        double x0[kB], x1[kB], c[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          const long long base = __shfl_sync(kFull, (long long)mine.base, q0 + q);
          const int as = __shfl_sync(kFull, mine.astride, q0 + q);
          c[q] = __shfl_sync(kFull, mine.v, q0 + q);
          const bool ok = q0 + q < nb;
          x0[q] = ok && v0 ? __ldg(t1 + base + (int64_t)a0 * as + b0) : 0.0;
          x1[q] = ok && v1 ? __ldg(t1 + base + (int64_t)a1 * as + b1) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          if (q0 + q >= nb) break;
          while (kb + q0 + q >= next) finish();
          s0 = fma(c[q], x0[q], s0);
          s1 = fma(c[q], x1[q], s1);
        }
      }
    }
    while (o < tk.o1) finish();  // the last channel and channels without couplings
  }
}

}  // namespace

void run_mpo_step64(Ctx &ctx, const MpoStep64 &p, const double *t1, double *t3,
                    const SlicePlan *next) {
  const int ntasks = (int)p.tasks.size();
  const bool scales = next && next->prescaled;
  if (scales) next->clear_scales();
  if (ntasks == 0) return;
  const int grid = std::min((ntasks + 7) / 8, 16 * ctx.num_sms);
  UDMRG_CHECK_CUDA(tc::launch_pdl(mpo_map64_kernel, dim3(grid), dim3(256), 0, ctx.stream,
                                  p.d_tasks, ntasks, p.d_pairs, p.d_outs, p.d_rowptr, p.d_nz, t1,
                                  t3, scales ? next->scale : nullptr));
  ctx.launches++;
}

void run_mpo_step(Ctx &ctx, const SgMatvecPlan &p) {
  const int ntasks = (int)p.tasks.size();
  if (ntasks == 0) return;
  const int blocks = (ntasks + kMpoWarps - 1) / kMpoWarps;
  const int grid = std::min(blocks, 16 * ctx.num_sms);
  UDMRG_CHECK_CUDA(tc::launch_pdl(mpo_chunk_kernel, dim3(grid), dim3(32 * kMpoWarps), 0,
                                  ctx.stream, p.d_tasks, ntasks, p.d_pairs, p.d_outs, p.d_rowptr,
                                  p.d_nz, p.t1, p.t3_img));
  ctx.launches++;
}

}  // namespace udmrg
