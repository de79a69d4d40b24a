// Kernel templates of the Chebyshev recurrence step (see kpmgb_recurrence.cu
// for the overview).  Instantiated per precision in kpmgb_step_f64.cu and
// kpmgb_step_ff.cu so that the two families compile in parallel.
#pragma once

#include <cuda_runtime.h>

#include "kpmgb_ffmath.cuh"
#include "kpmgb_internal.h"

namespace kpmgb {
namespace step {

// Tuning knobs of the float-float kernel: operator nonzeros gathered per chunk
// (registers hold CH x CPL float4 neighbour values) and the minimum number of
// resident blocks per SM requested from the register allocator.  Real
// operators with at most two columns per lane run 3 blocks (24 warps) per SM
// with chunks of 4: measured on GB300 (3D Anderson, NR=64) 35% of HBM
// bandwidth against 29% for 2 blocks with chunks of 8; wider shapes and
// complex operators keep 2 blocks (3 would spill).
#ifndef KPMGB_FF_CHUNK_CPL1
#define KPMGB_FF_CHUNK_CPL1 8
#endif
#ifndef KPMGB_FF_CHUNK_CPL2
#define KPMGB_FF_CHUNK_CPL2 8
#endif
#ifndef KPMGB_FF_CHUNK_CPL2_REAL
#define KPMGB_FF_CHUNK_CPL2_REAL 4
#endif
#ifndef KPMGB_FF_MIN_BLOCKS
#define KPMGB_FF_MIN_BLOCKS 2
#endif
#ifndef KPMGB_FF_PREFETCH
#define KPMGB_FF_PREFETCH 0
#endif
#ifndef KPMGB_FF_SMEM_ACC
#define KPMGB_FF_SMEM_ACC 0
#endif
// evict-first (streaming) hints on the z loads and y stores of the
// float-float kernel, which are touched once per step, so that the caches
// keep the neighbour rows of the gathers (3D Anderson L=128, NR=64: 34.2% ->
// 35.2% of measured HBM bandwidth)
#ifndef KPMGB_FF_STREAM_HINTS
#define KPMGB_FF_STREAM_HINTS 1
#endif
constexpr bool kStreamHints = KPMGB_FF_STREAM_HINTS != 0;
// the same for the operator's column indices and values (read once per step)
#ifndef KPMGB_FF_INDEX_STREAM
#define KPMGB_FF_INDEX_STREAM 0
#endif
constexpr bool kIndexStream = KPMGB_FF_INDEX_STREAM != 0;
#ifndef KPMGB_FF_MIN_BLOCKS_NARROW_REAL
#define KPMGB_FF_MIN_BLOCKS_NARROW_REAL 3
#endif
// complex operators with one column per lane (NR <= 32): 3 blocks/SM with
// chunks of 4 (Haldane 256x256 cells, NR=16, NC=512: kpm_2d 244 -> 211 ms)
#ifndef KPMGB_FF_MIN_BLOCKS_CPL1_COMPLEX
#define KPMGB_FF_MIN_BLOCKS_CPL1_COMPLEX 3
#endif
#ifndef KPMGB_FF_CHUNK_CPL1_COMPLEX
#define KPMGB_FF_CHUNK_CPL1_COMPLEX 4
#endif

template <int CPL, bool REALH>
struct FFTune {
  static constexpr bool narrow_real = REALH && CPL <= 2;
  static constexpr int min_blocks =
      narrow_real ? KPMGB_FF_MIN_BLOCKS_NARROW_REAL
                  : (CPL == 1 ? KPMGB_FF_MIN_BLOCKS_CPL1_COMPLEX : KPMGB_FF_MIN_BLOCKS);
  static constexpr int chunk =
      CPL >= 3 ? 4
               : (CPL == 2 ? (REALH ? KPMGB_FF_CHUNK_CPL2_REAL : KPMGB_FF_CHUNK_CPL2)
                           : (REALH ? KPMGB_FF_CHUNK_CPL1 : KPMGB_FF_CHUNK_CPL1_COMPLEX));
  // a row's last chunk with its exact length: measured on GB300 a gain for
  // complex operators (Haldane, 10 nonzeros: chunks 8 + 2 instead of 8 + 8,
  // kpm_2d at NC=512 352 -> 335 ms) and a loss for the real 3-block kernel (3D
  // Anderson, chunks 4 + 3: 33% -> 29% of HBM), so it applies to complex H
  static constexpr bool exact_tail = !REALH;
};

// Programmatic dependent launch: a step kernel waits for the previous kernel
// of the stream (whose outputs are its inputs) to complete and flush, and at
// once allows the next one to begin launching, so launch latency overlaps the
// tail of the running step.  Without the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCols = 128;  // columns per launch (larger NR runs in batches)

struct KParams {
  const int* rowptr;
  const int* col;
  const void* val;
  int64_t NH;
  int ld;      // row stride of the blocks (total NR)
  int c0;      // first column handled by this launch
  int ncols;   // columns handled by this launch
  int parts;   // parts of the columns (CSR kernels, consecutive blockIdx.y)
  const void* x;
  const void* z;
  void* y;
  const void* bra;
  double alpha;          // +-2^k
  double2* partials;     // [block][dots][ncols] sums of this launch (null: none)
  const int2* blk;       // rows [x, y) of each block (member steps), else null
  // fixed-width padded rows (k_step_ffe): NH x ell_w columns / values
  const int* ell_col;
  const void* ell_val;
  int ell_w;
  // alpha as a float and beta (0 or -1), set on the host so that
  // the float-float kernels execute no FP64 instruction per row
  float alpha_f;
  int beta_mode;
  // optional: the largest |high part| of y (float bits, atomicMax) for the
  // split contraction's exponent (the column-pair kernel only)
  unsigned* vmax;
};

// The columns of a block whose lanes hold W: the part blockIdx.y % parts of the
// launch's, from `off` on.
struct PartCols {
  int off, c0, n;
};
template <int W>
__device__ __forceinline__ PartCols part_columns(const KParams& p) {
  if constexpr (W == 12) return {0, p.c0, p.ncols};  // {4, 3}: never in parts
  const int off = (int)(blockIdx.y % (unsigned)p.parts) * W;
  return {off, p.c0 + off, min(W, p.ncols - off)};
}

// One launch applies up to kMaxBatch independent steps without dots (the
// chains and the current applications of kpm_2d): step blockIdx.y of the
// batch.  Steps with dots launch alone.
constexpr int kMaxBatch = 3;
struct KBatch {
  KParams p[kMaxBatch];
};

template <int DOT>
struct NDots {
  static constexpr int value = DOT == DOT_NONE ? 0 : (DOT == DOT_LR1 ? 1 : 2);
};

// ------------------------------------------------------------------ reduction
// Every block stores its sums of the dots at partials[block][dot][column];
// k_finish_moments (kpmgb_recurrence.cu) adds the blocks of many steps at
// once.  A step that added its blocks itself, in the block that finished
// last, spent ~20 us on that block's serial FP64 additions (two FP64
// additions per clock and SM: 304 blocks x 128 entries, or 1216 x 16) while
// the other SMs idled: NH = 13824, NR = 64 float-float 44.8 us per step.

// Butterfly over the lane offsets 16 .. LPR of V values per lane in which the
// lanes of a pair each take half of the values, so that a level costs half of
// the additions of the one before (an FP64 addition occupies an SM's FP64
// pipe for 16 clocks per warp).  Afterwards value base + i, i < count, of the
// lane's column is v[i]; add(a, b) merges.
template <int V, int LPR, int OFF = 16, bool MORE = (OFF >= LPR)>
struct Fold {  // values per lane afterwards
  static constexpr int count = Fold<(V > 1 && V % 2 == 0 ? V / 2 : V), LPR, OFF / 2>::count;
};
template <int V, int LPR, int OFF>
struct Fold<V, LPR, OFF, false> {
  static constexpr int count = V;
};

template <int V, int LPR, typename T, typename Shfl, typename Add>
__device__ __forceinline__ int lane_fold(T (&v)[V], int lane, Shfl shfl, Add add) {
  int base = 0, cnt = V;
#pragma unroll
  for (int off = 16; off >= LPR; off >>= 1) {
    if (cnt > 1 && cnt % 2 == 0) {
      const int h = cnt / 2;
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i)
        if (i < h) {
          const T keep = up ? v[i + h] : v[i];
          const T send = up ? v[i] : v[i + h];
          v[i] = add(keep, shfl(send, off));
        }
      base += up ? h : 0;
      cnt = h;
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (i < cnt) v[i] = add(v[i], shfl(v[i], off));
    }
  }
  return base;
}

// Unevaluated sums of three floats: block sums lose nothing of the 48 bits
// that each lane's float-float accumulators carry.
struct F3 {
  float s, c, d;
};
__device__ __forceinline__ F3 f3_merge(F3 a, F3 b) {
  float s, e, c, f, g;
  ff::two_sum(a.s, b.s, s, e);
  ff::two_sum(a.c, b.c, c, f);
  ff::two_sum(c, e, c, g);
  return F3{s, c, __fadd_rn(__fadd_rn(a.d, b.d), __fadd_rn(f, g))};
}
__device__ __forceinline__ double f3_join(F3 a) {
  return (double)a.s + ((double)a.c + (double)a.d);
}

// Shared memory of the two reductions below (a kernel that holds both uses
// one buffer).
template <int DOUBLES>
__device__ __forceinline__ double* red_buffer() {
  __shared__ __align__(16) double red[DOUBLES];
  return red;
}

// Block sums of FP64 dot accumulators (all warps of the block reach this
// point; warps that own no rows pass zeros), fixed order.  Lane l of a row owns
// the columns off + l, off + l + stride, ... of the launch; the first `lanes`
// lanes of a row have columns.
template <int ND, int LPR, int CPL, int NW = kWarps>
__device__ __forceinline__ void block_dots(const double2 (&d)[ND > 0 ? ND : 1][CPL],
                                           const KParams& p, int stride = LPR, int off = 0,
                                           int lanes = LPR) {
  if constexpr (ND > 0) {
    constexpr int V = ND * CPL * 2;
    double(*red)[V * LPR] = reinterpret_cast<double(*)[V * LPR]>(red_buffer<NW * V * LPR>());
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[V];
#pragma unroll
    for (int i = 0; i < V; ++i)
      v[i] = i & 1 ? d[i / (2 * CPL)][i / 2 % CPL].y : d[i / (2 * CPL)][i / 2 % CPL].x;
    const int base = lane_fold<V, LPR>(
        v, lane, [](double a, int off) { return __shfl_xor_sync(0xffffffffu, a, off); },
        [](double a, double b) { return a + b; });
    constexpr int kLeft = Fold<V, LPR>::count;
#pragma unroll
    for (int i = 0; i < kLeft; ++i)
      red[warp][(base + i) * LPR + lane % LPR] = v[i];
    __syncthreads();
    double* out = reinterpret_cast<double*>(p.partials + (size_t)blockIdx.x * ND * p.ncols);
    for (int e = threadIdx.x; e < 2 * ND * CPL * lanes; e += NW * 32) {
      const int l = (e >> 1) % lanes, kc = (e >> 1) / lanes;
      const int col = off + kc % CPL * stride + l;
      if (col >= p.ncols) continue;
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < NW; ++w) s += red[w][(2 * kc + (e & 1)) * LPR + l];
      out[2 * (kc / CPL * p.ncols + col) + (e & 1)] = s;
    }
  }
}

// The same for float-float accumulators (leading S, correction C; NP = 1: real
// parts only) that hold at most kFlushRows rows per lane: merged over lanes
// and warps on the FP32 pipe and joined into FP64 once per entry of the block
// (two conversions and an addition per lane and value otherwise, 48 clocks of
// the SM's FP64 pipe per warp and value).
template <int ND, int LPR, int CPL, int NP, int NW = kWarps>
__device__ __forceinline__ void block_dots_ff(const F3 (&d)[ND > 0 ? ND : 1][CPL][NP],
                                              const KParams& p, int stride = LPR, int off = 0,
                                              int lanes = LPR) {
  if constexpr (ND > 0 && CPL > 2) {
    // wide lanes (128 columns): the sums of three floats would take 48 KiB
    double2 f[ND][CPL];
#pragma unroll
    for (int k = 0; k < ND; ++k)
#pragma unroll
      for (int c = 0; c < CPL; ++c)
        f[k][c] = make_double2(f3_join(d[k][c][0]), NP > 1 ? f3_join(d[k][c][NP - 1]) : 0.0);
    block_dots<ND, LPR, CPL, NW>(f, p, stride, off, lanes);
  } else if constexpr (ND > 0) {
    constexpr int V = ND * CPL * NP;
    constexpr int kDoubles = NW * ND * CPL * 2 * LPR;  // block_dots' buffer
    F3(*red)[V * LPR] = reinterpret_cast<F3(*)[V * LPR]>(
        red_buffer<(NP > 1 ? (kDoubles * 3 + 1) / 2 : kDoubles)>());
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    F3 v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = d[i / (NP * CPL)][i / NP % CPL][i % NP];
    const int base = lane_fold<V, LPR>(
        v, lane,
        [](F3 a, int off) {
          return F3{__shfl_xor_sync(0xffffffffu, a.s, off),
                    __shfl_xor_sync(0xffffffffu, a.c, off),
                    __shfl_xor_sync(0xffffffffu, a.d, off)};
        },
        [](F3 a, F3 b) { return f3_merge(a, b); });
    constexpr int kLeft = Fold<V, LPR>::count;
#pragma unroll
    for (int i = 0; i < kLeft; ++i)
      red[warp][(base + i) * LPR + lane % LPR] = v[i];
    __syncthreads();
    double2* out = p.partials + (size_t)blockIdx.x * ND * p.ncols;
    for (int e = threadIdx.x; e < ND * CPL * lanes; e += NW * 32) {
      const int l = e % lanes, kc = e / lanes;
      const int col = off + kc % CPL * stride + l;
      if (col >= p.ncols) continue;
      double r[2] = {0.0, 0.0};
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const int at = (kc * NP + q) * LPR + l;
        F3 s = red[0][at];
#pragma unroll
        for (int w = 1; w < NW; ++w) s = f3_merge(s, red[w][at]);
        r[q] = f3_join(s);
      }
      out[kc / CPL * p.ncols + col] = make_double2(r[0], r[1]);
    }
  }
}

// Whether any lane of the grid has folded its float-float accumulators into
// FP64 (a lane does so every kFlushRows row tiles).
__device__ __forceinline__ bool any_flush(int64_t ntiles, int flush_rows) {
  return (ntiles + gridDim.x - 1) / gridDim.x >= flush_rows;
}

// ------------------------------------------------------------------ FP64 path
template <bool REALH>
struct F64Val;
template <>
struct F64Val<true> {
  using T = double;
};
template <>
struct F64Val<false> {
  using T = double2;
};

__device__ __forceinline__ void cmac(double2& acc, double h, double2 v) {
  acc.x = fma(h, v.x, acc.x);
  acc.y = fma(h, v.y, acc.y);
}
__device__ __forceinline__ void cmac(double2& acc, double2 h, double2 v) {
  acc.x = fma(h.x, v.x, acc.x);
  acc.x = fma(-h.y, v.y, acc.x);
  acc.y = fma(h.x, v.y, acc.y);
  acc.y = fma(h.y, v.x, acc.y);
}
// acc += conj(a) * b
__device__ __forceinline__ void cdot(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}

// Resident blocks: 42 or 85 registers suffice, and more blocks than this start
// out unevenly over the SMs when a launch has few tiles (150x150, 10 columns
// 16.2 us per step at 3 blocks of {4, 3}, 20.6 at 4).
template <int LPR, int CPL, bool REALH, int DOT>
__global__ void __launch_bounds__(kThreads, CPL == 1 ? 6 : CPL < 4 ? 3 : 2) k_step_f64(const __grid_constant__ KBatch batch) {
  const KParams& p = batch.p[DOT == DOT_NONE ? blockIdx.y / (unsigned)batch.p[0].parts : 0];
  pdl_enter();
  const PartCols cols = part_columns<LPR * CPL>(p);
  constexpr int ND = NDots<DOT>::value;
  constexpr int GROUPS = kThreads / LPR;
  using HV = typename F64Val<REALH>::T;
  const int g = threadIdx.x / LPR;
  const int lg = threadIdx.x - g * LPR;
  const double2* __restrict__ x = static_cast<const double2*>(p.x);
  const double2* z = static_cast<const double2*>(p.z);
  double2* y = static_cast<double2*>(p.y);
  const double2* __restrict__ bra = static_cast<const double2*>(p.bra);
  const HV* __restrict__ val = static_cast<const HV*>(p.val);
  double2 d[ND > 0 ? ND : 1][CPL];
#pragma unroll
  for (int k = 0; k < (ND > 0 ? ND : 1); ++k)
#pragma unroll
    for (int c = 0; c < CPL; ++c) d[k][c] = make_double2(0.0, 0.0);

  const int64_t ntiles = (p.NH + GROUPS - 1) / GROUPS;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t r = t * GROUPS + g;
    if (r >= p.NH) continue;
    const int k0 = __ldg(p.rowptr + r), k1 = __ldg(p.rowptr + r + 1);
    double2 acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      const int j = __ldg(p.col + k);
      const HV h = __ldg(val + k);
      const double2* xr = x + (int64_t)j * p.ld + cols.c0;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int cc = lg + c * LPR;
        if (cc < cols.n) cmac(acc[c], h, __ldg(xr + cc));
      }
    }
    const int64_t base = r * p.ld + cols.c0;
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int cc = lg + c * LPR;
      if (cc >= cols.n) continue;
      double2 yv = acc[c];
      if (p.beta_mode != 0) {  // alpha is a power of two: one rounding, as alpha acc, then - z
        const double2 zv = z[base + cc];
        yv.x = fma(p.alpha, yv.x, -zv.x);
        yv.y = fma(p.alpha, yv.y, -zv.y);
      } else if (p.alpha != 1.0) {
        yv.x *= p.alpha;
        yv.y *= p.alpha;
      }
      y[base + cc] = yv;
      if constexpr (DOT == DOT_DOUBLING) {
        const double2 xv = __ldg(x + base + cc);
        d[0][c].x = fma(xv.x, xv.x, d[0][c].x);
        d[0][c].x = fma(xv.y, xv.y, d[0][c].x);
        cdot(d[1][c], xv, yv);
      } else if constexpr (DOT == DOT_LR2) {
        const double2 bv = __ldg(bra + base + cc);
        cdot(d[0][c], bv, __ldg(x + base + cc));
        cdot(d[1][c], bv, yv);
      } else if constexpr (DOT == DOT_LR1) {
        cdot(d[0][c], __ldg(bra + base + cc), yv);
      }
    }
  }
  block_dots<ND, LPR, CPL>(d, p, LPR, cols.off);
}

// ------------------------------------------------------------ float-float path
template <bool REALH>
struct FFVal;
template <>
struct FFVal<true> {
  using T = float2;  // (hi, lo)
};
template <>
struct FFVal<false> {
  using T = float4;  // (re.hi, re.lo, im.hi, im.lo)
};

__device__ __forceinline__ float habs(float2 h) { return fabsf(h.x); }
__device__ __forceinline__ float habs(float4 h) { return fabsf(h.x) + fabsf(h.z); }
__device__ __forceinline__ void hzero(float2& h) { h = make_float2(0.f, 0.f); }
__device__ __forceinline__ void hzero(float4& h) { h = make_float4(0.f, 0.f, 0.f, 0.f); }

__device__ __forceinline__ void ffmac(float& Ar, float& Cr, float& Ai, float& Ci, float2 h,
                                      float4 v) {
  ff::amac(Ar, Cr, h.x, h.y, v.x, v.y);
  ff::amac(Ai, Ci, h.x, h.y, v.z, v.w);
}
__device__ __forceinline__ void ffmac(float& Ar, float& Cr, float& Ai, float& Ci, float4 h,
                                      float4 v) {
  ff::amac(Ar, Cr, h.x, h.y, v.x, v.y);
  ff::amac(Ar, Cr, -h.z, -h.w, v.z, v.w);
  ff::amac(Ai, Ci, h.x, h.y, v.z, v.w);
  ff::amac(Ai, Ci, h.z, h.w, v.x, v.y);
}

// y = alpha * (S + C) - z (beta_mode -1) or without z (0) for one real
// component, normalised.
__device__ __forceinline__ float2 ff_epilogue(float S, float C, float alpha, int beta_mode,
                                              float zh, float zl) {
  const float u = __fmul_rn(alpha, S);  // alpha is a power of two: exact
  const float c = __fmul_rn(alpha, C);
  float h, l;
  if (beta_mode == 0) {
    ff::renorm(u, c, h, l);
  } else {
    float s, e;
    ff::two_sum(u, -zh, s, e);
    ff::renorm(s, __fadd_rn(e, __fsub_rn(c, zl)), h, l);
  }
  return make_float2(h, l);
}

// conj(a) * b accumulated into compensated float accumulators (S, C) for the
// real (index 0) and imaginary (index 1) parts.
__device__ __forceinline__ void ffdot(float (&S)[2], float (&C)[2], float4 a, float4 b) {
  ff::dacc(S[0], C[0], a.x, a.y, b.x, b.y);
  ff::dacc(S[0], C[0], a.z, a.w, b.z, b.w);
  ff::dacc(S[1], C[1], a.x, a.y, b.z, b.w);
  ff::dacc(S[1], C[1], -a.z, -a.w, b.x, b.y);
}
__device__ __forceinline__ void ffnorm2(float (&S)[2], float (&C)[2], float4 a) {
  ff::dacc(S[0], C[0], a.x, a.y, a.x, a.y);
  ff::dacc(S[0], C[0], a.z, a.w, a.z, a.w);
}

#ifndef KPMGB_FF_FLUSH_ROWS
#define KPMGB_FF_FLUSH_ROWS 64
#endif
// per-lane float-float dot accumulators fold into FP64 every this many rows
// (measured on GB300 with the padded-row kernel, 3D Anderson L=128: 64 rows
// 42.8% of the HBM roofline against 42.0% with 16, whose FP64 conversions
// kept the FP64 pipe 39% busy)
constexpr int kFlushRows = KPMGB_FF_FLUSH_ROWS;

#ifndef KPMGB_FF_EXACT_TAIL
#define KPMGB_FF_EXACT_TAIL 1
#endif

// One chunk of exactly N nonzeros of a row for the CPL columns of this lane:
// gathers, the chunk anchor (|partial sums| <= R*M, accumulator started at
// 1.5 * 2^E with 2^E = 4P, P <= R*M (1 + tiny) < 2P, so every partial sum
// stays inside one binade), anchored products, and the TwoSum merge into the
// row sums.  A row's last chunk runs with its exact length (no padded slots).
template <int N, int LPR, int CPL, bool REALH>
__device__ __forceinline__ void ff_chunk(const KParams& p,
                                         const typename FFVal<REALH>::T* __restrict__ val,
                                         const float4* __restrict__ x, int kc, int lg, bool first,
                                         float (&Sr)[CPL], float (&Cr)[CPL], float (&Si)[CPL],
                                         float (&Ci)[CPL]) {
  using HV = typename FFVal<REALH>::T;
  const PartCols cols = part_columns<LPR * CPL>(p);
  int jj[N];
  HV hv[N];
  float R = 0.f;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    jj[u] = __ldg(p.col + kc + u);
    hv[u] = __ldg(val + kc + u);
    R = __fadd_rn(R, habs(hv[u]));
  }
  float4 xv[CPL][N];
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const int cc = lg + c * LPR;
#pragma unroll
    for (int u = 0; u < N; ++u)
      xv[c][u] = cc < cols.n ? __ldg(x + (int64_t)jj[u] * p.ld + cols.c0 + cc)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    float M = 0.f;
#pragma unroll
    for (int u = 0; u < N; ++u) M = fmaxf(M, fmaxf(fabsf(xv[c][u].x), fabsf(xv[c][u].z)));
    const float B = __fmul_rn(__fmul_rn(R, M), 1.0f + 0x1p-14f);
    const float sig = __fmul_rn(6.0f, ff::pow2_floor(B));
    float Ar = sig, Ai = sig, cr = 0.f, ci = 0.f;
#pragma unroll
    for (int u = 0; u < N; ++u) ffmac(Ar, cr, Ai, ci, hv[u], xv[c][u]);
    const float sr = __fsub_rn(Ar, sig), si = __fsub_rn(Ai, sig);
    if (first) {
      Sr[c] = sr;
      Cr[c] = cr;
      Si[c] = si;
      Ci[c] = ci;
    } else {
      float s, e;
      ff::two_sum(Sr[c], sr, s, e);
      Sr[c] = s;
      Cr[c] = __fadd_rn(Cr[c], __fadd_rn(cr, e));
      ff::two_sum(Si[c], si, s, e);
      Si[c] = s;
      Ci[c] = __fadd_rn(Ci[c], __fadd_rn(ci, e));
    }
  }
}

// ff_chunk with a run-time length 1..N (uniform within a lane group).
template <int N, int LPR, int CPL, bool REALH>
__device__ __forceinline__ void ff_chunk_n(int cnt, const KParams& p,
                                           const typename FFVal<REALH>::T* __restrict__ val,
                                           const float4* __restrict__ x, int kc, int lg,
                                           bool first, float (&Sr)[CPL], float (&Cr)[CPL],
                                           float (&Si)[CPL], float (&Ci)[CPL]) {
  if constexpr (N >= 1) {
    if (cnt == N)
      ff_chunk<N, LPR, CPL, REALH>(p, val, x, kc, lg, first, Sr, Cr, Si, Ci);
    else
      ff_chunk_n<N - 1, LPR, CPL, REALH>(cnt, p, val, x, kc, lg, first, Sr, Cr, Si, Ci);
  }
}

template <int LPR, int CPL, bool REALH, int DOT, int CH>
__global__ void __launch_bounds__(kThreads, (FFTune<CPL, REALH>::min_blocks +
                                            (DOT == DOT_NONE && CPL == 1 && !REALH))) k_step_ff(
    const __grid_constant__ KBatch batch) {
  // three and four columns per lane launch alone: parameters of a step known
  // at run time only cost them registers (square 360x360, 12 columns, kpm_2d
  // 9.6 ms against 10.5)
  const KParams& p =
      batch.p[DOT == DOT_NONE && CPL < 3 ? blockIdx.y / (unsigned)batch.p[0].parts : 0];
  pdl_enter();
  const PartCols cols = part_columns<LPR * CPL>(p);
  constexpr int ND = NDots<DOT>::value;
  constexpr int NDA = ND > 0 ? ND : 1;
  constexpr int GROUPS = kThreads / LPR;
  using HV = typename FFVal<REALH>::T;
  const int g = threadIdx.x / LPR;
  const int lg = threadIdx.x - g * LPR;
  const float4* __restrict__ x = static_cast<const float4*>(p.x);
  const float4* z = static_cast<const float4*>(p.z);
  float4* y = static_cast<float4*>(p.y);
  const float4* __restrict__ bra = static_cast<const float4*>(p.bra);
  const HV* __restrict__ val = static_cast<const HV*>(p.val);
  const float alpha = p.alpha_f;
  const int beta_mode = p.beta_mode;

  // FP64 dot accumulators: in registers, or (KPMGB_FF_SMEM_ACC, up to two
  // columns per lane) in a thread-private shared-memory slot, which frees
  // 16 registers in the row loop
  constexpr bool kSmemAcc = KPMGB_FF_SMEM_ACC && ND > 0 && CPL <= 2;
  __shared__ double2 sacc[kSmemAcc ? kThreads : 1][NDA * CPL];
  double2 d[NDA][CPL];
  float dS[NDA][CPL][2], dC[NDA][CPL][2];
#pragma unroll
  for (int k = 0; k < NDA; ++k)
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      d[k][c] = make_double2(0.0, 0.0);
      if constexpr (kSmemAcc) sacc[threadIdx.x][k * CPL + c] = make_double2(0.0, 0.0);
      dS[k][c][0] = dS[k][c][1] = dC[k][c][0] = dC[k][c][1] = 0.f;
    }
  int rows_since_flush = 0;

  const int64_t ntiles = (p.NH + GROUPS - 1) / GROUPS;
#if KPMGB_FF_PREFETCH
  // row bounds of the next row of this lane group are loaded one row ahead,
  // taking the row-pointer load off the dependent chain of every row
  int nk0 = 0, nk1 = 0;
  {
    const int64_t r0 = (int64_t)blockIdx.x * GROUPS + g;
    if (blockIdx.x < ntiles && r0 < p.NH) {
      nk0 = __ldg(p.rowptr + r0);
      nk1 = __ldg(p.rowptr + r0 + 1);
    }
  }
#endif
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t r = t * GROUPS + g;
#if KPMGB_FF_PREFETCH
    const int k0 = nk0, k1 = nk1;
    {
      const int64_t rn = r + (int64_t)gridDim.x * GROUPS;
      if (t + gridDim.x < ntiles && rn < p.NH) {
        nk0 = __ldg(p.rowptr + rn);
        nk1 = __ldg(p.rowptr + rn + 1);
      }
    }
    if (r >= p.NH) continue;
#else
    if (r >= p.NH) continue;
    const int k0 = __ldg(p.rowptr + r), k1 = __ldg(p.rowptr + r + 1);
#endif
    float Sr[CPL], Cr[CPL], Si[CPL], Ci[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) Sr[c] = Cr[c] = Si[c] = Ci[c] = 0.f;
    if constexpr (KPMGB_FF_EXACT_TAIL && FFTune<CPL, REALH>::exact_tail) {
      for (int kc = k0; kc < k1; kc += CH) {
        const int cnt = min(CH, k1 - kc);
        ff_chunk_n<CH, LPR, CPL, REALH>(cnt, p, val, x, kc, lg, kc == k0, Sr, Cr, Si, Ci);
      }
    } else {
      for (int kc = k0; kc < k1; kc += CH) {
        const int cnt = min(CH, k1 - kc);
        int jj[CH];
        HV hv[CH];
        float R = 0.f;
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          if (u < cnt) {
            if constexpr (kIndexStream) {
              jj[u] = __ldcs(p.col + kc + u);
              hv[u] = __ldcs(val + kc + u);
            } else {
              jj[u] = __ldg(p.col + kc + u);
              hv[u] = __ldg(val + kc + u);
            }
          } else {
            jj[u] = 0;
            hzero(hv[u]);
          }
          R = __fadd_rn(R, habs(hv[u]));
        }
        float4 xv[CPL][CH];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          const int cc = lg + c * LPR;
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            if (u < cnt && cc < cols.n)
              xv[c][u] = __ldg(x + (int64_t)jj[u] * p.ld + cols.c0 + cc);
            else
              xv[c][u] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          float M = 0.f;
#pragma unroll
          for (int u = 0; u < CH; ++u) M = fmaxf(M, fmaxf(fabsf(xv[c][u].x), fabsf(xv[c][u].z)));
          // |partial sums| <= R*M (1 + tiny); anchor at 1.5 * 2^E with 2^E = 4P,
          // P <= bound < 2P, so every partial sum stays inside the binade.
          const float B = __fmul_rn(__fmul_rn(R, M), 1.0f + 0x1p-14f);
          const float sig = __fmul_rn(6.0f, ff::pow2_floor(B));
          float Ar = sig, Ai = sig, cr = 0.f, ci = 0.f;
#pragma unroll
          for (int u = 0; u < CH; ++u)
            if (u < cnt) ffmac(Ar, cr, Ai, ci, hv[u], xv[c][u]);
          const float sr = __fsub_rn(Ar, sig), si = __fsub_rn(Ai, sig);
          if (kc == k0) {
            Sr[c] = sr;
            Cr[c] = cr;
            Si[c] = si;
            Ci[c] = ci;
          } else {
            float s, e;
            ff::two_sum(Sr[c], sr, s, e);
            Sr[c] = s;
            Cr[c] = __fadd_rn(Cr[c], __fadd_rn(cr, e));
            ff::two_sum(Si[c], si, s, e);
            Si[c] = s;
            Ci[c] = __fadd_rn(Ci[c], __fadd_rn(ci, e));
          }
        }
      }
    }
    const int64_t base = r * p.ld + cols.c0;
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int cc = lg + c * LPR;
      if (cc >= cols.n) continue;
      float4 zv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (beta_mode != 0) zv = kStreamHints ? __ldcs(z + base + cc) : z[base + cc];
      const float2 yr = ff_epilogue(Sr[c], Cr[c], alpha, beta_mode, zv.x, zv.y);
      const float2 yi = ff_epilogue(Si[c], Ci[c], alpha, beta_mode, zv.z, zv.w);
      const float4 yv = make_float4(yr.x, yr.y, yi.x, yi.y);
      if constexpr (kStreamHints) __stcs(y + base + cc, yv); else y[base + cc] = yv;
      if constexpr (DOT == DOT_DOUBLING) {
        const float4 xr = __ldg(x + base + cc);
        ffnorm2(dS[0][c], dC[0][c], xr);
        ffdot(dS[1][c], dC[1][c], xr, yv);
      } else if constexpr (DOT == DOT_LR2) {
        const float4 bv = __ldg(bra + base + cc);
        ffdot(dS[0][c], dC[0][c], bv, __ldg(x + base + cc));
        ffdot(dS[1][c], dC[1][c], bv, yv);
      } else if constexpr (DOT == DOT_LR1) {
        ffdot(dS[0][c], dC[0][c], __ldg(bra + base + cc), yv);
      }
    }
    if constexpr (ND > 0) {
      if (++rows_since_flush == kFlushRows) {
        rows_since_flush = 0;
#pragma unroll
        for (int k = 0; k < ND; ++k)
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            if constexpr (kSmemAcc) {
              double2 v = sacc[threadIdx.x][k * CPL + c];
              v.x += ff::join(dS[k][c][0], dC[k][c][0]);
              v.y += ff::join(dS[k][c][1], dC[k][c][1]);
              sacc[threadIdx.x][k * CPL + c] = v;
            } else {
              d[k][c].x += ff::join(dS[k][c][0], dC[k][c][0]);
              d[k][c].y += ff::join(dS[k][c][1], dC[k][c][1]);
            }
            dS[k][c][0] = dS[k][c][1] = dC[k][c][0] = dC[k][c][1] = 0.f;
          }
      }
    }
  }
  if constexpr (ND > 0) {
    if (any_flush(ntiles, kFlushRows)) {
#pragma unroll
      for (int k = 0; k < ND; ++k)
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          if constexpr (kSmemAcc) d[k][c] = sacc[threadIdx.x][k * CPL + c];
          d[k][c].x += ff::join(dS[k][c][0], dC[k][c][0]);
          d[k][c].y += ff::join(dS[k][c][1], dC[k][c][1]);
        }
      block_dots<ND, LPR, CPL>(d, p, LPR, cols.off);
    } else {
      F3 f[NDA][CPL][2];
#pragma unroll
      for (int k = 0; k < ND; ++k)
#pragma unroll
        for (int c = 0; c < CPL; ++c)
#pragma unroll
          for (int q = 0; q < 2; ++q) f[k][c][q] = F3{dS[k][c][q], dC[k][c][q], 0.f};
      block_dots_ff<ND, LPR, CPL, 2>(f, p, LPR, cols.off);
    }
  }
}

struct Shape {
  int lpr, cpl;
};

using KernelFn = void (*)(KBatch);

template <int LPR, int CPL, bool REALH, int DOT, int PREC>
KernelFn kernel_for_prec() {
  if constexpr (PREC == KPMGB_PREC_FF) {
    return k_step_ff<LPR, CPL, REALH, DOT, FFTune<CPL, REALH>::chunk>;
  } else {
    return k_step_f64<LPR, CPL, REALH, DOT>;
  }
}

template <int LPR, int CPL, bool REALH, int PREC>
KernelFn kernel_dot(int dot) {
  switch (dot) {
    case DOT_DOUBLING: return kernel_for_prec<LPR, CPL, REALH, DOT_DOUBLING, PREC>();
    case DOT_LR2: return kernel_for_prec<LPR, CPL, REALH, DOT_LR2, PREC>();
    case DOT_LR1: return kernel_for_prec<LPR, CPL, REALH, DOT_LR1, PREC>();
    default: return kernel_for_prec<LPR, CPL, REALH, DOT_NONE, PREC>();
  }
}

template <int LPR, int CPL, int PREC>
KernelFn kernel_real(int dot, bool real) {
  return real ? kernel_dot<LPR, CPL, true, PREC>(dot) : kernel_dot<LPR, CPL, false, PREC>(dot);
}

template <int PREC>
KernelFn select_kernel_impl(Shape s, int dot, bool real) {
  switch (s.lpr * 10 + s.cpl) {
    case 11: return kernel_real<1, 1, PREC>(dot, real);
    case 21: return kernel_real<2, 1, PREC>(dot, real);
    case 41: return kernel_real<4, 1, PREC>(dot, real);
    case 81: return kernel_real<8, 1, PREC>(dot, real);
    case 43: return kernel_real<4, 3, PREC>(dot, real);
    case 161: return kernel_real<16, 1, PREC>(dot, real);
    case 321: return kernel_real<32, 1, PREC>(dot, real);
    case 322: return kernel_real<32, 2, PREC>(dot, real);
    default: return kernel_real<32, 4, PREC>(dot, real);
  }
}

KernelFn select_kernel_f64(Shape s, int dot, bool real);
KernelFn select_kernel_ff(Shape s, int dot, bool real);
// Float-float kernel over fixed-width padded rows (kpmgb_step_ffe.cu): 5..64
// columns; nullptr otherwise.  ffe_lanes: lanes per row of its shape.
KernelFn select_kernel_ffe(int ncols, int dot, bool real);
int ffe_lanes(int ncols);
// Row-streaming float-float kernel for real operators over padded rows of
// stride 8 (kpmgb_step_ffe.cu): 33..64 columns (32 lanes x 2 per row), rows of
// at most 8 nonzeros; nullptr otherwise.  Rows per block tile: 8.
KernelFn select_kernel_ffr(int ncols, int dot, bool real, int max_row_nnz, int ell_w);
// Row-streaming float-float kernel for complex operators over padded rows of
// stride 8 or 12 (kpmgb_step_ffe.cu): 9..32 columns, one column per lane;
// nullptr otherwise.  ffc_lanes: lanes per row (16 or 32).
KernelFn select_kernel_ffc(int ncols, int dot, bool real, int ell_w, int max_row_nnz);
int ffc_lanes(int ncols);
// Row-streaming float-float kernels on packed FP32 pairs (kpmgb_step_ffpk.cu):
// real operators, 2..128 columns, steps with dots, rows of 5..8 nonzeros,
// vectors in the paired element layout (re.hi, im.hi, re.lo, im.lo).  The
// kernel to launch for such a call of NH rows (fn = nullptr when none
// applies): threads per block, rows per block tile and the parts of the columns
// (gridDim.y).
struct PackedStep {
  KernelFn fn = nullptr;
  int threads = 0;
  int rows_per_block = 0;
  int split = 1;
};
PackedStep select_packed_step(int ncols, int dot, bool real, int max_row_nnz, int ell_w,
                              int64_t NH);
// The same over blocks of given rows (KParams::blk), 2..32 columns.
PackedStep select_packed_members(int ncols, bool real, int max_row_nnz, int ell_w, int64_t NH);
// Complex operators on column pairs (kpmgb_step_ffcp.cu) over padded rows of
// stride 8 or 12, vectors in the column-pair layout: 2..128 columns, an even
// number from 6 on in steps without dots.
PackedStep select_colpair_step(int ncols, int dot, bool real, int ell_w, int max_row_nnz,
                               int64_t NH);

}  // namespace step
}  // namespace kpmgb
