// Row-streaming float-float step on packed FP32 pairs (k_step_ffpk): real
// operators with rows of 6..8, 49..64 columns (two per lane), doubling dots;
// k_step_ffpk1 below serves the others of 2..128 columns (one per lane) and the
// bra-ket dots (2D 512x512, 16 columns 131 us per step with the CSR kernel, 60
// here; 40 columns 212 with k_step_ffr, 138).
//
// Blackwell executes `fma/add/sub/mul.rn.f32x2` on a 64-bit register pair:
// one instruction for two correctly rounded FP32 operations.  For real H the
// real and imaginary parts of a float-float complex value go through
// identical operation sequences, so this kernel runs k_step_ffr's row
// arithmetic once on the pair {re, im}: 6 packed operations per nonzero and
// column for the anchored products instead of 12, and likewise for the
// epilogue and the compensated dots.  The pairs come straight from memory:
// the call stores its recurrence vectors as (re.hi, im.hi, re.lo, im.lo) per
// element ("paired" layout, written by the load kernel), so a 16-byte load
// yields the {hi} and {lo} pairs in register pairs and no packing is needed
// except for broadcasting the operator values.  Each lane of a pair performs
// exactly the scalar sequence of k_step_ffr (A - A_new stands for
// -(A_new - A), both exact), so y is bitwise k_step_ffr's; the dots add the
// real and imaginary terms in separate accumulators and join them at the
// FP64 fold.
//
// Layout and pipeline as k_step_ffr: a warp owns a row, each lane the two
// columns lane and lane + 32; the next row's 8 column indices and values are
// staged in the warp's shared memory with cp.async; all loads of a row are
// issued before its arithmetic; 2 blocks per SM.  Bound by the latency of the
// gathers at 16 warps per SM, so registers decide how far ahead the loads are
// scheduled: the operator values are read from shared memory where they are
// used (the broadcast pairs of a row held in registers took 28 of the 128),
// and the row stride of a full launch is a constant: 3D Anderson L=128, NR=64
// 1.530 -> 1.440 ms per step (4.68 TB/s of the step's 6.74 GB).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "kpmgb_pk.cuh"
#include "kpmgb_step.cuh"

namespace kpmgb {
namespace step {

using namespace f32x2;

// A shared-memory load that stays where it is written (not hoisted into
// registers held across the row).
__device__ __forceinline__ float2 ld_shared_f2(const float2* p) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
               : "=f"(v.x), "=f"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

// The sum of the two lanes of a pair of accumulators.
__device__ __forceinline__ F3 pair_sum(f2 S, f2 C) {
  F3 a{0.f, 0.f, 0.f}, b{0.f, 0.f, 0.f};
  upk(S, a.s, b.s);
  upk(C, a.c, b.c);
  return f3_merge(a, b);
}

// The first lane less the second.
__device__ __forceinline__ F3 pair_diff(f2 S, f2 C) {
  F3 a{0.f, 0.f, 0.f}, b{0.f, 0.f, 0.f};
  upk(S, a.s, b.s);
  upk(C, a.c, b.c);
  return f3_merge(a, F3{-b.s, -b.c, 0.f});
}
__device__ __forceinline__ double diff2(f2 S, f2 C) {
  float s0, s1, c0, c1;
  upk(S, s0, s1);
  upk(C, c0, c1);
  return ((double)s0 + (double)c0) - ((double)s1 + (double)c1);
}
__device__ __forceinline__ f2 swap2(f2 v) {
  float a, b;
  upk(v, a, b);
  return pk(b, a);
}

template <int W, bool FULL>
__global__ void __launch_bounds__(kThreads, 2) k_step_ffpk(
    const __grid_constant__ KBatch batch) {
  const KParams& p = batch.p[0];
  pdl_enter();
  constexpr int GROUPS = kThreads / 32;  // rows per block tile
  constexpr int CPL = 2;
  // 49..63 columns: the second column slot of the lanes past the last column
  // is dead (no loads, stores or dots)
  bool live[CPL];
#pragma unroll
  for (int c = 0; c < CPL; ++c) live[c] = FULL || (threadIdx.x & 31) + 32 * c < p.ncols;
  constexpr int kStride = 8;  // padded row stride (ints / float2 values)
  const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ulonglong2* __restrict__ x = static_cast<const ulonglong2*>(p.x);
  const ulonglong2* z = static_cast<const ulonglong2*>(p.z);
  ulonglong2* y = static_cast<ulonglong2*>(p.y);
  const int* __restrict__ ecol = p.ell_col;
  const float2* __restrict__ eval = static_cast<const float2*>(p.ell_val);
  const f2 alpha2 = pk(p.alpha_f, p.alpha_f);
  const int beta_mode = p.beta_mode;
  const int ld = FULL ? 64 : p.ld;  // one column batch: c0 = 0

  __shared__ double sacc[2 * CPL][kThreads];  // FP64 dots of each thread
  // per warp, two buffers of one padded row: 8 column indices, 8 values
  __shared__ __align__(16) int sidx[GROUPS][2][3 * kStride];
  // dot accumulators per column: norm {sum re^2, sum im^2}, cross
  // {sum re x re y, sum im x im y}
  f2 nS[CPL], nC[CPL], xS[CPL], xC[CPL];
  const f2 zero2 = pk(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    sacc[c][threadIdx.x] = sacc[CPL + c][threadIdx.x] = 0.0;
    nS[c] = nC[c] = xS[c] = xC[c] = zero2;
  }
  int rows_since_flush = 0;

  auto stage = [&](int64_t r, int b) {
    if (lane < 6) {
      const char* src = lane < 2 ? reinterpret_cast<const char*>(ecol + r * kStride) + lane * 16
                                 : reinterpret_cast<const char*>(eval + r * kStride) + (lane - 2) * 16;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&sidx[g][b][lane * 4]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // row tiles of this block: every gridDim.x-th tile, so that the rows in
  // flight on the whole GPU lie in one window and their distant neighbours
  // (the ±L^2 planes of a 3D lattice) are still in L2 (contiguous ranges of
  // tiles per block measured 2.18 ms per step against 1.57 ms)
  const int64_t ntiles = (p.NH + GROUPS - 1) / GROUPS;
  int buf = 0;
  {
    const int64_t r0 = (int64_t)blockIdx.x * GROUPS + g;
    if ((int64_t)blockIdx.x < ntiles && r0 < p.NH) stage(r0, 0);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t r = t * GROUPS + g;
    if (r >= p.NH) continue;
    {
      const int64_t rn = r + (int64_t)gridDim.x * GROUPS;
      if (t + gridDim.x < ntiles && rn < p.NH) stage(rn, buf ^ 1);
      else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const int* jrow = &sidx[g][buf][0];
    const float4* hrow = reinterpret_cast<const float4*>(&sidx[g][buf][kStride]);
    const int64_t base = r * ld;
    // every load of the row, before any arithmetic
    ulonglong2 zv[CPL], xo[CPL], xv[CPL][W];
    const ulonglong2 zero4 = make_ulonglong2(0ull, 0ull);
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int64_t e = base + lane + 32 * c;
      zv[c] = live[c] && beta_mode != 0 ? __ldcs(z + e) : zero4;
      xo[c] = live[c] ? __ldg(x + e) : zero4;
    }
    {
      const int4 j0 = reinterpret_cast<const int4*>(jrow)[0];
      const int4 j1 = reinterpret_cast<const int4*>(jrow)[1];
      const int jj[8] = {j0.x, j0.y, j0.z, j0.w, j1.x, j1.y, j1.z, j1.w};
#pragma unroll
      for (int c = 0; c < CPL; ++c)
#pragma unroll
        for (int u = 0; u < W; ++u)
          xv[c][u] = live[c] ? __ldg(x + (int64_t)jj[u] * ld + lane + 32 * c) : zero4;
    }
    const float2* hv = reinterpret_cast<const float2*>(hrow);
    float R = 0.f;
#pragma unroll
    for (int u = 0; u < W; ++u) R = __fadd_rn(R, fabsf(hv[u].x));
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      float M = 0.f;
#pragma unroll
      for (int u = 0; u < W; ++u) {
        float re, im;
        upk(xv[c][u].x, re, im);
        M = fmaxf(M, fmaxf(fabsf(re), fabsf(im)));
      }
      // anchor 1.5 * 2^E with 2^E = 4P, P <= R*M (1 + tiny) < 2P (k_step_ffr)
      const float B = __fmul_rn(__fmul_rn(R, M), 1.0f + 0x1p-14f);
      const float sig = __fmul_rn(6.0f, ff::pow2_floor(B));
      const f2 sig2 = pk(sig, sig);
      f2 A = sig2, C = zero2;
#pragma unroll
      for (int u = 0; u < W; ++u) {
        const float2 h = ld_shared_f2(hv + u);
        amac2(A, C, pk(h.x, h.x), pk(h.y, h.y), xv[c][u].x, xv[c][u].y);
      }
      const f2 S = sub2(A, sig2);
      // y = alpha (S + C) + beta z, normalised (ff_epilogue on both lanes)
      const f2 u2 = mul2(alpha2, S);  // alpha is a power of two: exact
      const f2 c2 = mul2(alpha2, C);
      f2 yh, yl;
      if (beta_mode == 0) {
        two_sum2(u2, c2, yh, yl);
      } else {
        // beta = -1: two_sum(u, -zh) and e + (c - zl), the negations are exact
        const f2 s = sub2(u2, zv[c].x);
        const f2 bb = sub2(s, u2);
        const f2 e = sub2(sub2(u2, sub2(s, bb)), add2(zv[c].x, bb));
        two_sum2(s, add2(e, sub2(c2, zv[c].y)), yh, yl);
      }
      if (live[c]) {
        __stcs(y + base + lane + 32 * c, make_ulonglong2(yh, yl));
        const f2 nxh = sub2(zero2, xo[c].x);  // exact negation
        dacc2(nS[c], nC[c], xo[c].x, nxh, xo[c].y, xo[c].x, xo[c].y);
        dacc2(xS[c], xC[c], xo[c].x, nxh, xo[c].y, yh, yl);
      }
    }
    __syncwarp();  // the buffer is restaged two rows later
    buf ^= 1;
    if (++rows_since_flush == kFlushRows) {
      rows_since_flush = 0;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        sacc[c][threadIdx.x] += join2(nS[c], nC[c]);
        sacc[CPL + c][threadIdx.x] += join2(xS[c], xC[c]);
        nS[c] = nC[c] = xS[c] = xC[c] = zero2;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // the block's sums straight from the thread slots: one column's terms lie
  // in the same lane of every warp
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    sacc[c][threadIdx.x] += join2(nS[c], nC[c]);
    sacc[CPL + c][threadIdx.x] += join2(xS[c], xC[c]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * p.ncols; e += kThreads) {
    const int k = e / p.ncols, col = e % p.ncols;
    const double* v = &sacc[k * CPL + col / 32][col % 32];
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < GROUPS; ++w) s += v[32 * w];
    p.partials[(size_t)blockIdx.x * 2 * p.ncols + e] = make_double2(s, 0.0);
  }
}

// ---------------------------------------------------------------------------
// One column per lane (k_step_ffpk1): the packed row-streaming step for 2..128
// columns in parts of LPR, LPR lanes per row (RPW = 32 / LPR rows per warp; all
// parts of the columns in one launch), with half the loads per lane of k_step_ffpk and so three blocks per SM.  Half of the issue
// slots and the latency of the gathers bound it (57% issued with 22 warps per
// SM at NH = 262144, NR = 8), so the loop keeps to 32-bit indices, the staging
// addresses advance by constants and lanes past the last column repeat it
// instead of holding zeros: 26.1 -> 23.0 us per step (65536, 8 8.6 -> 7.6; 3D
// L = 128, NR = 16 414 -> 386).  Four blocks per SM (64 registers, rows of 5)
// pay where the slots come from HBM: 1048576, 8 95 -> 92 us, 262144, 32 90 -> 85,
// but 65536, 8 7.5 -> 8.1.  Below 9
// columns the CSR kernel, whose rows wait for their row pointers and column
// indices in turn, took 14.4 us at NH = 65536, NR = 8.
//
// MEMBERS: each block takes the consecutive rows p.blk[block] (the rows of one
// member of an ensemble) instead of every gridDim-th tile.
template <int LPR, int W, int BLOCKS, int DOT, bool MEMBERS>
__global__ void __launch_bounds__(kThreads, BLOCKS) k_step_ffpk1(
    const __grid_constant__ KBatch batch) {
  const KParams& p = batch.p[0];
  pdl_enter();
  constexpr int RPW = 32 / LPR;           // rows per warp
  constexpr int GROUPS = kThreads / LPR;  // rows per block tile
  constexpr int kStride = 8;              // padded row stride (ints / float2 values)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lg = lane % LPR, sub = lane / LPR;  // column, and row within the warp
  // the columns of blockIdx.y: LPR each, the rest in the last
  const int off = blockIdx.y * LPR, ncols = min(LPR, p.ncols - off);
  const bool live = lg < ncols;
  // tiles t0, t0 + dt, .. of rows origin + t GROUPS .. up to NH (below 2^31)
  const int2 rows = MEMBERS ? __ldg(p.blk + blockIdx.x) : make_int2(0, (int)p.NH);
  const unsigned origin = (unsigned)rows.x, NH = (unsigned)rows.y;
  const unsigned t0 = MEMBERS ? 0 : blockIdx.x, dt = MEMBERS ? 1 : gridDim.x;
  const unsigned row_bytes = p.ld * 16;
  // this lane's column (lanes past the last one repeat it and store nothing)
  const int64_t col_bytes = (p.c0 + off + (live ? lg : ncols - 1)) * 16;
  const char* const xl = static_cast<const char*>(p.x) + col_bytes;
  const char* const zl = static_cast<const char*>(p.z) + col_bytes;
  char* const yl = static_cast<char*>(p.y) + col_bytes;
  const char* const bl = DOT == DOT_DOUBLING ? nullptr : static_cast<const char*>(p.bra) + col_bytes;
  const f2 alpha2 = pk(p.alpha_f, p.alpha_f);
  const int beta_mode = p.beta_mode;
  const f2 zero2 = pk(0.f, 0.f);
  constexpr int ND = NDots<DOT>::value;
  constexpr int NV = DOT == DOT_DOUBLING ? 2 : 2 * ND;
  __shared__ double2 sacc[kThreads][ND];
  // per warp, two buffers of RPW padded rows: 8 column indices, 8 values
  __shared__ __align__(16) int sidx[kThreads / 32][2][RPW][3 * kStride];
  // DOUBLING: <x|x>, Re<x|y>; LR: of <b|x> (LR2) and <b|y> the products
  // {re re, im im} and {re im, im re}
  f2 dS[NV], dC[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) dS[v] = dC[v] = zero2;
#pragma unroll
  for (int n = 0; n < ND; ++n) sacc[threadIdx.x][n] = make_double2(0.0, 0.0);
  auto fold = [&](double2 (&d)[ND][1]) {
#pragma unroll
    for (int n = 0; n < ND; ++n) {
      d[n][0] = sacc[threadIdx.x][n];
      if constexpr (DOT == DOT_DOUBLING) {
        d[n][0].x += join2(dS[n], dC[n]);
      } else {
        d[n][0].x += join2(dS[2 * n], dC[2 * n]);
        d[n][0].y += diff2(dS[2 * n + 1], dC[2 * n + 1]);
      }
    }
  };
  int rows_since_flush = 0;
  const unsigned ntiles = (NH - origin + GROUPS - 1) / GROUPS;
  // the warp's lanes copy the RPW rows of a tile: 6 pieces of 16 bytes each, at
  // most kPer of them per lane, whose places in the tile stay the same
  constexpr int kPer = (RPW * 6 + 31) / 32;
  const char* src[kPer];
  int step_bytes[kPer];
  unsigned first_row[kPer], dst[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int q = lane + 32 * i;
    const int rr = q / 6, piece = q % 6;
    const bool idx = piece < 2;
    first_row[i] = origin + warp * RPW + rr;
    const int64_t r = origin + (int64_t)t0 * GROUPS + warp * RPW + rr;
    src[i] = idx ? reinterpret_cast<const char*>(p.ell_col) + r * (kStride * 4) + piece * 16
                 : static_cast<const char*>(p.ell_val) + r * (kStride * 8) + (piece - 2) * 16;
    step_bytes[i] = (int)dt * GROUPS * kStride * (idx ? 4 : 8);
    dst[i] = (unsigned)__cvta_generic_to_shared(&sidx[warp][0][rr < RPW ? rr : 0][piece * 4]);
  }
  auto stage = [&](unsigned t, int b) {  // called for the tiles of this block in order
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (lane + 32 * i < RPW * 6 && t * GROUPS + first_row[i] < NH)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         dst[i] + b * (unsigned)sizeof(sidx[0][0])),
                     "l"(src[i])
                     : "memory");
      src[i] += step_bytes[i];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int buf = 0;
  stage(t0, 0);
  for (unsigned t = t0; t < ntiles; t += dt) {
    if (t + dt < ntiles) stage(t + dt, buf ^ 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const unsigned row = origin + t * GROUPS + warp * RPW + sub;
    const bool ok = row < NH && live;
    const int* jrow = &sidx[warp][buf][sub][0];
    const float4* hrow = reinterpret_cast<const float4*>(&sidx[warp][buf][sub][kStride]);
    const uint64_t e = (uint64_t)row * row_bytes;
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
    ulonglong2 zv = zero, xo = zero, bv = zero, xv[W];
    if (row < NH) {
      if (beta_mode != 0) zv = __ldcs(reinterpret_cast<const ulonglong2*>(zl + e));
      if constexpr (DOT != DOT_LR1) xo = __ldg(reinterpret_cast<const ulonglong2*>(xl + e));
      if constexpr (DOT != DOT_DOUBLING) bv = __ldg(reinterpret_cast<const ulonglong2*>(bl + e));
#pragma unroll
      for (int u = 0; u < W; ++u)
        xv[u] = __ldg(reinterpret_cast<const ulonglong2*>(xl + (uint64_t)(unsigned)jrow[u] * row_bytes));
    } else {
#pragma unroll
      for (int u = 0; u < W; ++u) xv[u] = zero;
    }
    float hh[8], hl[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = hrow[q];
      hh[2 * q] = v.x;
      hl[2 * q] = v.y;
      hh[2 * q + 1] = v.z;
      hl[2 * q + 1] = v.w;
    }
    __syncwarp();  // the buffer is restaged two tiles later
    buf ^= 1;
    float R = 0.f, M = 0.f;
#pragma unroll
    for (int u = 0; u < W; ++u) {
      R = __fadd_rn(R, fabsf(hh[u]));
      float re, im;
      upk(xv[u].x, re, im);
      M = fmaxf(M, fmaxf(fabsf(re), fabsf(im)));
    }
    const float sig = __fmul_rn(6.0f, ff::pow2_floor(__fmul_rn(__fmul_rn(R, M), 1.0f + 0x1p-14f)));
    const f2 sig2 = pk(sig, sig);
    f2 A = sig2, C = zero2;
#pragma unroll
    for (int u = 0; u < W; ++u) amac2(A, C, pk(hh[u], hh[u]), pk(hl[u], hl[u]), xv[u].x, xv[u].y);
    if (ok) {
      const f2 S = sub2(A, sig2);
      const f2 u2 = mul2(alpha2, S);
      const f2 c2 = mul2(alpha2, C);
      f2 yh, yl2;
      if (beta_mode == 0) {
        two_sum2(u2, c2, yh, yl2);
      } else {
        const f2 s2 = sub2(u2, zv.x);
        const f2 bb = sub2(s2, u2);
        const f2 e2 = sub2(sub2(u2, sub2(s2, bb)), add2(zv.x, bb));
        two_sum2(s2, add2(e2, sub2(c2, zv.y)), yh, yl2);
      }
      __stcs(reinterpret_cast<ulonglong2*>(yl + e), make_ulonglong2(yh, yl2));
      if constexpr (DOT == DOT_DOUBLING) {
        const f2 nxh = sub2(zero2, xo.x);
        dacc2(dS[0], dC[0], xo.x, nxh, xo.y, xo.x, xo.y);
        dacc2(dS[1], dC[1], xo.x, nxh, xo.y, yh, yl2);
      } else {
        const f2 nbh = sub2(zero2, bv.x);
        auto dot = [&](int v, f2 h, f2 l) {
          dacc2(dS[v], dC[v], bv.x, nbh, bv.y, h, l);
          dacc2(dS[v + 1], dC[v + 1], bv.x, nbh, bv.y, swap2(h), swap2(l));
        };
        if constexpr (DOT == DOT_LR2) dot(0, xo.x, xo.y);
        dot(NV - 2, yh, yl2);
      }
    }
    if (++rows_since_flush == kFlushRows) {
      rows_since_flush = 0;
      double2 d[ND][1];
      fold(d);
#pragma unroll
      for (int n = 0; n < ND; ++n) sacc[threadIdx.x][n] = d[n][0];
#pragma unroll
      for (int v = 0; v < NV; ++v) dS[v] = dC[v] = zero2;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (MEMBERS ? ntiles >= kFlushRows : any_flush(ntiles, kFlushRows)) {
    double2 d[ND][1];
    fold(d);
    block_dots<ND, LPR, 1>(d, p, LPR, off);
  } else if constexpr (DOT == DOT_DOUBLING) {
    const F3 f[2][1][1] = {{{pair_sum(dS[0], dC[0])}}, {{pair_sum(dS[1], dC[1])}}};
    block_dots_ff<2, LPR, 1, 1>(f, p, LPR, off);
  } else {
    F3 f[ND][1][2];
#pragma unroll
    for (int n = 0; n < ND; ++n) {
      f[n][0][0] = pair_sum(dS[2 * n], dC[2 * n]);
      f[n][0][1] = pair_diff(dS[2 * n + 1], dC[2 * n + 1]);
    }
    block_dots_ff<ND, LPR, 1, 2>(f, p, LPR, off);
  }
}

namespace {
template <int LPR, int DOT, bool MEMBERS>
KernelFn ffpk1_w(int max_row_nnz, bool from_hbm) {
  switch (max_row_nnz) {
    case 5:
      return from_hbm ? k_step_ffpk1<LPR, 5, 4, DOT, MEMBERS> : k_step_ffpk1<LPR, 5, 3, DOT, MEMBERS>;
    case 6: return k_step_ffpk1<LPR, 6, 3, DOT, MEMBERS>;
    case 7: return k_step_ffpk1<LPR, 7, 3, DOT, MEMBERS>;
    case 8: return k_step_ffpk1<LPR, 8, 3, DOT, MEMBERS>;
    default: return nullptr;
  }
}

// both slots within about 100 MB stay in L2 from step to step
bool slots_from_hbm(int64_t NH, int ncols) { return NH * ncols * 32 > (int64_t)100 << 20; }

template <int DOT, bool MEMBERS>
KernelFn ffpk1_lanes(int lanes, int max_row_nnz, bool from_hbm) {
  switch (lanes) {
    case 2: return ffpk1_w<2, DOT, MEMBERS>(max_row_nnz, from_hbm);
    case 4: return ffpk1_w<4, DOT, MEMBERS>(max_row_nnz, from_hbm);
    case 8: return ffpk1_w<8, DOT, MEMBERS>(max_row_nnz, from_hbm);
    case 16: return ffpk1_w<16, DOT, MEMBERS>(max_row_nnz, from_hbm);
    default: return ffpk1_w<32, DOT, MEMBERS>(max_row_nnz, from_hbm);
  }
}

int ffpk1_cols(int ncols, int lanes) { return (ncols + lanes - 1) / lanes * lanes; }

// Lanes per row of k_step_ffpk1 (the columns run in parts of that many, one
// per gridDim.y): 32, or 16 or 8 where that saves over an eighth of the lanes.
// Idle lanes cost as much as live ones, narrow parts little: 2D L = 1024, 40
// columns 8 x 5 lanes 509 us per step, 32 x 2 670; 24 columns 8 x 3 306, 32 363;
// 48 columns 16 x 3 586, 32 x 2 677; but 50 columns 8 x 7 746, 32 x 2 701.  Parts
// of 4 read half lines of 64 bytes and gain nothing (12 columns 229, 16 lanes 217).
int ffpk1_lanes_for(int ncols) {
  if (ncols <= 8) return ncols <= 2 ? 2 : ncols <= 4 ? 4 : 8;
  int best = 32;
  for (int lanes : {16, 8})
    if (ffpk1_cols(ncols, lanes) * 8 < ffpk1_cols(ncols, best) * 7) best = lanes;
  return best;
}

template <int W>
KernelFn ffpk_w(bool full) {
  return full ? k_step_ffpk<W, true> : k_step_ffpk<W, false>;
}
}  // namespace

PackedStep select_packed_members(int ncols, bool real, int max_row_nnz, int ell_w, int64_t NH) {
  PackedStep ps;
  if (!real || ell_w != 8 || max_row_nnz > 8 || ncols < 2 || ncols > 32) return ps;
  const int lanes = ffpk1_lanes_for(ncols);
  ps.fn = ffpk1_lanes<DOT_DOUBLING, true>(lanes, max_row_nnz, slots_from_hbm(NH, ncols));
  ps.threads = kThreads;
  ps.rows_per_block = kThreads / lanes;
  ps.split = (ncols + lanes - 1) / lanes;
  return ps;
}

PackedStep select_packed_step(int ncols, int dot, bool real, int max_row_nnz, int ell_w,
                              int64_t NH) {
  PackedStep ps;
  if (dot == DOT_NONE || !real || ell_w != 8 || max_row_nnz > 8 || ncols < 2 || ncols > kMaxCols) return ps;
  // bra-ket steps of 57..64 columns with rows of 6..8: k_step_ffr (3D L = 100, 64
  // columns 930 us per step, k_step_ffpk1 967; 56 columns 1013 and 937)
  if (dot != DOT_DOUBLING && ncols > 56 && ncols <= 64 && max_row_nnz > 5) return ps;
  const int lanes = ffpk1_lanes_for(ncols);
  ps.threads = kThreads;
  // 49..64 columns with rows of 6..8: two columns per lane (3D L = 100, 64
  // columns 732 us per step, k_step_ffpk1 829); rows of 5: one per lane (2D
  // L = 1024 708 against 702 us, L = 150 17.7 against 15.3)
  if (dot == DOT_DOUBLING && ncols > 48 && ncols <= 64 && max_row_nnz > 5) {
    const bool full = ncols == 64;
    switch (max_row_nnz) {
      case 6: ps.fn = ffpk_w<6>(full); break;
      case 7: ps.fn = ffpk_w<7>(full); break;
      case 8: ps.fn = ffpk_w<8>(full); break;
      default: break;
    }
    ps.rows_per_block = kThreads / 32;
    return ps;
  }
  const bool hbm = slots_from_hbm(NH, ncols);
  ps.fn = dot == DOT_DOUBLING ? ffpk1_lanes<DOT_DOUBLING, false>(lanes, max_row_nnz, hbm)
          : dot == DOT_LR2    ? ffpk1_lanes<DOT_LR2, false>(lanes, max_row_nnz, hbm)
                              : ffpk1_lanes<DOT_LR1, false>(lanes, max_row_nnz, hbm);
  ps.rows_per_block = kThreads / lanes;
  ps.split = (ncols + lanes - 1) / lanes;
  return ps;
}

}  // namespace step
}  // namespace kpmgb
