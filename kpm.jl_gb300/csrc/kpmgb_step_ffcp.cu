// Complex operators on column pairs (k_step_ffcp): kpm_2d's steps without dots
// (chains and current applications, an even number of columns) and kpm_1d's with
// them (2..128 columns, in parts of 4, 8 or 16 pairs, all parts in one launch).
// A lane owns columns q and q + h of a row, h = ceil(NR / 2), and the call
// stores its vectors in the column-pair layout: per row and q one 32-byte block
// (re.hi, re.hi', re.lo, re.lo', im.hi, im.hi', im.lo, im.lo') for the two
// columns (0 for the second of an odd NR's last pair), so two 16-byte loads
// give the {re.hi}, {re.lo}, {im.hi}, {im.lo} pairs of both columns.  Both
// columns meet the same operator value, so every anchored product of
// k_step_ffc runs once on the pair: per nonzero 4 packed anchored products for
// two columns instead of 8 scalar ones, and likewise for the dots.  Rows of up
// to 8 live slots take one anchored chunk, each lane of a pair then performing
// k_step_ffc's scalar sequence (y bitwise k_step_ffc's); longer rows take two
// chunks merged by TwoSum (the gathers of one row and two columns would not
// fit the registers of two blocks per SM).
// Doubling dots: <x|x> and Re<x|y> (k_step_ffr); LPH lanes hold a row's pairs.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "kpmgb_pk.cuh"
#include "kpmgb_step.cuh"

namespace kpmgb {
namespace step {

using namespace f32x2;

// One lane of a pair of accumulators.
__device__ __forceinline__ F3 side_f3(f2 S, f2 C, int side) {
  float s0, s1, c0, c1;
  upk(S, s0, s1);
  upk(C, c0, c1);
  return side ? F3{s1, c1, 0.f} : F3{s0, c0, 0.f};
}
__device__ __forceinline__ double side_join(f2 S, f2 C, int side) {
  return f3_join(side_f3(S, C, side));
}

template <int LPH, int W, int WL, int DOT, bool FULL>
__global__ void __launch_bounds__(kThreads, 2) k_step_ffcp(
    const __grid_constant__ KBatch batch) {
  const KParams& p = batch.p[DOT == DOT_NONE ? blockIdx.y / (unsigned)batch.p[0].parts : 0];
  pdl_enter();
  constexpr int RPW = 32 / LPH;            // rows per warp
  constexpr int GROUPS = kThreads / LPH;   // rows per block tile
  constexpr int kPieces = W / 4 + W;       // 16-byte pieces of one padded row
  const int lane_q = threadIdx.x % LPH;
  const int half = FULL ? LPH : (p.ncols + 1) / 2;  // pairs per row
  // the pairs of this part of the columns (LPH each, the rest in the last); lanes
  // past the last pair repeat it and store nothing
  const int off = FULL ? 0 : (int)(blockIdx.y % (unsigned)p.parts) * LPH;
  const int pairs = FULL ? LPH : min(LPH, half - off);
  const bool live = FULL || lane_q < pairs;
  const int lg = live ? lane_q : pairs - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPH;              // row of this lane within the warp
  const ulonglong2* __restrict__ x = static_cast<const ulonglong2*>(p.x) + 2 * off;
  const ulonglong2* z = static_cast<const ulonglong2*>(p.z) + 2 * off;
  ulonglong2* y = static_cast<ulonglong2*>(p.y) + 2 * off;
  const f2 alpha2 = pk(p.alpha_f, p.alpha_f);
  const int beta_mode = p.beta_mode;
  const f2 zero2 = pk(0.f, 0.f);
  // per warp, two buffers of RPW padded rows: W indices then W values each
  __shared__ __align__(16) float4 sidx[kThreads / 32][2][RPW][kPieces];
  const unsigned NH = (unsigned)p.NH;  // below 2^31
  const unsigned ntiles = (NH + GROUPS - 1) / GROUPS;
  // the warp's lanes copy the RPW rows of a tile, at most kPer pieces of 16
  // bytes per lane, whose places in the tile stay the same
  constexpr int kPer = (RPW * kPieces + 31) / 32;
  const char* src[kPer];
  int step_bytes[kPer];
  unsigned first_row[kPer], dst[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int q = lane + 32 * i;
    const int rr = q / kPieces, piece = q % kPieces;
    const bool idx = piece < W / 4;
    first_row[i] = warp * RPW + rr;
    const int64_t r = (int64_t)blockIdx.x * GROUPS + warp * RPW + rr;
    src[i] = idx ? reinterpret_cast<const char*>(p.ell_col) + r * (W * 4) + piece * 16
                 : static_cast<const char*>(p.ell_val) + r * (W * 16) + (piece - W / 4) * 16;
    step_bytes[i] = (int)gridDim.x * GROUPS * W * (idx ? 4 : 16);
    dst[i] = (unsigned)__cvta_generic_to_shared(&sidx[warp][0][rr < RPW ? rr : 0][piece]);
  }
  auto stage = [&](unsigned t, int b) {  // called for the tiles of this block in order
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (lane + 32 * i < RPW * kPieces && t * GROUPS + first_row[i] < NH)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         dst[i] + b * (unsigned)sizeof(sidx[0][0])),
                     "l"(src[i])
                     : "memory");
      src[i] += step_bytes[i];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // dots of the two columns: DOUBLING norm, Re<x|y>; LR2 <b|x>, <b|y> (re, im);
  // LR1 <b|y> (re, im)
  constexpr int ND = NDots<DOT>::value;
  constexpr int NP = DOT == DOT_DOUBLING ? 1 : 2;
  constexpr int NV = ND * NP > 0 ? ND * NP : 1;
  const ulonglong2* __restrict__ bra = static_cast<const ulonglong2*>(p.bra) + 2 * off;
  __shared__ double sacc[ND > 0 ? 2 * NV : 1][ND > 0 ? kThreads : 1];
  f2 dS[NV], dC[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    dS[v] = dC[v] = zero2;
    if constexpr (ND > 0) sacc[2 * v][threadIdx.x] = sacc[2 * v + 1][threadIdx.x] = 0.0;
  }
  int rows_since_flush = 0;
  int buf = 0;
  float ymax = 0.f;  // largest |high part| of this thread's outputs (p.vmax)
  stage(blockIdx.x, 0);
  for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x) {
    if (t + gridDim.x < ntiles) stage(t + gridDim.x, buf ^ 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const unsigned r = t * GROUPS + warp * RPW + sub;
    const bool row_ok = r < NH;
    const int* jrow = reinterpret_cast<const int*>(&sidx[warp][buf][sub][0]);
    const float4* hrow = &sidx[warp][buf][sub][W / 4];
    // blocks of 32 bytes: [2 q] = {re.hi pair, re.lo pair}, [2 q + 1] = {im.hi, im.lo}
    const int64_t base = ((int64_t)r * half + lg) * 2;
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
    ulonglong2 z0 = zero, z1 = zero;
    if (row_ok && beta_mode != 0) {
      z0 = __ldcs(z + base);
      z1 = __ldcs(z + base + 1);
    }
    // the row's slots in chunks of at most 8 (one anchor each, merged by
    // TwoSum as in k_step_ff), so that the gathers of a chunk fit the
    // registers of two blocks per SM
    constexpr int CA = WL > 8 ? (WL + 1) / 2 : WL;
    // row sums with the anchors removed: S (leading) + C (correction)
    f2 Sr = zero2, Si = zero2, Cr = zero2, Ci = zero2;
    auto chunk = [&](auto first_tag, int u0, auto n_tag) {
      constexpr int N = decltype(n_tag)::value;
      constexpr bool FIRST = decltype(first_tag)::value;
      ulonglong2 g0[N], g1[N];
      if (row_ok) {
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const int64_t e = ((int64_t)jrow[u0 + u] * half + lg) * 2;
          g0[u] = __ldg(x + e);
          g1[u] = __ldg(x + e + 1);
        }
      } else {
#pragma unroll
        for (int u = 0; u < N; ++u) g0[u] = g1[u] = zero;
      }
      float R = 0.f, M0 = 0.f, M1 = 0.f;
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float4 h = hrow[u0 + u];
        R = __fadd_rn(R, __fadd_rn(fabsf(h.x), fabsf(h.z)));
        float a0, a1, b0, b1;
        upk(g0[u].x, a0, a1);
        upk(g1[u].x, b0, b1);
        M0 = fmaxf(M0, fmaxf(fabsf(a0), fabsf(b0)));
        M1 = fmaxf(M1, fmaxf(fabsf(a1), fabsf(b1)));
      }
      const float s0 =
          __fmul_rn(6.0f, ff::pow2_floor(__fmul_rn(__fmul_rn(R, M0), 1.0f + 0x1p-14f)));
      const float s1 =
          __fmul_rn(6.0f, ff::pow2_floor(__fmul_rn(__fmul_rn(R, M1), 1.0f + 0x1p-14f)));
      const f2 sg = pk(s0, s1);
      f2 ar = sg, ai = sg, cr = zero2, ci = zero2;
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float4 h = hrow[u0 + u];
        const f2 hrh = pk(h.x, h.x), hrl = pk(h.y, h.y);
        const f2 hih = pk(h.z, h.z), hil = pk(h.w, h.w);
        const f2 nih = pk(-h.z, -h.z), nil = pk(-h.w, -h.w);
        amac2(ar, cr, hrh, hrl, g0[u].x, g0[u].y);  // re += h.re x.re
        amac2(ar, cr, nih, nil, g1[u].x, g1[u].y);  // re -= h.im x.im
        amac2(ai, ci, hrh, hrl, g1[u].x, g1[u].y);  // im += h.re x.im
        amac2(ai, ci, hih, hil, g0[u].x, g0[u].y);  // im += h.im x.re
      }
      // the anchor leaves exactly (Sterbenz: the accumulator stayed in the
      // anchor's binade); later chunks merge by TwoSum as in k_step_ff
      const f2 sr = sub2(ar, sg), si = sub2(ai, sg);
      if constexpr (FIRST) {
        Sr = sr;
        Si = si;
        Cr = cr;
        Ci = ci;
      } else {
        f2 s, e;
        two_sum2(Sr, sr, s, e);
        Sr = s;
        Cr = add2(Cr, add2(cr, e));
        two_sum2(Si, si, s, e);
        Si = s;
        Ci = add2(Ci, add2(ci, e));
      }
    };
    chunk(std::true_type{}, 0, std::integral_constant<int, CA>{});
    if constexpr (WL > CA) chunk(std::false_type{}, CA, std::integral_constant<int, WL - CA>{});
    __syncwarp();  // the buffer is restaged two tiles later
    buf ^= 1;
    if (row_ok) {
      f2 out[4];
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const f2 S = part == 0 ? Sr : Si;
        const f2 C = part == 0 ? Cr : Ci;
        const ulonglong2 zz = part == 0 ? z0 : z1;
        const f2 u2 = mul2(alpha2, S);
        const f2 c2 = mul2(alpha2, C);
        f2 yh, yl;
        if (beta_mode == 0) {
          two_sum2(u2, c2, yh, yl);
        } else {
          const f2 s2 = sub2(u2, zz.x);
          const f2 bb = sub2(s2, u2);
          const f2 e2 = sub2(sub2(u2, sub2(s2, bb)), add2(zz.x, bb));
          two_sum2(s2, add2(e2, sub2(c2, zz.y)), yh, yl);
        }
        out[2 * part] = yh;
        out[2 * part + 1] = yl;
      }
      if (live) {
        __stcs(y + base, make_ulonglong2(out[0], out[1]));
        __stcs(y + base + 1, make_ulonglong2(out[2], out[3]));
      }
      if constexpr (ND > 0) {
        if (live) {
          // conj(a) b of both columns into accumulators v (re) and v + 1 (im)
          auto dot = [&](int v, ulonglong2 a0, ulonglong2 a1, f2 br, f2 brl, f2 bi, f2 bil,
                         bool imag) {
            const f2 nr = sub2(zero2, a0.x), ni = sub2(zero2, a1.x);  // exact
            dacc2(dS[v], dC[v], a0.x, nr, a0.y, br, brl);
            dacc2(dS[v], dC[v], a1.x, ni, a1.y, bi, bil);
            if (imag) {
              dacc2(dS[v + 1], dC[v + 1], a0.x, nr, a0.y, bi, bil);
              dacc2(dS[v + 1], dC[v + 1], ni, a1.x, sub2(zero2, a1.y), br, brl);
            }
          };
          if constexpr (DOT == DOT_DOUBLING) {
            const ulonglong2 x0 = __ldg(x + base), x1 = __ldg(x + base + 1);
            dot(0, x0, x1, x0.x, x0.y, x1.x, x1.y, false);
            dot(1, x0, x1, out[0], out[1], out[2], out[3], false);
          } else {
            const ulonglong2 b0 = __ldg(bra + base), b1 = __ldg(bra + base + 1);
            if constexpr (DOT == DOT_LR2) {
              const ulonglong2 x0 = __ldg(x + base), x1 = __ldg(x + base + 1);
              dot(0, b0, b1, x0.x, x0.y, x1.x, x1.y, true);
            }
            dot(NP * (ND - 1), b0, b1, out[0], out[1], out[2], out[3], true);
          }
        }
      }
      if (DOT == DOT_NONE && p.vmax) {
        float a0, a1, b0, b1;
        upk(out[0], a0, a1);
        upk(out[2], b0, b1);
        ymax = fmaxf(ymax, fmaxf(fmaxf(fabsf(a0), fabsf(a1)), fmaxf(fabsf(b0), fabsf(b1))));
      }
    }
    if constexpr (ND > 0) {
      if (++rows_since_flush == kFlushRows) {
        rows_since_flush = 0;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          sacc[2 * v][threadIdx.x] += side_join(dS[v], dC[v], 0);
          sacc[2 * v + 1][threadIdx.x] += side_join(dS[v], dC[v], 1);
          dS[v] = dC[v] = zero2;
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if constexpr (ND > 0) {
    if (any_flush(ntiles, kFlushRows)) {
      double2 d[ND][2];
#pragma unroll
      for (int n = 0; n < ND; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          double part[2] = {0.0, 0.0};
#pragma unroll
          for (int q = 0; q < NP; ++q)
            part[q] = sacc[2 * (n * NP + q) + c][threadIdx.x] +
                      side_join(dS[n * NP + q], dC[n * NP + q], c);
          d[n][c] = make_double2(part[0], part[1]);
        }
      block_dots<ND, LPH, 2>(d, p, half, off, pairs);
    } else {
      F3 f[ND][2][NP];
#pragma unroll
      for (int n = 0; n < ND; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int q = 0; q < NP; ++q) f[n][c][q] = side_f3(dS[n * NP + q], dC[n * NP + q], c);
      block_dots_ff<ND, LPH, 2, NP>(f, p, half, off, pairs);
    }
    return;
  }
  if (p.vmax) {
    // non-negative floats order as their bit patterns
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ymax = fmaxf(ymax, __shfl_xor_sync(0xffffffffu, ymax, off));
    if (lane == 0) atomicMax(p.vmax, __float_as_uint(ymax));
  }
}

namespace {
template <int LPH, int W, int DOT, bool FULL>
KernelFn ffcp_live(int live) {
  switch (W - live) {
    case 0: return k_step_ffcp<LPH, W, W, DOT, FULL>;
    case 1: return k_step_ffcp<LPH, W, W - 1, DOT, FULL>;
    case 2: return k_step_ffcp<LPH, W, W - 2, DOT, FULL>;
    default: return k_step_ffcp<LPH, W, W - 3, DOT, FULL>;
  }
}
template <int LPH, int DOT, bool FULL>
KernelFn ffcp_w(int ell_w, int max_row_nnz) {
  switch (ell_w) {
    case 8: return ffcp_live<LPH, 8, DOT, FULL>(std::max(max_row_nnz, 5));
    case 12: return ffcp_live<LPH, 12, DOT, FULL>(std::max(max_row_nnz, 9));
    default: return nullptr;
  }
}
template <int DOT>
KernelFn ffcp_lanes_of(int lanes, int ell_w, int max_row_nnz) {
  switch (lanes) {
    case 2: return ffcp_w<2, DOT, false>(ell_w, max_row_nnz);
    case 4: return ffcp_w<4, DOT, false>(ell_w, max_row_nnz);
    case 8: return ffcp_w<8, DOT, false>(ell_w, max_row_nnz);
    default: return ffcp_w<16, DOT, false>(ell_w, max_row_nnz);
  }
}

// Lanes per row: 16, or 8 or (long vectors) 4 where that saves over an eighth of
// the lanes.  Doubling step, Haldane 256x256: 24 columns 4 x 3 lanes 70 us, 16
// lanes 82; 40 columns 4 x 5 112 (CSR kernel 264); 72 columns 4 x 9 208 (440);
// 128 columns 310 (495).  100x100, 18 columns: 4 x 3 15.1 us, 16 lanes 14.0.
int ffcp_lanes(int half, int64_t NH) {
  if (half <= 8) return half <= 2 ? 2 : half <= 4 ? 4 : 8;
  auto held = [&](int lanes) { return (half + lanes - 1) / lanes * lanes; };
  int best = 16;
  for (int lanes : {8, 4})
    if (held(lanes) * 8 < held(best) * 7 && (lanes > 4 || NH > 1 << 16 || half > 16)) best = lanes;
  return best;
}
}  // namespace

PackedStep select_colpair_step(int ncols, int dot, bool real, int ell_w, int max_row_nnz,
                               int64_t NH) {
  PackedStep ps;
  if (real || max_row_nnz < 1 || max_row_nnz > ell_w || ncols < 2 || ncols > kMaxCols) return ps;
  const int half = (ncols + 1) / 2, lanes = ffcp_lanes(half, NH);
  ps.threads = kThreads;
  ps.rows_per_block = kThreads / lanes;
  ps.split = (half + lanes - 1) / lanes;
  switch (dot) {
    case DOT_NONE:
      // the contraction walks memory order, whole pairs only; below 6 columns a
      // step has too few lanes in flight (kpm_2d of a Haldane 64x64, 128 moments,
      // NR = 4 1.15 ms, CSR steps 0.96; NR = 6 1.36 and 1.39; 200x150, 64
      // moments, NR = 6 2.86 and 3.72, NR = 24 8.6 and 12.2)
      if (ncols % 2 || ncols < 6) return PackedStep{};
      if (ncols == 16) ps.fn = ffcp_w<8, DOT_NONE, true>(ell_w, max_row_nnz);
      else if (ncols == 32) ps.fn = ffcp_w<16, DOT_NONE, true>(ell_w, max_row_nnz);
      else ps.fn = ffcp_lanes_of<DOT_NONE>(lanes, ell_w, max_row_nnz);
      break;
    case DOT_DOUBLING:
      ps.fn = ffcp_lanes_of<DOT_DOUBLING>(lanes, ell_w, max_row_nnz);
      break;
    case DOT_LR2:
      ps.fn = ffcp_lanes_of<DOT_LR2>(lanes, ell_w, max_row_nnz);
      break;
    default:
      ps.fn = ffcp_lanes_of<DOT_LR1>(lanes, ell_w, max_row_nnz);
  }
  return ps;
}

}  // namespace step
}  // namespace kpmgb
