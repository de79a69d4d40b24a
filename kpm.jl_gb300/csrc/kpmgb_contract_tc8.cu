// The double-precision contraction of kpm_2d on the tensor cores: eight digit
// planes per operand (Planes8, kpmgb_tc.cuh; the scheme of
// kpmgb_contract_tc.cu).
//
// GB300 multiplies FP64 at 0.53 TFMA/s and BF16 at about 1 PFMA/s, so 36 BF16
// products per FP64 product are still some fifty times the FP64 rate.  Every
// entry becomes the integer N = round(v 2^(62-e)), |v| < 2^e over its row
// (exact for entries within 2^-9 of the row maximum, within 2^-63 of it for
// the rest), cut into eight balanced base-256 digits; the digit products of
// i + j <= 7 add up exactly, the dropped ones are 2^-62 of 2^(eL + eR) per term
// (root mean square).  FP64 FMAs round every partial sum: runs of n of them
// cost more than that, unless the terms are far below the product of the
// maxima.  So the planes serve a call when, for every pair of vectors, real and
// imaginary part of the sum by themselves, the terms are large enough to make
// the FP64 sum the worse one (k_pair_gate, from mean squares over chunks of
// 8192 sites), and each chunk is evenly filled, 9 in 16 or more of its parts
// within 2^-5 of its largest, so that its mean squares tell its terms
// (k_vec_gate; at most one chunk in eight may be filled in part).  Random
// probes and what the recurrence makes of them pass, halves that are 0 or small
// as well; probes on single sites, wave packets, parts that are small
// throughout, infinities and NaN do not and keep the FP64 kernel.  The decision
// is a word on the device that each kernel of either form reads first.
//
// The planes of a K range are laid out, multiplied and added to the moments
// before those of the next, in scratch that the call's budget bounds
// (contract_range, kpmgb_contract_plan.h).
#include <mutex>
#include <type_traits>

#include "kpmgb_tc.cuh"

namespace kpmgb {

namespace {

using C8 = Planes8;
constexpr int S8 = C8::kSlices;
// Rounding per product, root mean square, in units of 2^(eL + eR): of the
// planes (digit products beyond i + j = 7: seven of two digits of 74 each at
// 2^-76, and what to_integer rounds), and of a run of n FP64 FMAs over products
// of root mean square 1, times the square root of n.
constexpr double kPlaneNoise = 0x1p-62;
constexpr double kRunNoise = 0.42 * 0x1p-54;

template <bool FF>
__device__ __forceinline__ double2 load_f64(const void* base, int64_t idx) {
  if constexpr (FF) {
    const float4 v = __ldg(static_cast<const float4*>(base) + idx);
    return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
  } else {
    return __ldg(static_cast<const double2*>(base) + idx);
  }
}

__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// A chunk's real parts: exponent field of the largest (of a double), sum of
// squares in units of its power of two squared (0: all are 0), and how many
// reach 2^-4 of that power; the same of its imaginary parts in the high halves.
struct VecStat {
  float re, im;
  unsigned exps, large;
};
static_assert(sizeof(VecStat) == kVecStatBytes, "size of the statistics in the scratch");
// What k_vec_gate leaves in their place: mean squares over 2^2e of the vector.
struct VecLevel {
  float re, im;
  float unused[2];
};
static_assert(sizeof(VecLevel) == sizeof(VecStat), "levels replace the statistics");

// The magnitudes of an entry's parts as bits that order like them.  Float-float
// parts stand for themselves by their leading float, which keeps the FP64
// conversions (a third of the FP64 kernel's own time for a few vectors) out of
// the statistics: |hi| < 2^e bounds hi + lo by 2^e as well.
template <bool FF>
struct Magnitude;
template <>
struct Magnitude<false> {
  using T = unsigned long long;
  static constexpr int kMant = 52;
  static __device__ __forceinline__ void load(const void* base, int64_t i, T& re, T& im) {
    const double2 v = __ldg(static_cast<const double2*>(base) + i);
    re = abs_bits(v.x);
    im = abs_bits(v.y);
  }
  static __device__ __forceinline__ unsigned long long peak(T b) { return b; }
  static __device__ __forceinline__ int mantissa(T b) { return (int)((b >> 29) & 0x7fffff); }
};
template <>
struct Magnitude<true> {
  using T = unsigned;
  static constexpr int kMant = 23;
  static __device__ __forceinline__ void load(const void* base, int64_t i, T& re, T& im) {
    const float4 v = __ldg(static_cast<const float4*>(base) + i);
    re = __float_as_uint(v.x) & 0x7fffffffu;
    im = __float_as_uint(v.z) & 0x7fffffffu;
  }
  static __device__ __forceinline__ unsigned long long peak(T b) {
    return (unsigned long long)__double_as_longlong((double)__uint_as_float(b));
  }
  static __device__ __forceinline__ int mantissa(T b) { return (int)(b & 0x7fffff); }
};

// A magnitude over 2 to the power of exponent field ex, at least its own, as a
// float with 23 bits (0 below 2^-40): integer operations only
template <bool FF>
__device__ __forceinline__ float relative(typename Magnitude<FF>::T b, int ex) {
  const int d = (int)(b >> Magnitude<FF>::kMant) - ex;
  return d < -40 || b == 0 ? 0.f : __int_as_float(((127 + d) << 23) | Magnitude<FF>::mantissa(b));
}

// stat[v][chunk]
template <bool FF>
__global__ void __launch_bounds__(256) k_vec_stat(const void* vecs, int64_t K, int chunks,
                                                  VecStat* stat) {
  using Mag = Magnitude<FF>;
  using B = typename Mag::T;
  __shared__ B peak_re[256], peak_im[256];
  __shared__ float sum_re[256], sum_im[256];
  __shared__ unsigned count[256];
  const int v = blockIdx.y, tid = threadIdx.x;
  const int64_t k0 = (int64_t)blockIdx.x * kStatChunk, k1 = min(K, k0 + kStatChunk);
  B mr = 0, mi = 0;
#pragma unroll 4
  for (int64_t k = k0 + tid; k < k1; k += 256) {
    B re, im;
    Mag::load(vecs, (int64_t)v * K + k, re, im);
    mr = max(mr, re);
    mi = max(mi, im);
  }
  peak_re[tid] = mr;
  peak_im[tid] = mi;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) {
      peak_re[tid] = max(peak_re[tid], peak_re[tid + w]);
      peak_im[tid] = max(peak_im[tid], peak_im[tid + w]);
    }
    __syncthreads();
  }
  const int er = (int)(peak_re[0] >> Mag::kMant), ei = (int)(peak_im[0] >> Mag::kMant);
  float sr = 0.f, si = 0.f;
  unsigned large = 0;
#pragma unroll 4
  for (int64_t k = k0 + tid; k < k1; k += 256) {
    B rb, ib;
    Mag::load(vecs, (int64_t)v * K + k, rb, ib);
    const float re = relative<FF>(rb, er), im = relative<FF>(ib, ei);
    sr = fmaf(re, re, sr);
    si = fmaf(im, im, si);
    large += (re >= 0.0625f ? 1u : 0u) + (im >= 0.0625f ? 1u << 16 : 0u);
  }
  sum_re[tid] = sr;
  sum_im[tid] = si;
  count[tid] = large;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) {
      sum_re[tid] += sum_re[tid + w];
      sum_im[tid] += sum_im[tid + w];
      count[tid] += count[tid + w];
    }
    __syncthreads();
  }
  if (tid == 0)
    stat[(size_t)v * chunks + blockIdx.x] =
        VecStat{sum_re[0], sum_im[0],
                (unsigned)(Mag::peak(peak_re[0]) >> 52) |
                    (unsigned)(Mag::peak(peak_im[0]) >> 52) << 16,
                count[0]};
}

// The mean square of n parts over 2^2e, e one above the exponent field ex.
__device__ __forceinline__ float level_of(float sumsq, int part_ex, int ex, int n) {
  if (sumsq == 0.f) return 0.f;
  return fmaxf(ldexpf(sumsq / (float)n, max(2 * (part_ex - ex) - 2, -200)), 1.18e-38f);
}

// exps[v]: max |part| < 2^e (0 for a zero vector); *fp64 set when a vector is
// not finite or its chunks are unevenly filled; levels in place of the
// statistics.  One warp per vector.
__global__ void __launch_bounds__(32) k_vec_gate(VecStat* stat, int chunks, int64_t K, int nl,
                                                 int* expL, int* expR, unsigned* fp64) {
  const int v = blockIdx.x, lane = threadIdx.x;
  VecStat* const st = stat + (size_t)v * chunks;
  int ex = 0;
  for (int c = lane; c < chunks; c += 32)
    ex = max(ex, (int)max(st[c].exps & 0xffffu, st[c].exps >> 16));
  ex = __reduce_max_sync(0xffffffffu, ex);
  int used = 0, thin = 0;  // chunks that hold parts, and unevenly
  for (int c = lane; c < chunks; c += 32) {
    const VecStat t = st[c];
    const int n = (int)min((int64_t)kStatChunk, K - (int64_t)c * kStatChunk);
    // a short last chunk says little by itself
    const bool judged = n == kStatChunk || chunks == 1;
    const bool re = t.re != 0.f, im = t.im != 0.f;
    used += re || im ? 1 : 0;
    thin += judged && ((re && 16 * (int)(t.large & 0xffffu) < 9 * n) ||
                       (im && 16 * (int)(t.large >> 16) < 9 * n))
                ? 1
                : 0;
    reinterpret_cast<VecLevel*>(st)[c] =
        VecLevel{level_of(t.re, (int)(t.exps & 0xffffu), ex, n),
                 level_of(t.im, (int)(t.exps >> 16), ex, n), {0.f, 0.f}};
  }
  used = __reduce_add_sync(0xffffffffu, used);
  thin = __reduce_add_sync(0xffffffffu, thin);
  if (lane == 0) {
    (v < nl ? expL + v : expR + (v - nl))[0] = used == 0 ? 0 : max(ex, 1) - 1022;
    if (ex == 0x7ff || 8 * thin > used) atomicOr(fp64, 1u);
  }
}

// *fp64 set when a wanted pair's products are too small for the planes: the
// mean square of the products over the sites where both vectors hold parts,
// over 2^2(eL + eR), below `least`; for the real and the imaginary part of the
// sum by itself.
__global__ void __launch_bounds__(256) k_pair_gate(const VecLevel* level, int chunks, int64_t K,
                                                   int nl, int nr, int n0, int m0, int parity,
                                                   int nmax_row, float least, unsigned* fp64) {
  __shared__ float2 sl[16][17], sr[16][17];
  if (*fp64) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int b0 = blockIdx.x * 16, a0 = blockIdx.y * 16;
  float re = 0.f, im = 0.f, nre = 0.f, nim = 0.f;
  for (int c0 = 0; c0 < chunks; c0 += 16) {
    const float2 zero = make_float2(0.f, 0.f);
    auto at = [&](int64_t v, bool have) {
      return have && c0 + tx < chunks
                 ? *reinterpret_cast<const float2*>(level + v * chunks + c0 + tx)
                 : zero;
    };
    sl[ty][tx] = at(b0 + ty, b0 + ty < nl);
    sr[ty][tx] = at(nl + a0 + ty, a0 + ty < nr);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const float2 l = sl[tx][u], r = sr[ty][u];
      const float n = (float)max((int64_t)0, min((int64_t)kStatChunk, K - (int64_t)(c0 + u) * kStatChunk));
      const float rr = l.x * r.x, ii = l.y * r.y, ri = l.x * r.y, ir = l.y * r.x;
      re = fmaf(n, rr + ii, re);
      im = fmaf(n, ri + ir, im);
      nre += (l.x != 0.f && r.x != 0.f) || (l.y != 0.f && r.y != 0.f) ? n : 0.f;
      nim += (l.x != 0.f && r.y != 0.f) || (l.y != 0.f && r.x != 0.f) ? n : 0.f;
    }
    __syncthreads();
  }
  const int n = n0 + a0 + ty, m = m0 + b0 + tx;
  if (a0 + ty < nr && b0 + tx < nl && n < nmax_row && keep_parity(parity, n, m) &&
      !(re >= least * nre && im >= least * nim))
    atomicOr(fp64, 1u);
}

// round(v 2^(62-e)) for |v| < 2^e
__device__ __forceinline__ long long to_integer(double v, int e) {
  const unsigned long long b = abs_bits(v);
  const int ex = (int)(b >> 52);
  unsigned long long m = b & 0xfffffffffffffull;
  if (ex > 0) m |= 0x10000000000000ull;
  const int sh = 62 - e + (ex > 0 ? ex : 1) - 1075;  // at most 9
  if (sh >= 0) {
    m <<= sh;
  } else {
    m = sh >= -54 ? (m + (1ull << (-sh - 1))) >> -sh : 0;
  }
  return __double_as_longlong(v) < 0 ? -(long long)m : (long long)m;
}

// Balanced base-256 digits of n, least significant first: digit i in byte i,
// [-128, 127] below the top one (|top| <= 64).  Adding 128 to every lower byte
// carries exactly where a digit is negative; taking it off per byte (an
// exclusive or of the top bit) leaves two's complement digits.
__device__ __forceinline__ unsigned long long digit_bytes(long long n) {
  return ((unsigned long long)n + 0x0080808080808080ull) ^ 0x0080808080808080ull;
}

// The BF16 bits of digit byte d (two's complement) of plane i: d 2^(-8 i).
template <int I>
__device__ __forceinline__ uint32_t plane_bits(int d) {
  // float(d) by the 1.5 2^23 offset, exact; BF16 keeps its 8 leading bits
  const float f = __int_as_float(0x4B400000 + d) - 12582912.f;
  constexpr float kScale = I == 0 ? 1.f : I == 1 ? 0x1p-8f : I == 2 ? 0x1p-16f : I == 3 ? 0x1p-24f
                         : I == 4 ? 0x1p-32f : I == 5 ? 0x1p-40f : I == 6 ? 0x1p-48f : 0x1p-56f;
  return __float_as_uint(__fmul_rn(f, kScale)) >> 16;
}

// Digit planes of the K range kb .. ke (complex elements) of nvec vectors in
// the pre-tiled layout: blocks of 8 vectors x 32 groups of 8 K' elements;
// warp w reads vector v0 + w, the 16-byte pieces meet in shared memory (rows
// padded to 9) and leave as whole 128-byte core-matrix rows.  Elements at or
// past ke are 0.  IS_B: rows v hold (Re, Im), rows nvec + v (-Im, Re).
template <bool FF, bool IS_B>
__global__ void __launch_bounds__(256) k_slice_f64(const void* vecs, int64_t K, int64_t kb,
                                                   int64_t ke, int nvec, const int* exps,
                                                   int64_t ktiles, uint8_t* planes,
                                                   const unsigned* skip) {
  if (*skip) return;
  constexpr int ROWS = IS_B ? C8::kN : TC_M;
  constexpr uint32_t TILE = IS_B ? C8::kBTile : C8::kATile;
  __shared__ __align__(16) uint4 piece[S8][32][9];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int v0 = blockIdx.y * 8, v = v0 + w;
  const int64_t groups = ktiles * (C8::KT / 8);
  const int64_t g0 = (int64_t)blockIdx.x * 32, g = g0 + l;
  const bool have = v < nvec && g < groups;
  unsigned long long dr[4] = {}, di[4] = {};
  if (have) {
    const int e = exps[v];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t k = kb + g * 4 + j;
      if (k < ke) {
        const double2 x = load_f64<FF>(vecs, (int64_t)v * K + k);
        dr[j] = digit_bytes(to_integer(x.x, e));
        di[j] = digit_bytes(to_integer(x.y, e));
      }
    }
  }
#pragma unroll
  for (int set = 0; set < (IS_B ? 2 : 1); ++set) {
    if (set) __syncthreads();  // the pieces of the first set have left
    if (have) {
      auto put = [&](auto plane) {
        constexpr int i = decltype(plane)::value;
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = (int)(signed char)(dr[j] >> (8 * (S8 - 1 - i)));
          const int m = (int)(signed char)(di[j] >> (8 * (S8 - 1 - i)));
          h[j] = set == 0 ? plane_bits<i>(r) | plane_bits<i>(m) << 16
                          : plane_bits<i>(-m) | plane_bits<i>(r) << 16;
        }
        piece[i][l][w] = make_uint4(h[0], h[1], h[2], h[3]);
      };
      put(std::integral_constant<int, 0>{});
      put(std::integral_constant<int, 1>{});
      put(std::integral_constant<int, 2>{});
      put(std::integral_constant<int, 3>{});
      put(std::integral_constant<int, 4>{});
      put(std::integral_constant<int, 5>{});
      put(std::integral_constant<int, 6>{});
      put(std::integral_constant<int, 7>{});
    }
    __syncthreads();
    for (int q = threadIdx.x; q < S8 * 32 * 8; q += 256) {
      const int rr = q & 7, gl = (q >> 3) & 31, i = q >> 8;
      const int64_t gg = g0 + gl;
      if (gg >= groups || v0 + rr >= nvec) continue;
      const int row = (set == 0 ? 0 : nvec) + v0 + rr;
      const int64_t kt = gg / (C8::KT / 8);
      const int kin = (int)(gg % (C8::KT / 8)) * 8;
      uint8_t* tbase = planes + (size_t)(row / ROWS * ktiles + kt) * (S8 * TILE);
      *reinterpret_cast<uint4*>(tbase + tile_off<S8 * ROWS>(i * ROWS + row % ROWS, kin)) =
          piece[i][gl][rr];
    }
  }
}

template <bool FF>
int launch_planes(const ContractArgs& a, const Layout8& l, uint8_t* base, cudaStream_t s) {
  const TcPlan& pl = l.pl;
  uint8_t *B = base + l.b, *A = base + l.a;
  int* expB = reinterpret_cast<int*>(base + l.expB);
  int* expA = reinterpret_cast<int*>(base + l.expA);
  VecStat* stat = reinterpret_cast<VecStat*>(base + l.stat);
  unsigned* gate = reinterpret_cast<unsigned*>(base + l.gate);
  double* part = reinterpret_cast<double*>(base + l.part);
  KPMGB_CUDA(cudaMemsetAsync(gate, 0, sizeof(unsigned), s));
  auto stats = [&](const void* vecs, int nvec, VecStat* out) -> int {
    for (int v0 = 0; v0 < nvec; v0 += 65535) {  // the grid's y limit
      const int nv = std::min(nvec - v0, 65535);
      const void* p = static_cast<const char*>(vecs) + (size_t)v0 * a.K * 16;
      k_vec_stat<FF><<<dim3((unsigned)l.chunks, (unsigned)nv), 256, 0, s>>>(
          p, a.K, l.chunks, out + (size_t)v0 * l.chunks);
      KPMGB_LAUNCHED();
    }
    return KPMGB_OK;
  };
  KPMGB_TRY(stats(a.L, a.nl, stat));
  KPMGB_TRY(stats(a.R, a.nr, stat + (size_t)a.nl * l.chunks));
  k_vec_gate<<<(unsigned)(a.nl + a.nr), 32, 0, s>>>(stat, l.chunks, a.K, a.nl, expB, expA, gate);
  KPMGB_LAUNCHED();
  // a slice of the FP64 kernel adds at least this many products one by one
  const int64_t run =
      std::max<int64_t>(1, a.K / simt_slices(a.K, a.nr, a.nl, contract_sms()));
  const float least = (float)(kPlaneNoise * kPlaneNoise / (kRunNoise * kRunNoise * (double)run));
  k_pair_gate<<<dim3((unsigned)((a.nl + 15) / 16), (unsigned)((a.nr + 15) / 16)), 256, 0, s>>>(
      reinterpret_cast<const VecLevel*>(stat), l.chunks, a.K, a.nl, a.nr, a.n0, a.m0, a.parity,
      a.nmax_row, least, gate);
  KPMGB_LAUNCHED();
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  constexpr int kSmem = (int)(C8::kStages * C8::kStage);
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(k_contract_tc<C8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmem);
  });
  if (attr_err != cudaSuccess)
    return fail(KPMGB_ERR_CUDA, "cannot configure the tensor-core contraction: %s",
                cudaGetErrorString(attr_err));
  const unsigned gx = (unsigned)((pl.ktiles * (C8::KT / 8) + 31) / 32);
  for (int64_t kb = 0; kb < a.K; kb += l.range) {
    const int64_t ke = std::min(a.K, kb + l.range);
    k_slice_f64<FF, true><<<dim3(gx, (unsigned)((a.nl + 7) / 8)), 256, 0, s>>>(
        a.L, a.K, kb, ke, a.nl, expB, pl.ktiles, B, gate);
    KPMGB_LAUNCHED();
    k_slice_f64<FF, false><<<dim3(gx, (unsigned)((a.nr + 7) / 8)), 256, 0, s>>>(
        a.R, a.K, kb, ke, a.nr, expA, pl.ktiles, A, gate);
    KPMGB_LAUNCHED();
    TcArgs t;
    t.A = A;
    t.B = B;
    t.ktiles = pl.ktiles;
    t.kt_per_split = pl.kt_per_split;
    t.nr = a.nr;
    t.ncols = 2 * a.nl;
    t.expA = expA;
    t.expB = expB;
    t.nl = a.nl;
    t.part = part;
    t.status = a.status;
    t.skip = gate;
    k_contract_tc<C8><<<dim3(pl.mtiles, pl.ntiles, pl.nsplit), kThreadsTC, kSmem, s>>>(t);
    KPMGB_LAUNCHED();
    const int64_t total = (int64_t)a.nr * a.nl;
    k_tc_reduce<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 31) / 32, 8192)), 256,
                  0, s>>>(part, pl.nsplit, a.nr, a.nl, a.n0, a.m0, a.NC, a.inv_nr, a.dscale,
                          a.parity, a.nmax_row, a.mu, gate);
    KPMGB_LAUNCHED();
  }
  return KPMGB_OK;
}

}  // namespace

// The gate word (nonzero: the FP64 kernel has to run) is the first of scratch.
int launch_contract_planes8(const ContractArgs& a, int precision, cudaStream_t s) {
  if (!a.status) return fail(KPMGB_ERR_ARGUMENT, "the contraction needs a status word");
  const Layout8 l = layout8(a.K, a.nr, a.nl, a.range, contract_sms());
  if (l.bytes > a.scratch_bytes)
    return fail(KPMGB_ERR_ALLOC, "scratch too small for the contraction's digit planes");
  uint8_t* base = static_cast<uint8_t*>(a.scratch);
  return precision == KPMGB_PREC_FF ? launch_planes<true>(a, l, base, s)
                                    : launch_planes<false>(a, l, base, s);
}

}  // namespace kpmgb
