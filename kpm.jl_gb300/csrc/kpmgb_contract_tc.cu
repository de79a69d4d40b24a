// kpm_2d moment-matrix contraction on the tensor cores (tcgen05), split form.
//
// Gamma[a, b] = sum_k R[a][k] conj(L[b][k]) is one real GEMM over K' = 2K:
// row a of A holds (Re R_0, Im R_0, Re R_1, ...), row b of B holds
// (Re L_0, Im L_0, ...) for the real part and row nl + b holds
// (-Im L_0, Re L_0, ...) for the imaginary part.
//
// Precision (slicing in the manner of Ozaki's scheme): every row is scaled by
// 2^-e (e: exponent of the row's largest entry) and written as five signed
// 8-bit digits d_0..d_4 (|d| <= 128), stored pre-scaled as BF16 planes
// p_i = d_i 2^(-8i) (exact), so that
//     v = 2^(e-7) * sum_i p_i          (rounding <= 2^-39 of the row max)
// and every plane product carries its own weight.  The 15 plane pairs with
// i + j <= 4 feed five TMEM accumulators (128 x 48 FP32 each), one per digit
// level i + j: level l holds multiples of 2^-8l and stays below
// (l+1) 2^22 of them over a chunk of 256 K' elements, so levels 0-3
// accumulate exactly in the tensor core's FP32 and level 4 (2^-32 of the
// leading products) rounds at most to its own last bit.  After each chunk the
// epilogue warps fold the five accumulators into one int64 per output in
// units of 2^-24 (exact for levels 0-3, level 4 rounded to 2^-25) and the
// chunk accumulators are reused.  A K split holds at most 2^24 K' elements,
// so the int64 stays below 2^62.
//
// The double-precision contraction takes the same form with eight digits
// (Planes8 below): every entry becomes a 63-bit integer of its row's scale, the
// 36 plane pairs with i + j <= 7 feed eight accumulators, each exact over a
// chunk of 128 K' elements ((l+1) 2^21 multiples of 2^-8l, l <= 7: at most
// 2^24), folded into two int64 per output (levels 0-3 in units of 2^-24,
// levels 4-7 in units of 2^-56).  What it drops, and when it is nearer than FP64
// FMAs: kpmgb_contract_tc8.cu.
//
// MMA shape: the five B planes of a stage lie one after another along N, so
// A plane i meets B planes 0..4-i in ONE tcgen05.mma of N = 48 (5 - i)
// whose output columns land on the accumulators of levels i..4 (the level
// blocks are adjacent in TMEM): 5 MMAs per 16 K' elements instead of 15, with
// N up to 240 (the tensor pipe's issue cost per instruction was the limit of
// the 15 x N=64 form: 77 % tc-pipe activity at 40 % tensor math).
//
// Data movement: the digit planes are pre-tiled in global memory in the
// canonical no-swizzle K-major UMMA layout, each k-tile's five planes of one
// operand as one (5 x rows) x 32 block, so each pipeline stage is two bulk
// copies (cp.async.bulk, 40 KiB of A planes and 15 KiB of B planes)
// completed on an mbarrier.  Warp roles per CTA: 0 producer, 1 MMA issuer
// (one thread), 2-5 epilogue (one TMEM lane each).  All waits are bounded.
#include <mutex>
#include <type_traits>

#include "kpmgb_tc.cuh"

namespace kpmgb {

namespace {

constexpr int TC_N = Planes5::kN;
constexpr int TC_KT = Planes5::KT;
constexpr int TC_SLICES = Planes5::kSlices;
constexpr uint32_t A_TILE = Planes5::kATile, B_TILE = Planes5::kBTile;

// --------------------------------------------------------------- pre-passes
template <bool FF>
__device__ __forceinline__ void load_pair(const void* base, int64_t idx, float& rh, float& rl,
                                          float& ih, float& il) {
  if constexpr (FF) {
    const float4 v = __ldg(static_cast<const float4*>(base) + idx);
    rh = v.x; rl = v.y; ih = v.z; il = v.w;
  } else {
    const double2 v = __ldg(static_cast<const double2*>(base) + idx);
    rh = __double2float_rn(v.x); rl = __double2float_rn(v.x - (double)rh);
    ih = __double2float_rn(v.y); il = __double2float_rn(v.y - (double)ih);
  }
}

// Four consecutive complex elements kc0..kc0+3 (kc0 a multiple of 4) of a
// float-float block in the column-pair layout, taken in memory order: two
// 32-byte blocks, element 2b + s at floats 8b + s + {0, 2, 4, 6}.  Elements
// at or past `count` read as 0 (count is even).
__device__ __forceinline__ void load4_colpair(const void* base, int64_t e0, int64_t count,
                                              float (&rh)[4], float (&rl)[4], float (&ih)[4],
                                              float (&il)[4]) {
  const float4* f = static_cast<const float4*>(base);
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (2 * b < count) {
      lo = __ldg(f + (e0 / 2 + b) * 2);      // re.hi, re.hi', re.lo, re.lo'
      hi = __ldg(f + (e0 / 2 + b) * 2 + 1);  // im.hi, im.hi', im.lo, im.lo'
    }
    rh[2 * b] = lo.x; rh[2 * b + 1] = lo.y;
    rl[2 * b] = lo.z; rl[2 * b + 1] = lo.w;
    ih[2 * b] = hi.x; ih[2 * b + 1] = hi.y;
    il[2 * b] = hi.z; il[2 * b + 1] = hi.w;
  }
}

// Exponent e of each vector with max |entry| < 2^e (0 for a zero vector).
// colpair: float-float vectors in the column-pair layout (the high parts are
// the first two floats of every 16 bytes).
template <bool FF>
__global__ void __launch_bounds__(256) k_vec_exp(const void* vecs, int64_t K, int nvec, int* exps,
                                                 bool colpair) {
  const int v = blockIdx.x;
  if (v >= nvec) return;
  float m = 0.f;
  if (FF && colpair) {
    const float4* f = static_cast<const float4*>(vecs) + (int64_t)v * K;  // K float4 per vector
    for (int64_t k = threadIdx.x; k < K; k += 256) {
      const float4 q = __ldg(f + k);
      m = fmaxf(m, fmaxf(fabsf(q.x), fabsf(q.y)));
    }
  } else {
    for (int64_t k = threadIdx.x; k < K; k += 256) {
      float rh, rl, ih, il;
      load_pair<FF>(vecs, (int64_t)v * K + k, rh, rl, ih, il);
      m = fmaxf(m, fmaxf(fabsf(rh), fabsf(ih)));
    }
  }
  __shared__ float red[256];
  red[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float mx = red[0];
    int e = 0;
    if (mx > 0.f && isfinite(mx)) {
      frexpf(mx, &e);  // mx in [2^(e-1), 2^e)
      // (hi + lo) stays below 2^e as well: |lo| <= ulp(hi)/2
    }
    exps[v] = e;
  }
}

// Largest |high part| of column-pair vectors (float bits), and the exponent
// of a gathered maximum (as k_vec_exp).
// grid (chunks, nvec): each block folds its strided share of vector
// blockIdx.y into out[v] (zeroed before) with one atomicMax
__global__ void __launch_bounds__(256) k_vec_absmax(const void* vecs, int64_t K, int nvec,
                                                    unsigned* out) {
  const int v = blockIdx.y;
  if (v >= nvec) return;
  const float4* f = static_cast<const float4*>(vecs) + (int64_t)v * K;
  float m = 0.f;
  for (int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x; k < K; k += (int64_t)gridDim.x * 256) {
    const float4 q = __ldg(f + k);
    m = fmaxf(m, fmaxf(fabsf(q.x), fabsf(q.y)));
  }
  __shared__ float red[256];
  red[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  // non-negative floats order as their bit patterns
  if (threadIdx.x == 0) atomicMax(out + v, __float_as_uint(red[0]));
}

__global__ void k_max_to_exp(const unsigned* mx, int n, int* exps) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float m = __uint_as_float(mx[i]);
    int e = 0;
    if (m > 0.f && isfinite(m)) frexpf(m, &e);
    exps[i] = e;
  }
}

// Five signed base-256 digits of the scaled value (vh + vl) * 2^(7-e).  The
// value is first made an integer, N = round(vh 2^(39-e)) + round(vl 2^(39-e))
// (|N| <= 2^39; within one unit, 2^-39 of the vector maximum), so no digit
// loses the low half's bits to an FP32 rounding; the digits then come off N
// from the least significant end, balanced: d_i in [-128, 127] for i >= 1 and
// |d_0| <= 128, with (vh + vl) 2^(7-e) = sum_i d_i 256^-i to that unit.
// `sc` is 2^(39-e) when that is a normal float (then v * sc is the exact
// scaling), else 0 and the scaling goes through ldexpf.  After two digits the
// rest of N (|N| < 2^40) fits 32 bits.
__device__ __forceinline__ void digits(float vh, float vl, int e, float sc,
                                       float (&d)[TC_SLICES]) {
  const float xh = sc != 0.f ? __fmul_rn(vh, sc) : ldexpf(vh, 39 - e);
  const float xl = sc != 0.f ? __fmul_rn(vl, sc) : ldexpf(vl, 39 - e);
  long long n = __float2ll_rn(xh) + __float2ll_rn(xl);
  // balanced digits from the least significant end: d = ((n + 128) mod 256)
  // - 128 in [-128, 127], and n - d is a multiple of 256 (exact shift)
#pragma unroll
  for (int i = TC_SLICES - 1; i >= TC_SLICES - 2; --i) {
    const int di = (((int)n + 128) & 255) - 128;
    d[i] = (float)di;
    n = (n - di) >> 8;
  }
  int m = (int)n;
#pragma unroll
  for (int i = TC_SLICES - 3; i >= 1; --i) {
    const int di = ((m + 128) & 255) - 128;
    d[i] = (float)di;
    m = (m - di) >> 8;
  }
  d[0] = (float)m;
}

// 2^(39-e) as a float when it is normal, else 0 (digits() then uses ldexpf).
__device__ __forceinline__ float digit_scale(int e) {
  const int k = 39 - e;
  return (k >= -126 && k <= 127) ? __int_as_float((k + 127) << 23) : 0.f;
}

// The exact BF16 value of digit d of plane i: d * 2^(-8 i).
template <int I>
__device__ __forceinline__ __nv_bfloat16 plane_bf16(float d) {
  constexpr float kScale = I == 0 ? 1.f : I == 1 ? 0x1p-8f : I == 2 ? 0x1p-16f : I == 3 ? 0x1p-24f
                                                                                       : 0x1p-32f;
  return __float2bfloat16_rn(__fmul_rn(d, kScale));
}

// Write the digit planes of A (R vectors) or B/B' (L vectors) in the
// pre-tiled layout.  One thread per (row, group of 8 real K' elements).
template <bool FF, bool IS_B>
__global__ void __launch_bounds__(256) k_slice(const void* vecs, int64_t K, int nvec,
                                               const int* exps, int64_t ktiles, int rows_pad,
                                               uint8_t* planes, bool colpair) {
  constexpr int ROWS = IS_B ? TC_N : TC_M;
  constexpr uint32_t TILE = IS_B ? B_TILE : A_TILE;
  const int64_t groups = ktiles * (TC_KT / 8);
  const int64_t total = (int64_t)nvec * groups;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    // vector fastest: consecutive threads write consecutive 16-byte rows of
    // one 8-row core matrix (128 contiguous bytes); each thread reads 64
    // contiguous bytes of its own vector
    const int64_t g = idx / nvec;
    const int v = (int)(idx - g * nvec);
    const int64_t kp0 = g * 8;  // first real K' element
    const int e = exps[v];
    const float sc = digit_scale(e);
    float d[8][TC_SLICES];
    float dq[8][TC_SLICES];  // B' digits (IS_B only)
    float rh4[4], rl4[4], ih4[4], il4[4];
    if (FF && colpair) {
      load4_colpair(vecs, (int64_t)v * K + kp0 / 2, K - kp0 / 2, rh4, rl4, ih4, il4);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t kc = kp0 / 2 + j;  // complex element
        rh4[j] = rl4[j] = ih4[j] = il4[j] = 0.f;
        if (kc < K) load_pair<FF>(vecs, (int64_t)v * K + kc, rh4[j], rl4[j], ih4[j], il4[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float rh = rh4[j], rl = rl4[j], ih = ih4[j], il = il4[j];
      digits(rh, rl, e, sc, d[2 * j]);
      digits(ih, il, e, sc, d[2 * j + 1]);
      if constexpr (IS_B) {
#pragma unroll
        for (int i = 0; i < TC_SLICES; ++i) {
          dq[2 * j][i] = -d[2 * j + 1][i];
          dq[2 * j + 1][i] = d[2 * j][i];
        }
      }
    }
    const int64_t kt = kp0 / TC_KT;
    const int kin = (int)(kp0 % TC_KT);
    auto store = [&](int row, float (&dd)[8][TC_SLICES]) {
      const int tile = row / ROWS, r = row % ROWS;
      uint8_t* tbase = planes + (size_t)(tile * ktiles + kt) * (TC_SLICES * TILE);
      auto put = [&](auto plane) {
        constexpr int i = decltype(plane)::value;
        __nv_bfloat16 h[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) h[q] = plane_bf16<i>(dd[q][i]);
        *reinterpret_cast<uint4*>(tbase + tile_off<TC_SLICES * ROWS>(i * ROWS + r, kin)) =
            *reinterpret_cast<const uint4*>(h);
      };
      put(std::integral_constant<int, 0>{});
      put(std::integral_constant<int, 1>{});
      put(std::integral_constant<int, 2>{});
      put(std::integral_constant<int, 3>{});
      put(std::integral_constant<int, 4>{});
    };
    store(v, d);
    if constexpr (IS_B) store(nvec + v, dq);
  }
}

// The same slicing for blocks of 8 consecutive vectors (an 8-row core-matrix
// group; nvec a multiple of 8) and 32 consecutive groups of 8 K' elements:
// warp w reads vector v0 + w (each lane 64 contiguous bytes, the warp
// 2 KB), the digit pieces meet in shared memory, and each store instruction
// then writes whole 128-byte core-matrix rows (two 256-byte runs per warp)
// instead of one 16-byte piece per row.
template <bool FF, bool IS_B>
__global__ void __launch_bounds__(256) k_slice8(const void* vecs, int64_t K, int nvec,
                                                const int* exps, int64_t ktiles,
                                                uint8_t* planes, bool colpair) {
  constexpr int ROWS = IS_B ? TC_N : TC_M;
  constexpr uint32_t TILE = IS_B ? B_TILE : A_TILE;
  constexpr int NSET = IS_B ? 2 : 1;  // B: rows v and nvec + v
  // [..][group][row]: the row index padded to 9 so that a warp's stores
  // (one row, 32 groups) fall on distinct banks
  __shared__ __align__(16) uint4 piece[NSET][TC_SLICES][32][9];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int v0 = blockIdx.y * 8;
  const int64_t groups = ktiles * (TC_KT / 8);
  const int64_t g0 = (int64_t)blockIdx.x * 32;
  const int v = v0 + w;
  const int64_t g = g0 + l;
  if (g < groups) {
    const int64_t kp0 = g * 8;  // first real K' element
    const int e = exps[v];
    const float sc = digit_scale(e);
    float rh4[4], rl4[4], ih4[4], il4[4];
    if (FF && colpair) {
      load4_colpair(vecs, (int64_t)v * K + kp0 / 2, K - kp0 / 2, rh4, rl4, ih4, il4);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t kc = kp0 / 2 + j;
        rh4[j] = rl4[j] = ih4[j] = il4[j] = 0.f;
        if (kc < K) load_pair<FF>(vecs, (int64_t)v * K + kc, rh4[j], rl4[j], ih4[j], il4[j]);
      }
    }
    float d[8][TC_SLICES];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      digits(rh4[j], rl4[j], e, sc, d[2 * j]);
      digits(ih4[j], il4[j], e, sc, d[2 * j + 1]);
    }
    auto put = [&](auto plane) {
      constexpr int i = decltype(plane)::value;
      __nv_bfloat16 h[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) h[q] = plane_bf16<i>(d[q][i]);
      piece[0][i][l][w] = *reinterpret_cast<const uint4*>(h);
      if constexpr (IS_B) {
        // B' row: (-Im, Re) per complex element
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          h[2 * j] = plane_bf16<i>(-d[2 * j + 1][i]);
          h[2 * j + 1] = plane_bf16<i>(d[2 * j][i]);
        }
        piece[NSET - 1][i][l][w] = *reinterpret_cast<const uint4*>(h);
      }
    };
    put(std::integral_constant<int, 0>{});
    put(std::integral_constant<int, 1>{});
    put(std::integral_constant<int, 2>{});
    put(std::integral_constant<int, 3>{});
    put(std::integral_constant<int, 4>{});
  }
  __syncthreads();
  // write phase: rows fastest, then groups (kin 0 and 8 are adjacent 128-byte
  // rows of one 256-byte run), then planes
#pragma unroll
  for (int set = 0; set < NSET; ++set) {
    const int row0 = set == 0 ? v0 : nvec + v0;
    const int tile = row0 / ROWS, r0 = row0 % ROWS;
    for (int q = threadIdx.x; q < TC_SLICES * 32 * 8; q += 256) {
      const int rr = q & 7, gl = (q >> 3) & 31, i = q >> 8;
      const int64_t gg = g0 + gl;
      if (gg >= groups) continue;
      const int64_t kt = gg / (TC_KT / 8);
      const int kin = (int)(gg % (TC_KT / 8)) * 8;
      uint8_t* tbase = planes + (size_t)(tile * ktiles + kt) * (TC_SLICES * TILE);
      *reinterpret_cast<uint4*>(tbase + tile_off<TC_SLICES * ROWS>(i * ROWS + r0 + rr, kin)) =
          piece[set][i][gl][rr];
    }
  }
}

}  // namespace

int launch_vec_absmax(const void* vecs, int64_t K, int nvec, unsigned* out, cudaStream_t s) {
  if (nvec < 1) return KPMGB_OK;
  KPMGB_CUDA(cudaMemsetAsync(out, 0, (size_t)nvec * sizeof(unsigned), s));
  const int chunks = (int)std::max<int64_t>(1, std::min<int64_t>((K + 4095) / 4096, 512));
  // at most 65535 vectors per launch (the grid's y limit)
  for (int v0 = 0; v0 < nvec; v0 += 65535) {
    const int nv = std::min(nvec - v0, 65535);
    k_vec_absmax<<<dim3((unsigned)chunks, (unsigned)nv), 256, 0, s>>>(
        static_cast<const float4*>(vecs) + (int64_t)v0 * K, K, nv, out + v0);
    KPMGB_LAUNCHED();
  }
  return KPMGB_OK;
}

int launch_contract_split(const ContractArgs& a, int precision, cudaStream_t s) {
  const TcPlan pl = plan_for<Planes5>(a.K, a.nr, a.nl, contract_sms());
  if (split_scratch_bytes(a.K, a.nr, a.nl, contract_sms()) > a.scratch_bytes)
    return fail(KPMGB_ERR_ALLOC, "split contraction scratch too small");
  if (!a.status) return fail(KPMGB_ERR_ARGUMENT, "split contraction needs a status word");
  // Layout: the L (B) planes and exponents first, at offsets that depend only
  // on (K, nl), so a caller contracting several right blocks against the same
  // left block (a.reuse_l) skips re-slicing L; then the R (A) planes.
  uint8_t* base = static_cast<uint8_t*>(a.scratch);
  base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(base) + 1023) & ~uintptr_t(1023));
  uint8_t* B = base;
  int* expB = reinterpret_cast<int*>(B + pl.b_bytes);
  uint8_t* A = reinterpret_cast<uint8_t*>(expB) + pl.exp_bytes;
  int* expA = reinterpret_cast<int*>(A + pl.a_bytes);
  double* part = reinterpret_cast<double*>(reinterpret_cast<uint8_t*>(expA) + pl.exp_bytes);
  const bool ff = precision == KPMGB_PREC_FF;
  const int rowsA = pl.mtiles * TC_M, rowsB = pl.ntiles * TC_N;
  const int64_t groupsA = (int64_t)a.nr * pl.ktiles * (TC_KT / 8);
  const int64_t groupsB = (int64_t)a.nl * pl.ktiles * (TC_KT / 8);
  const int gA = (int)std::min<int64_t>((groupsA + 255) / 256, 65535 * 16);
  const int gB = (int)std::min<int64_t>((groupsB + 255) / 256, 65535 * 16);
  // The padding rows of the last A and B tiles (rows nr.. and 2 nl.. of the
  // plane arrays) are not written: the MMAs multiply them only into output
  // rows and columns that the epilogue discards, each output being its own
  // dot product.
  if (!a.reuse_l) {
    if (a.maxL) {
      k_max_to_exp<<<(a.nl + 255) / 256, 256, 0, s>>>(a.maxL, a.nl, expB);
    } else if (ff) {
      k_vec_exp<true><<<a.nl, 256, 0, s>>>(a.L, a.K, a.nl, expB, a.colpair);
    } else {
      k_vec_exp<false><<<a.nl, 256, 0, s>>>(a.L, a.K, a.nl, expB, false);
    }
    KPMGB_LAUNCHED();
    if (a.nl % 8 == 0) {
      const dim3 g8((unsigned)((pl.ktiles * (TC_KT / 8) + 31) / 32), (unsigned)(a.nl / 8));
      if (ff)
        k_slice8<true, true><<<g8, 256, 0, s>>>(a.L, a.K, a.nl, expB, pl.ktiles, B, a.colpair);
      else
        k_slice8<false, true><<<g8, 256, 0, s>>>(a.L, a.K, a.nl, expB, pl.ktiles, B, false);
    } else if (ff) {
      k_slice<true, true><<<gB, 256, 0, s>>>(a.L, a.K, a.nl, expB, pl.ktiles, rowsB, B,
                                              a.colpair);
    } else {
      k_slice<false, true><<<gB, 256, 0, s>>>(a.L, a.K, a.nl, expB, pl.ktiles, rowsB, B,
                                               false);
    }
    KPMGB_LAUNCHED();
  }
  if (a.maxR) {
    k_max_to_exp<<<(a.nr + 255) / 256, 256, 0, s>>>(a.maxR, a.nr, expA);
  } else if (ff) {
    k_vec_exp<true><<<a.nr, 256, 0, s>>>(a.R, a.K, a.nr, expA, a.colpair);
  } else {
    k_vec_exp<false><<<a.nr, 256, 0, s>>>(a.R, a.K, a.nr, expA, false);
  }
  KPMGB_LAUNCHED();
  if (a.nr % 8 == 0) {
    const dim3 g8((unsigned)((pl.ktiles * (TC_KT / 8) + 31) / 32), (unsigned)(a.nr / 8));
    if (ff)
      k_slice8<true, false><<<g8, 256, 0, s>>>(a.R, a.K, a.nr, expA, pl.ktiles, A, a.colpair);
    else
      k_slice8<false, false><<<g8, 256, 0, s>>>(a.R, a.K, a.nr, expA, pl.ktiles, A, false);
  } else if (ff) {
    k_slice<true, false><<<gA, 256, 0, s>>>(a.R, a.K, a.nr, expA, pl.ktiles, rowsA, A,
                                             a.colpair);
  } else {
    k_slice<false, false><<<gA, 256, 0, s>>>(a.R, a.K, a.nr, expA, pl.ktiles, rowsA, A,
                                              false);
  }
  KPMGB_LAUNCHED();
  // GEMM
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(k_contract_tc<Planes5>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(Planes5::kStages * Planes5::kStage));
  });
  if (attr_err != cudaSuccess)
    return fail(KPMGB_ERR_CUDA, "cannot configure the tensor-core contraction: %s",
                cudaGetErrorString(attr_err));
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
  t.skip = nullptr;
  dim3 grid(pl.mtiles, pl.ntiles, pl.nsplit);
  cudaEvent_t t0 = timing_mark(s);
  k_contract_tc<Planes5><<<grid, kThreadsTC, Planes5::kStages * Planes5::kStage, s>>>(t);
  KPMGB_LAUNCHED();
  timing_add(TIMED_CONTRACT_SPLIT, t0, timing_mark(s));
  const int64_t total = (int64_t)a.nr * a.nl;
  const int blocks = (int)std::min<int64_t>((total + 31) / 32, 8192);
  k_tc_reduce<<<std::max(blocks, 1), 256, 0, s>>>(part, pl.nsplit, a.nr, a.nl, a.n0, a.m0, a.NC,
                                                  a.inv_nr, a.dscale, a.parity, a.nmax_row, a.mu, nullptr);
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

}  // namespace kpmgb
