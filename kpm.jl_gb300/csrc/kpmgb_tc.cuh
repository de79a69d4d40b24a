// The digit-plane contraction on the tensor cores (tcgen05): PTX helpers and
// the GEMM kernel, shared by the five-digit split form (kpmgb_contract_tc.cu,
// where the scheme is described) and the eight-digit double-precision form
// (kpmgb_contract_tc8.cu).  Tile shapes, K splits and scratch sizes:
// kpmgb_contract_plan.h.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "kpmgb_contract_plan.h"
#include "kpmgb_internal.h"

namespace kpmgb {

namespace {

constexpr int TMEM_COLS = 512;  // 2 buffers of 256 columns
constexpr int TMEM_BUF = 256;
constexpr int kSpin = 1 << 22;
constexpr int kThreadsTC = 192;  // 6 warps

// --------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t saddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(uint32_t b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t b, uint32_t tx) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(tx)
               : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint32_t b, uint32_t parity) {
  for (int i = 0; i < kSpin; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(b), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// UMMA shared-memory descriptor, no swizzle, K-major: LBO = 128 B between the
// two K-adjacent 8x16-byte core matrices, SBO = 256 B between 8-row groups.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(128 >> 4) << 16;
  d |= (uint64_t)(256 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// kind::f16 instruction descriptor: D = F32, A = B = BF16, both K-major,
// M = TC_M, N = n (a multiple of 16 up to 256).
__host__ __device__ constexpr uint32_t idesc_for(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(TC_M >> 4) << 24);
}
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                     uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}
// 16 consecutive TMEM columns of this thread's lane (no wait).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Byte offset of element (r, k) inside a ROWS x KT tile (canonical layout);
// the planes of a k-tile form one (S ROWS) x KT tile, plane i in rows
// i ROWS .. (i+1) ROWS - 1.
template <int ROWS>
__host__ __device__ __forceinline__ uint32_t tile_off(int r, int k) {
  return (uint32_t)((k >> 4) * (ROWS * 32) + (r >> 3) * 256 + ((k >> 3) & 1) * 128 + (r & 7) * 16 +
                    (k & 7) * 2);
}

// --------------------------------------------------------------- GEMM
struct TcArgs {
  const uint8_t* A;      // planes [mtiles][ktiles][kAStage]
  const uint8_t* B;      // planes [ntiles][ktiles][kBStage]
  int64_t ktiles;
  int64_t kt_per_split;
  int nr, ncols;         // real rows of A, real rows of B (2 nl)
  const int* expA;
  const int* expB;       // per B row (L vector index = row % nl)
  int nl;
  double* part;          // [split][nr][ncols]
  unsigned* status;
  const unsigned* skip;  // null, or nonzero: nothing to do
};

template <class C>
__global__ void __launch_bounds__(kThreadsTC, 1) k_contract_tc(TcArgs p) {
  constexpr int S = C::kSlices, N = C::kN, STAGES = C::kStages;
  if (p.skip && *p.skip) return;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[4 * STAGES];  // full, empty, tfull, tempty
  __shared__ uint32_t s_tmem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = blockIdx.x, nt = blockIdx.y, sp = blockIdx.z;
  const int64_t kt0 = (int64_t)sp * p.kt_per_split;
  const int64_t kt1 = min(p.ktiles, kt0 + p.kt_per_split);
  const int64_t nkt = kt1 > kt0 ? kt1 - kt0 : 0;
  const int64_t nchunks = (nkt + C::kChunk - 1) / C::kChunk;
  const uint32_t full0 = saddr(&bars[0]), empty0 = saddr(&bars[STAGES]);
  const uint32_t tfull0 = saddr(&bars[2 * STAGES]), tempty0 = saddr(&bars[3 * STAGES]);
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1);
      bar_init(tfull0 + 8 * s, 1);
      bar_init(tempty0 + 8 * s, 4);
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     saddr(&s_tmem)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  const uint32_t sm0 = saddr(smem);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      for (int64_t i = 0; i < nkt; ++i) {
        const int s = (int)(i % STAGES);
        const uint32_t ph = (uint32_t)((i / STAGES) & 1);
        if (!bar_wait(empty0 + 8 * s, ph ^ 1)) {
          atomicOr(p.status, (unsigned)STATUS_TIMEOUT);
          break;
        }
        const int64_t kt = kt0 + i;
        bar_expect(full0 + 8 * s, C::kStage);
        bulk_copy(sm0 + s * C::kStage, p.A + (size_t)(mt * p.ktiles + kt) * C::kAStage, C::kAStage,
                  full0 + 8 * s);
        bulk_copy(sm0 + s * C::kStage + C::kAStage, p.B + (size_t)(nt * p.ktiles + kt) * C::kBStage,
                  C::kBStage, full0 + 8 * s);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int64_t i = 0;
      bool ok = true;
      for (int64_t c = 0; c < nchunks && ok; ++c) {
        const int buf = (int)(c & 1);
        if (!bar_wait(tempty0 + 8 * buf, (uint32_t)(((c >> 1) & 1) ^ 1))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int64_t rem = nkt - c * C::kChunk;
        const int64_t tiles = rem < C::kChunk ? rem : C::kChunk;
        for (int64_t t = 0; t < tiles; ++t, ++i) {
          const int s = (int)(i % STAGES);
          if (!bar_wait(full0 + 8 * s, (uint32_t)((i / STAGES) & 1))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a0 = sm0 + s * C::kStage, b0 = a0 + C::kAStage;
#pragma unroll
          for (int ks = 0; ks < C::KT / 16; ++ks) {
            // the B planes of this K step: rows 0 .. S N - 1 of one tile
            const uint64_t bd = umma_desc(b0 + ks * (S * N * 32));
#pragma unroll
            for (int ia = 0; ia < S; ++ia) {
              // A plane ia x B planes 0 .. S-1-ia -> level blocks ia .. S-1;
              // the chunk's first MMA (ia = 0 covers every block) initialises
              const uint64_t ad =
                  umma_desc(a0 + ks * (S * TC_M * 32) + ia * (TC_M / 8) * 256);
              const bool init = t == 0 && ks == 0 && ia == 0;
              umma(tmem + buf * TMEM_BUF + ia * N, ad, bd, idesc_for(N * (S - ia)),
                   init ? 0u : 1u);
            }
          }
          umma_commit(empty0 + 8 * s);  // stage free once these MMAs retire
        }
        if (ok) umma_commit(tfull0 + 8 * buf);
      }
      if (!ok) atomicOr(p.status, (unsigned)STATUS_TIMEOUT);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;          // TMEM lane quarter this warp may access
    const int row = q * 32 + lane;   // tile row = TMEM lane
    // in units of 2^-24; with eight digits levels 4-7 in units of 2^-56
    long long acc[C::kAcc][N];
#pragma unroll
    for (int h = 0; h < C::kAcc; ++h)
#pragma unroll
      for (int j = 0; j < N; ++j) acc[h][j] = 0;
    bool ok = true;
    for (int64_t c = 0; c < nchunks; ++c) {
      const int buf = (int)(c & 1);
      if (!bar_wait(tfull0 + 8 * buf, (uint32_t)((c >> 1) & 1))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int ac = 0; ac < S; ++ac) {
        // level l is a multiple of 2^-8l below 2^24 of them (exact), but for
        // the five digits' level 4 (below 5 2^-10), which is rounded to 2^-24
        const bool rounded = C::kAcc == 1 && ac == 4;
        const int h = ac / 4 < C::kAcc ? ac / 4 : C::kAcc - 1;
        const float unit = rounded ? 16777216.f : __int_as_float((127 + 8 * ac) << 23);
        const int shift = rounded ? 0 : 24 + 32 * h - 8 * ac;
#pragma unroll
        for (int q16 = 0; q16 < N / 16; ++q16) {
          uint32_t v[16];
          tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + buf * TMEM_BUF + ac * N + q16 * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const long long iv =
                (long long)__float2int_rn(__fmul_rn(__uint_as_float(v[j]), unit));
            acc[h][q16 * 16 + j] += iv << shift;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(tempty0 + 8 * buf);
    }
    if (!ok) atomicOr(p.status, (unsigned)STATUS_TIMEOUT);
    const int a = mt * TC_M + row;
    if (a < p.nr) {
      // value = acc * 2^-24 (+ acc' * 2^-56) * 2^(eA - kLead) * 2^(eB - kLead)
      const int ea = p.expA[a];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const int col = nt * N + j;
        if (col < p.ncols) {
          const int e = ea + p.expB[col % p.nl] - 24 - 2 * C::kLead;
          double vv = (double)acc[0][j];
          if constexpr (C::kAcc == 2) vv = fma((double)acc[1][j], 0x1p-32, vv);
          p.part[((size_t)sp * p.nr + a) * p.ncols + col] = ldexp(vv, e);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TMEM_COLS));
  }
}

__device__ __forceinline__ bool keep_parity(int parity, int n, int m) {
  if (parity == KPMGB_PARITY_NONE) return true;
  const bool odd = ((n + m) & 1) != 0;
  return parity == KPMGB_PARITY_ODD ? odd : !odd;
}

// mu += the sum of the K splits' partials: 32 outputs per block, the splits in
// 8 interleaved parts, then the parts in order (one thread per output walked
// up to 64 splits: 29 us of dependent FP64 additions at 64 x 64 outputs).
__global__ void __launch_bounds__(256)
k_tc_reduce(const double* __restrict__ part, int nsplit, int nr, int nl, int n0, int m0, int NC,
            double inv_nr, const double* __restrict__ dscale, int parity, int nmax_row,
            double2* __restrict__ mu, const unsigned* __restrict__ skip) {
  if (skip && *skip) return;
  __shared__ double2 sum[8][32];
  const int64_t total = (int64_t)nr * nl;
  const int ncols = 2 * nl;
  const int q = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int64_t e0 = blockIdx.x * 32ll; e0 < total; e0 += gridDim.x * 32ll) {
    const int64_t e = e0 + l;
    const int a = (int)(e / nl), b = (int)(e % nl);
    double re = 0.0, im = 0.0;
    if (e < total) {
      for (int s = q; s < nsplit; s += 8) {
        const double* p = part + ((size_t)s * nr + a) * ncols + b;
        re += p[0];
        im += p[nl];
      }
    }
    sum[q][l] = make_double2(re, im);
    __syncthreads();
    if (q == 0 && e < total) {
      for (int k = 1; k < 8; ++k) {
        re += sum[k][l].x;
        im += sum[k][l].y;
      }
      const int n = n0 + a, m = m0 + b;
      if (n < nmax_row && keep_parity(parity, n, m)) {
        const double f = dscale ? inv_nr * dscale[0] : inv_nr;
        double2* dst = mu + (size_t)n + (size_t)NC * m;
        dst->x += re * f;
        dst->y += im * f;
      }
    }
    __syncthreads();
  }
}

}  // namespace

}  // namespace kpmgb
