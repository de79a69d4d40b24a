// Cluster-resident kpm_1d recurrence (kernel variant 10).
//
// For operators small enough that one probe column's two recurrence slots fit
// in the shared memory of a thread-block cluster (NH up to ~100k rows with 16
// CTAs), the recurrence of a column runs inside one cluster: CTA q of the
// cluster owns rows [q R, (q+1) R) of both slots in its own shared memory,
// gathers neighbour rows owned by other CTAs through distributed shared memory
// (ld.shared::cluster), and the steps are separated by the hardware cluster
// barrier.  After the initial load nothing touches global memory but the
// operator's index and value arrays where they do not fit in shared memory,
// and each warp's sums of its rows' dots, which k_finish_moments turns into
// moments afterwards.
//
// A step is a chain of latencies: gather, row sum, barrier.  What is not on
// that chain is kept off it: y is stored, the barrier's arrival is signalled,
// and only then are the dots of the step taken, summed over the warp and
// stored, while the other CTAs arrive.  FP64 runs at one warp instruction per
// 64 clocks and SM quarter, so FP64 rows are split over two lanes, one for the
// real and one for the imaginary part, and the warp sum halves its values per
// level (lane_fold).  The operator's column indices are kept as shared-memory
// addresses within the cluster.
//
// The moments are those of the step kernels in a fixed order, whatever the
// schedule.  Every thread of every CTA executes the same sequence of cluster
// barriers (CTAs without rows still take part); there is no spin-wait.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <type_traits>

#include "kpmgb_step.cuh"

namespace kpmgb {
namespace {

using step::FFVal;
using step::ffdot;
using step::ffmac;
using step::ffnorm2;
using step::ff_epilogue;

constexpr int kMaxThreads = 512;
constexpr int kMaxCluster = 16;   // non-portable cluster size limit
constexpr int kChunk = 8;         // nonzeros per anchored chunk (float-float)
// shared memory kept free beside the slots (bounds the rows per CTA)
constexpr size_t kReserved = 1280;
// sums of the dots that one launch may store; longer recurrences take several
// launches that pass the two slots through global memory
constexpr size_t kSumBytes = size_t(64) << 20;

struct ClusterParams {
  const int* rowptr;
  const int* col;
  const void* val;
  int64_t NH;
  int NR;
  int lr;
  int64_t n0, n1;            // steps n0 .. n1 - 1 (1 is the first)
  int last;                  // no launch follows
  void* slot[2];             // row-major NH x NR blocks: v_{n0-1} and (n0 > 1)
                             // v_{n0-2} in, at parity n & 1
  const void* bra;           // row-major NH x NR bra block (lr) or null
  double2* first;            // [warps][2][NR] sums of step 1
  double2* later;            // [step][warps][dots][NR] sums of steps max(n0, 2) ..
  int rows;                  // rows per CTA (the last CTAs may own fewer)
  int cs;                    // CTAs per cluster
  int cap;                   // nonzeros a CTA's shared copy of its rows holds
};

template <bool FF>
struct CVal;
template <>
struct CVal<true> {
  using T = float4;
};
template <>
struct CVal<false> {
  using T = double2;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// shared::cluster address of the same offset in CTA `rank`'s shared memory
__device__ __forceinline__ uint32_t map_rank(uint32_t local, unsigned rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void ld_dsmem(uint32_t a, float4& v) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ld_dsmem(uint32_t a, double2& v) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ void ld_dsmem(uint32_t a, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}

// CACHE: the CTA copies its rows of the operator (row pointers, neighbour
// addresses, values) into shared memory once, so a step reads no global memory
// but the bra of the l/r path.
template <bool FF, bool REALH, bool CACHE>
__global__ void __launch_bounds__(kMaxThreads, 1) k_kpm1d_cluster(
    const __grid_constant__ ClusterParams p) {
  using V = typename CVal<FF>::T;
  using HT = typename std::conditional<FF, typename FFVal<REALH>::T,
                                       typename std::conditional<REALH, double, double2>::type>::type;
  constexpr uint32_t kElem = sizeof(V);
  // lanes per row: FP64 splits a row into its real and imaginary part
  constexpr int LR = FF ? 1 : 2;
  extern __shared__ __align__(16) unsigned char smem[];
  V* slot = reinterpret_cast<V*>(smem);                               // [2][rows]
  HT* s_val = reinterpret_cast<HT*>(slot + 2 * p.rows);                // [cap]  (CACHE)
  uint32_t* s_adr = reinterpret_cast<uint32_t*>(s_val + (CACHE ? p.cap : 0));  // [cap]
  int* s_rowptr = reinterpret_cast<int*>(s_adr + (CACHE ? p.cap : 0));         // [rows + 1]
  const unsigned rank = cluster_rank();
  const int c = (int)cluster_id();  // probe column of this cluster
  const int tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
  const int64_t r0 = (int64_t)rank * p.rows;
  const int64_t left = p.NH - r0;
  const int own = left <= 0 ? 0 : (left < p.rows ? (int)left : p.rows);
  const uint32_t slot_base = (uint32_t)__cvta_generic_to_shared(slot);
  const HT* __restrict__ val = static_cast<const HT*>(p.val);
  const V* __restrict__ bra = static_cast<const V*>(p.bra);
  // slot-0 address of row j within the cluster (row j lives in CTA j / rows)
  auto address = [&](int j) -> uint32_t {
    const unsigned q = (unsigned)(j / p.rows);
    return map_rank(slot_base + (uint32_t)(j - (int)q * p.rows) * kElem, q);
  };

  // v_{n0-1} and, past the first step, v_{n0-2}
  for (int i = tid; i < own; i += nt) {
    const int64_t g = (r0 + i) * p.NR + c;
    const int x = (int)((p.n0 - 1) & 1);
    slot[x * p.rows + i] = static_cast<const V*>(p.slot[x])[g];
    if (p.n0 > 1) slot[(x ^ 1) * p.rows + i] = static_cast<const V*>(p.slot[x ^ 1])[g];
  }
  if constexpr (CACHE) {
    if (own > 0) {
      const int kb = __ldg(p.rowptr + r0);
      const int nk = __ldg(p.rowptr + r0 + own) - kb;  // <= cap (host bound)
      for (int i = tid; i <= own; i += nt) s_rowptr[i] = __ldg(p.rowptr + r0 + i) - kb;
      for (int k = tid; k < nk && k < p.cap; k += nt) {
        s_adr[k] = address(__ldg(p.col + kb + k));
        s_val[k] = __ldg(val + kb + k);
      }
    }
  }
  cluster_arrive();
  cluster_wait();

  const int work = own * LR;
  for (int64_t n = p.n0; n < p.n1; ++n) {
    const int xs = (int)((n - 1) & 1), ys = xs ^ 1;
    const bool first = n == 1;
    const uint32_t xoff = (uint32_t)(xs * p.rows) * kElem;
    // ---- y = H x, or 2 H x - z over z
    for (int e = tid; e < work; e += nt) {
      const int i = e / LR;
      // CACHE: row-local indices into the shared copy; else CSR positions
      const int k0 = CACHE ? s_rowptr[i] : __ldg(p.rowptr + r0 + i);
      const int k1 = CACHE ? s_rowptr[i + 1] : __ldg(p.rowptr + r0 + i + 1);
      auto adr_at = [&](int k) { return (CACHE ? s_adr[k] : address(__ldg(p.col + k))) + xoff; };
      auto val_at = [&](int k) { return CACHE ? s_val[k] : __ldg(val + k); };
      if constexpr (!FF) {
        const int part = e & 1;
        double acc = 0.0;
        for (int k = k0; k < k1; k += 4) {
          // four gathers in flight
          HT h[4];
          double a[4], b[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (k + u >= k1) break;
            h[u] = val_at(k + u);
            if constexpr (REALH) {
              ld_dsmem(adr_at(k + u) + 8 * part, a[u]);
            } else {
              double2 v;
              ld_dsmem(adr_at(k + u), v);
              a[u] = part ? v.y : v.x;
              b[u] = part ? v.x : -v.y;
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (k + u >= k1) break;
            if constexpr (REALH) {
              acc = fma(h[u], a[u], acc);
            } else {
              acc = fma(h[u].x, a[u], acc);
              acc = fma(h[u].y, b[u], acc);
            }
          }
        }
        double* const yp = reinterpret_cast<double*>(slot + ys * p.rows) + e;
        *yp = first ? acc : fma(2.0, acc, -*yp);
      } else {
        float Sr = 0.f, Cr = 0.f, Si = 0.f, Ci = 0.f;
        for (int kc = k0; kc < k1; kc += kChunk) {
          const int cnt = min(kChunk, k1 - kc);
          HT hv[kChunk];
          float4 xv[kChunk];
          float R = 0.f, M = 0.f;
          // issue the chunk's remote loads back to back, then use them
#pragma unroll
          for (int u = 0; u < kChunk; ++u) {
            if (u < cnt) {
              hv[u] = val_at(kc + u);
              ld_dsmem(adr_at(kc + u), xv[u]);
            } else {
              step::hzero(hv[u]);
              xv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
#pragma unroll
          for (int u = 0; u < kChunk; ++u) {
            R = __fadd_rn(R, step::habs(hv[u]));
            M = fmaxf(M, fmaxf(fabsf(xv[u].x), fabsf(xv[u].z)));
          }
          // anchor as the step kernels: 1.5 * 2^E, 2^E = 4P, P <= R*M (1 + tiny) < 2P
          const float B = __fmul_rn(__fmul_rn(R, M), 1.0f + 0x1p-14f);
          const float sig = __fmul_rn(6.0f, ff::pow2_floor(B));
          float Ar = sig, Ai = sig, cr = 0.f, ci = 0.f;
#pragma unroll
          for (int u = 0; u < kChunk; ++u)
            if (u < cnt) ffmac(Ar, cr, Ai, ci, hv[u], xv[u]);
          const float sr = __fsub_rn(Ar, sig), si = __fsub_rn(Ai, sig);
          if (kc == k0) {
            Sr = sr;
            Cr = cr;
            Si = si;
            Ci = ci;
          } else {
            float s, t;
            ff::two_sum(Sr, sr, s, t);
            Sr = s;
            Cr = __fadd_rn(Cr, __fadd_rn(cr, t));
            ff::two_sum(Si, si, s, t);
            Si = s;
            Ci = __fadd_rn(Ci, __fadd_rn(ci, t));
          }
        }
        const int beta_mode = first ? 0 : -1;
        const float alpha = first ? 1.f : 2.f;
        float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!first) z = slot[ys * p.rows + i];
        const float2 yr = ff_epilogue(Sr, Cr, alpha, beta_mode, z.x, z.y);
        const float2 yi = ff_epilogue(Si, Ci, alpha, beta_mode, z.z, z.w);
        // y overwrites z (this row only; other CTAs read the x slot this step)
        slot[ys * p.rows + i] = make_float4(yr.x, yr.y, yi.x, yi.y);
      }
    }
    __syncwarp();
    cluster_arrive();  // y of step n
    // ---- the dots of the thread's own rows, while the others arrive:
    // <x|x>, <x|y> (doubling), <b|x>, <b|y> or <b|y> alone (bra/ket)
    const bool two = !p.lr || first;
    double2 d[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
    if constexpr (!FF) {
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      const double* xp = reinterpret_cast<const double*>(slot + xs * p.rows);
      const double* yp = reinterpret_cast<const double*>(slot + ys * p.rows);
      for (int e = tid; e < work; e += nt) {
        const double x = xp[e], y = yp[e], yo = yp[e ^ 1];
        if (!p.lr) {
          v[0] = fma(x, x, v[0]);
          v[2] = fma(x, y, v[2]);
          v[3] = fma(e & 1 ? -x : x, yo, v[3]);
        } else {
          const double b =
              __ldg(reinterpret_cast<const double*>(bra + (r0 + (e >> 1)) * p.NR + c) + (e & 1));
          if (first) {
            v[0] = fma(b, x, v[0]);
            v[1] = fma(e & 1 ? -b : b, xp[e ^ 1], v[1]);
          }
          v[2] = fma(b, y, v[2]);
          v[3] = fma(e & 1 ? -b : b, yo, v[3]);
        }
      }
      // four values over 32 lanes: after two levels each lane holds one
      step::lane_fold<4, 1>(
          v, lane, [](double a, int off) { return __shfl_xor_sync(0xffffffffu, a, off); },
          [](double a, double b) { return a + b; });
      d[0] = make_double2(__shfl_sync(0xffffffffu, v[0], 0), __shfl_sync(0xffffffffu, v[0], 8));
      d[1] = make_double2(__shfl_sync(0xffffffffu, v[0], 16), __shfl_sync(0xffffffffu, v[0], 24));
    } else {
      float S[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, C[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
      for (int i = tid; i < own; i += nt) {
        const float4 x = slot[xs * p.rows + i], y = slot[ys * p.rows + i];
        if (!p.lr) {
          ffnorm2(S[0], C[0], x);
          ffdot(S[1], C[1], x, y);
        } else {
          const float4 b = __ldg(bra + (r0 + i) * p.NR + c);
          if (first) ffdot(S[0], C[0], b, x);
          ffdot(S[1], C[1], b, y);
        }
      }
      step::F3 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = step::F3{S[q >> 1][q & 1], C[q >> 1][q & 1], 0.f};
      step::lane_fold<4, 1>(
          v, lane,
          [](step::F3 a, int off) {
            return step::F3{__shfl_xor_sync(0xffffffffu, a.s, off),
                            __shfl_xor_sync(0xffffffffu, a.c, off),
                            __shfl_xor_sync(0xffffffffu, a.d, off)};
          },
          [](step::F3 a, step::F3 b) { return step::f3_merge(a, b); });
      const double w = step::f3_join(v[0]);
      d[0] = make_double2(__shfl_sync(0xffffffffu, w, 0), __shfl_sync(0xffffffffu, w, 8));
      d[1] = make_double2(__shfl_sync(0xffffffffu, w, 16), __shfl_sync(0xffffffffu, w, 24));
    }
    if (lane < 2) {
      const int64_t g = (int64_t)rank * nwarps + warp, G = (int64_t)p.cs * nwarps;
      if (first) {
        p.first[(g * 2 + lane) * p.NR + c] = d[lane];
      } else if (two) {
        const int64_t q = n - (p.n0 > 2 ? p.n0 : 2);
        p.later[((q * G + g) * 2 + lane) * p.NR + c] = d[lane];
      } else if (lane == 1) {
        const int64_t q = n - (p.n0 > 2 ? p.n0 : 2);
        p.later[(q * G + g) * p.NR + c] = d[1];
      }
    }
    __syncwarp();
    cluster_wait();  // y of step n is visible cluster-wide, x no longer read
  }
  // the two slots for the next launch
  if (!p.last) {
    for (int i = tid; i < own; i += nt) {
      const int64_t g = (r0 + i) * p.NR + c;
      static_cast<V*>(p.slot[0])[g] = slot[i];
      static_cast<V*>(p.slot[1])[g] = slot[p.rows + i];
    }
  }
}

template <bool FF, bool REALH>
const void* cluster_fn(bool cache) {
  return cache ? (const void*)k_kpm1d_cluster<FF, REALH, true>
               : (const void*)k_kpm1d_cluster<FF, REALH, false>;
}

}  // namespace

namespace {

// Clusters of 1..16 CTAs that the device holds side by side with one CTA per
// SM (clusters lie within one of its processing clusters, so 16 CTAs fit far
// fewer times than SMs / 16).  The first call on a device also allows every
// form of the kernel the most shared memory and the largest clusters, for good:
// the limits belong to the process, and a limit of one call's size would fail
// a larger launch of another thread that had just set its own.
const int* clusters_side_by_side() {
  static std::mutex mtx;
  static std::map<int, std::array<int, kMaxCluster + 1>> table;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mtx);
  auto it = table.find(dev);
  if (it != table.end()) return it->second.data();
  std::array<int, kMaxCluster + 1> side{};
  const void* fn = cluster_fn<false, true>(true);
  constexpr int kOnePerSm = 120 * 1024;  // more than half of an SM's shared memory
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  for (const bool cache : {false, true})
    for (const void* f : {cluster_fn<false, false>(cache), cluster_fn<false, true>(cache),
                          cluster_fn<true, false>(cache), cluster_fn<true, true>(cache)}) {
      cudaFuncAttributes fa{};
      cudaFuncGetAttributes(&fa, f);
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           optin - (int)fa.sharedSizeBytes);
      cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
  for (int cs = 1; cs <= kMaxCluster; ++cs) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cs);
    cfg.blockDim = dim3(64);
    cfg.dynamicSmemBytes = kOnePerSm;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess) side[cs] = n;
  }
  cudaGetLastError();
  return table.emplace(dev, side).first->second.data();
}

struct ClusterShape {
  int cs = 0;         // CTAs per cluster; 0: no cluster holds the rows
  int64_t waves = 0;  // clusters that follow one another on the busiest SM
  int64_t load = 0;   // their rows
};

int64_t max_rows_per_cta() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return ((int64_t)optin - (int64_t)kReserved) / 32;  // two slots of 16 bytes
}

// The cluster size that leaves the busiest SM the fewest rows, counting the
// columns that have to share SMs; rows per CTA stay at 32 or more.
ClusterShape cluster_shape(int64_t NH, int NR) {
  const int* side = clusters_side_by_side();
  const int64_t max_rows = max_rows_per_cta();
  ClusterShape s;
  for (int k = 1; k <= kMaxCluster; ++k) {
    const int64_t r = (NH + k - 1) / k;
    if (r > max_rows || (k > 1 && r < 32) || side[k] < 1) continue;
    const int64_t waves = (NR + side[k] - 1) / side[k];
    if (s.cs == 0 || waves * r < s.load) s = ClusterShape{k, waves, waves * r};
  }
  return s;
}

// Shared memory of one CTA of `rows` rows with its rows of the operator; false
// when that is more than a CTA can have.
bool cached_bytes(const DeviceCSR& H, bool ff, int64_t rows, size_t* bytes, int64_t* cap) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const bool real = H.is_real != 0;
  const size_t hbytes = ff ? (real ? sizeof(float2) : sizeof(float4))
                           : (real ? sizeof(double) : sizeof(double2));
  *cap = rows * (int64_t)std::max(H.max_row_nnz, 1);
  *bytes = 32 * (size_t)rows + (size_t)*cap * (hbytes + sizeof(int)) +
           (size_t)(rows + 1) * sizeof(int);
  return *cap < (1ll << 30) && *bytes + kReserved <= (size_t)optin;
}

}  // namespace

// Whether one cluster launch is expected to beat a launch per step: times per
// step (us) fitted to 6984 measured calls on GB300 (300..32768 rows of 3..19
// entries, 1..400 columns).  Cluster: linear in the rows that the busiest SM
// holds and their entries, with the operator beside the slots (c) or read from
// global memory (u).  Launches of at most 128 columns: the greater of the chain
// of a row, longer with several columns per lane, and all rows x columns, idle
// lanes included.  Measured, cluster / launches: FP64 real NH = 1024, NR = 8
// 1.8 / 4.2; 4096, 12 3.8 / 7.2; 16384, 4 6.6 / 5.3; 15876, 5 8.0 / 11.6; 2048,
// 129 22 / 31; complex 2048, 8 4.7 / 6.6; 8192, 4 11.2 / 6.6; 2450, 11 6.8 /
// 13.4; float-float real 4096, 12 2.2 / 3.5; 32761, 1 4.8 / 3.7; 2048, 129 10.7 /
// 24.  Beyond 2048 rows on an SM, or with the operator in global memory, the
// cluster only serves many columns of few rows, where launches take several
// passes (doubling ones a tenth more than the fit says).  Over those calls the
// choice costs 0.3 to 1.2% more than the faster of the two.
bool cluster_is_faster(const DeviceCSR& H, int64_t NH, int NR, int precision, bool lr, bool pairs) {
  struct Cluster {
    double c[4], u[4];  // chain, per row, per entry, each further wave
  };
  struct Launch {
    double chain[3];  // once, per entry, per entry and further column of a lane
    double work[3];   // once, per row x column, per entry x column
    double lr;        // bra/ket steps, which take fewer dots, against doubling ones
  };
  static constexpr Cluster kCluster[2][2] = {
      {{{2.2, 3.5e-3, 1.8e-3, 0.41}, {3.0, 2.9e-3, 1.7e-3, 0.5}},
       {{2.0, 3.2e-3, 5.5e-4, 0.54}, {1.1, 2.3e-3, 9.8e-4, 0.51}}},
      {{{2.3, 1.5e-3, 3.0e-4, 0.21}, {1.8, 7.4e-4, 7.2e-4, 0.87}},
       {{2.2, 1.3e-3, 2.2e-4, 0.25}, {1.3, 1.0e-3, 5.9e-4, 0.61}}}};  // [float-float][real]
  static constexpr Launch kCsr[2][2] = {
      {{{3.7, 0.34, 0.30}, {4.0, 1.9e-5, 7.8e-6}, 0.94}, {{3.8, 0.20, 0.18}, {3.9, 1.8e-5, 4.2e-6}, 0.91}},
      {{{4.5, 0.10, 0.15}, {5.0, 2.4e-5, 1.3e-6}, 0.92}, {{4.2, 0.12, 0.17}, {4.6, 1.3e-5, 1.8e-6}, 0.91}}};
  static constexpr Launch kPairs[2] = {{{2.4, 0.25, 0.034}, {3.8, 1.4e-5, 5.3e-7}, 1.0},
                                       {{0.84, 0.36, 0.049}, {3.3, 2.6e-6, 1.6e-6}, 0.98}};
  const bool ff = precision == KPMGB_PREC_FF, real = H.is_real != 0;
  const ClusterShape shape = cluster_shape(NH, NR);
  if (shape.cs < 1) return false;
  size_t bytes = 0;
  int64_t cap = 0;
  const bool cache = cached_bytes(H, ff, (NH + shape.cs - 1) / shape.cs, &bytes, &cap);
  const double w = (double)H.nnz / (double)NH;
  const double(&c)[4] = cache ? kCluster[ff][real].c : kCluster[ff][real].u;
  const double cluster = c[0] + (double)shape.load * (c[1] + c[2] * w) +
                         c[3] * (double)(std::min<int64_t>(shape.waves, 4) - 1);
  const Launch& l = pairs ? kPairs[real] : kCsr[ff][real];
  double launches = 0.0;
  for (int c0 = 0; c0 < NR; c0 += step::kMaxCols) {
    const int n = std::min(step::kMaxCols, NR - c0);
    int held = 0, cpl = 1;
    launch_columns(NH, n, precision, lr ? DOT_LR1 : DOT_DOUBLING, pairs, &held, &cpl);
    // a few last columns find theirs far apart in rows of many
    const double apart = n < 8 && c0 > 0 ? 2.0 : 1.0;
    launches += std::max(apart * (l.chain[0] + w * (l.chain[1] + l.chain[2] * (cpl - 1))),
                         l.work[0] + (double)NH * held * (l.work[1] + l.work[2] * w));
  }
  if (lr) launches *= l.lr;
  if (cache && shape.load <= 2048) return cluster < launches;
  return NR > 64 && NH <= 8192 && cluster < (lr ? 1.0 : 1.1) * launches;
}

int launch_kpm1d_cluster(const DeviceCSR& H, int64_t NH, int NR, int64_t NC, bool lr,
                         int precision, void* const (&slots)[2], const void* bra, DevBuf& sums,
                         const MomentArgs& m0, cudaStream_t s) {
  if (NR < 1) return fail(KPMGB_ERR_ARGUMENT, "Invalid NR=%d", NR);
  const bool ff = precision == KPMGB_PREC_FF;
  const bool real = H.is_real != 0;
  const int64_t max_rows = max_rows_per_cta();
  if ((NH + kMaxCluster - 1) / kMaxCluster > max_rows)
    return fail(KPMGB_ERR_ARGUMENT,
                "the cluster-resident kernel holds at most %lld rows per probe column "
                "(%d CTAs of %lld rows)",
                (long long)(kMaxCluster * max_rows), kMaxCluster, (long long)max_rows);
  const int cs = cluster_shape(NH, NR).cs;
  if (cs < 1) return fail(KPMGB_ERR_ARGUMENT, "the device holds no thread-block clusters");
  const int64_t rows = (NH + cs - 1) / cs;
  // the CTA's rows of the operator in shared memory when they fit
  size_t smem = 0;
  int64_t cap = 0;
  const bool cache = cached_bytes(H, ff, rows, &smem, &cap);
  if (!cache) smem = 32 * (size_t)rows;
  const int64_t lanes = rows * (ff ? 1 : 2);
  const int threads = (int)std::min<int64_t>(kMaxThreads, std::max<int64_t>(64, (lanes + 31) / 32 * 32));
  const void* fn = ff ? (real ? cluster_fn<true, true>(cache) : cluster_fn<true, false>(cache))
                      : (real ? cluster_fn<false, true>(cache) : cluster_fn<false, false>(cache));
  // setup failures (no cluster support, attribute limits) are "does not
  // apply here" (argument status), so automatic selection falls back
  auto setup = [&](cudaError_t e) {
    if (e == cudaSuccess) return KPMGB_OK;
    cudaGetLastError();
    return fail(KPMGB_ERR_ARGUMENT, "the cluster-resident kernel cannot run here: %s",
                cudaGetErrorString(e));
  };
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(NR * cs));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  KPMGB_TRY(setup(cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg)));
  if (nclusters < 1)
    return fail(KPMGB_ERR_ARGUMENT, "a cluster of %d CTAs with %zu bytes of shared memory each "
                                    "cannot be resident on this device", cs, smem);
  const int64_t N = lr ? NC - 1 : NC / 2;  // steps
  const int G = cs * (threads / 32);
  const int nd = lr ? 1 : 2;
  const size_t first_bytes = (size_t)G * 2 * NR * sizeof(double2);
  const size_t step_bytes = (size_t)G * nd * NR * sizeof(double2);
  const int64_t most = std::max<int64_t>(
      1, std::min<int64_t>(N - 1, (int64_t)(kSumBytes / step_bytes)));
  size_t room = 0;
  KPMGB_TRY(sums.ensure_some(first_bytes + (size_t)most * step_bytes, first_bytes + step_bytes,
                             &room));
  const int64_t hold = (int64_t)((room - first_bytes) / step_bytes);
  ClusterParams p;
  p.rowptr = H.rowptr;
  p.col = H.col;
  p.val = ff ? H.val_ff : (real ? (const void*)H.val_real : (const void*)H.val);
  p.NH = NH;
  p.NR = NR;
  p.lr = lr ? 1 : 0;
  p.slot[0] = slots[0];
  p.slot[1] = slots[1];
  p.bra = bra;
  p.first = sums.as<double2>();
  p.later = reinterpret_cast<double2*>(sums.as<char>() + first_bytes);
  p.rows = (int)rows;
  p.cs = cs;
  p.cap = cache ? (int)cap : 0;
  MomentArgs m = m0;
  for (int64_t n = 1; n <= N;) {
    const int64_t later = std::max<int64_t>(n, 2);
    p.n0 = n;
    p.n1 = std::min<int64_t>(N + 1, later + hold);
    p.last = p.n1 > N;
    void* args[] = {&p};
    KPMGB_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
    KPMGB_LAUNCHED();
    if (n == 1) {
      m.mom = MOM_STORE;
      m.i0 = 0;
      m.growth_limit = 0.0;
      KPMGB_TRY(launch_finish_sums(p.first, G, 2, NR, 1, m, s));
    }
    m.mom = lr ? MOM_STORE : MOM_DOUBLING;
    m.i0 = lr ? later : 2 * later - 2;
    m.growth_limit = m0.growth_limit;
    if (p.n1 > later) KPMGB_TRY(launch_finish_sums(p.later, G, nd, NR, p.n1 - later, m, s));
    n = p.n1;
  }
  return KPMGB_OK;
}

}  // namespace kpmgb
