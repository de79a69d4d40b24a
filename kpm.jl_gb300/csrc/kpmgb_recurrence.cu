// Chebyshev recurrence kernels with fused moment reductions.
//
// One launch applies y = alpha * H x + beta * z to a row-major NH x NR block
// (row r holds the NR probe columns contiguously), which is the GPU form of
// chebyshev_iter_single (src/utils/chebyshev_iteration.jl:59-75,
// ext/KPMCUDAExt.jl:84-88), and in the same pass accumulates the column-wise
// inner products that the reference computes with separate columnwise_dot!
// passes (src/utils/vectors.jl:103-117, ext/KPMCUDAExt.jl:128-145).
//
// Thread mapping: a group of LPR consecutive lanes owns one row; lane g of the
// group owns columns g, g + LPR, ..., g + (CPL-1) LPR.  For NR = 64 a full
// warp owns a row and every neighbour's row of x is read as two coalesced
// 512-byte warp loads (16 bytes per lane).  The operator row (column indices
// and values) is read once per group and broadcast.
//
// Reductions are deterministic: warp shuffles, then a fixed-order sum over the
// warps of a block, per-block partials in global memory, and a fixed-order
// sum over blocks by k_finish_moments, one launch for the steps whose
// partials the scratch buffer holds.
// The grid size is a pure function of the problem shape, so two identical
// calls give bitwise-identical moments.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <mutex>
#include <unordered_map>

#include "kpmgb_step.cuh"

namespace kpmgb {
namespace {

using namespace step;

// --------------------------------------------------------------- dispatch
// 9..12 columns: four lanes of three columns, which leave no lane idle (FP64
// NH = 262144, 12 columns 106 us per step against the 144 of 16 lanes; kpm_2d of
// a square 360x360, float-float, 64 moments, 12 columns 9.4 ms, 16 lanes 12.9).
// Float-float steps with dots take 16 lanes, more rows in flight, below 40000
// rows (9 real entries, 12 columns: 2000 rows 7.6 us against 12.0, 20000 19.3
// and 18.8, 40000 30.2 and 25.8, 250000 172 and 115; 19 entries 2000 8.8 and
// 13.9, 250000 237 and 148; 5 complex entries 20000 15.1 and 17.8, 80000 39.5
// and 35.3).
// Lanes per row times columns per lane; a shape narrower than the launch runs
// the columns in parts.  Idle lanes cost as much as live ones (FP64: the pipe
// serves whole warps; float-float: the issue slots), so parts of 16 or 8 serve
// where they save over a sixteenth of the lanes.  FP64, per step: Haldane
// 256x256, 20 columns 8 x 3 268 us, 32 lanes 347; 40 columns 8 x 5 440, 32 x 2
// 681; 72 columns 8 x 9 786, 32 x 4 1373; square 512x512, 48 columns 16 x 3
// 409, 8 x 6 413, 32 x 2 553; 150x150, 20 columns 24.1, 32 lanes 28.1.
// Float-float bra moments, square 512x512, 72 columns 531 us, 32 x 4 lanes 705.
// Below 8192 rows, where parts leave few rows in flight, they have to save more
// (3D L = 14, bra moments, 56 columns 8 x 7 19.4 us, 32 x 2 16.3).
Shape pick_shape(int ncols, int precision, int dot, int64_t NH) {
  if (ncols <= 1) return {1, 1};
  if (ncols <= 2) return {2, 1};
  if (ncols <= 4) return {4, 1};
  if (ncols <= 8) return {8, 1};
  if (ncols <= 12 && (precision == KPMGB_PREC_FP64 || dot == DOT_NONE || NH >= 40000))
    return {4, 3};
  if (ncols <= 16) return {16, 1};
  Shape best = ncols <= 32 ? Shape{32, 1} : ncols <= 64 ? Shape{32, 2} : Shape{32, 4};
  int width = best.lpr * best.cpl;
  // float-float shapes of one and two columns per lane anchor other chunks of a
  // row; up to 64 columns keep theirs
  if (precision == KPMGB_PREC_FF && ncols <= 64) return best;
  for (int lanes : {32, 16, 8}) {
    const int held = (ncols + lanes - 1) / lanes * lanes;
    if (held * 16 < width * (NH < 8192 ? 13 : 15)) {
      best = {lanes, 1};
      width = held;
    }
  }
  return best;
}

// Register-gather shapes that cover ncols columns with at most 4x idle lanes,
// the automatic one first (candidates of the autotuner).
std::vector<Shape> candidate_shapes(int ncols, int precision, int dot, int64_t NH) {
  static const Shape all[] = {{1, 1}, {2, 1}, {4, 1}, {8, 1}, {4, 3},
                              {16, 1}, {32, 1}, {32, 2}, {32, 4}};
  std::vector<Shape> out{pick_shape(ncols, precision, dot, NH)};
  for (const Shape& s : all) {
    const int cover = s.lpr * s.cpl;
    if (cover >= ncols && cover <= 4 * std::max(ncols, 8) &&
        !(s.lpr == out[0].lpr && s.cpl == out[0].cpl))
      out.push_back(s);
  }
  return out;
}

Shape shape_for(const StepArgs& a, int ncols, int precision) {
  if (a.shape > 0) {
    const Shape s{a.shape / 10, a.shape % 10};
    if (s.lpr * s.cpl >= ncols) return s;
  }
  return pick_shape(ncols, precision, a.dot, a.NH);
}

KernelFn select_kernel(Shape s, int precision, int dot, bool real) {
  return precision == KPMGB_PREC_FF ? select_kernel_ff(s, dot, real)
                                    : select_kernel_f64(s, dot, real);
}

int num_sms() {
  static int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return sms;
}

// Grid size: resident blocks per SM times the SM count, capped by the number
// of row tiles.  Depends only on the kernel and the shape (determinism).
int blocks_per_sm(KernelFn fn) {
  static std::mutex m;
  static std::unordered_map<const void*, int> cache;
  std::lock_guard<std::mutex> lk(m);
  auto it = cache.find((const void*)fn);
  if (it != cache.end()) return it->second;
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, 0) != cudaSuccess)
    per_sm = 1;
  per_sm = std::max(per_sm, 1);
  // Shared-memory carve-out: the step kernels need only their reduction
  // buffers, so ask for the smallest carve-out that still holds the resident
  // blocks and leave the rest of the unified storage to L1 for the neighbour
  // gathers (measured +3% on the 3D Anderson workload).  KPMGB_CARVEOUT
  // (percent) overrides; the hint is dropped if it would lower occupancy.
  static const int forced = [] {
    const char* e = std::getenv("KPMGB_CARVEOUT");
    return e ? std::atoi(e) : -1;
  }();
  cudaFuncAttributes fa{};
  int dev = 0, maxsm = 0;
  if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) ==
          cudaSuccess &&
      maxsm > 0) {
    const size_t need = (size_t)per_sm * (fa.sharedSizeBytes + 1024);
    int pct = forced >= 0 && forced <= 100 ? forced
                                           : (int)std::min<size_t>(100, (100 * need + maxsm - 1) / maxsm);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct) ==
        cudaSuccess) {
      int again = 0;
      const bool ok =
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&again, fn, kThreads, 0) == cudaSuccess;
      if (forced < 0) {
        if (!ok || again < per_sm)
          cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, -1);
      } else if (ok && again > 0) {
        per_sm = again;
      }
    }
    cudaGetLastError();
  }
  cache.emplace((const void*)fn, per_sm);
  return per_sm;
}

// The kernel of a step for a launch of some columns, with its grid.
struct StepChoice {
  KernelFn fn = nullptr;
  int grid = 0;
  int threads = kThreads;
  int slots = 0;  // resident blocks where early launches depend on them, else 0
  int split = 1;  // parts of the columns
  int batch = kMaxBatch;  // steps without dots per launch
};

// Step kernels launch with programmatic stream serialization (see pdl_enter)
// on every stream, the default ones included: the next step's blocks are in
// place when a step ends, 1.5-3 us less per step (square 150x150, NR = 14,
// float-float 8.3 -> 5.9 us; 512x512, NR = 4, FP64 40.6 -> 37.5 us).
// KPMGB_PDL=0 in the environment turns it off.
int launch_step_kernel(const StepChoice& c, int n, cudaStream_t s, const KBatch& p) {
  static const bool on = [] {
    const char* e = std::getenv("KPMGB_PDL");
    return !(e && e[0] == '0');
  }();
  const dim3 grid((unsigned)c.grid, (unsigned)(n * c.split));
  const int blocks = c.grid * n * c.split;
  const bool early = c.slots == 0 || blocks >= c.slots || 2 * blocks <= c.slots;
  if (!on || !early) {
    c.fn<<<grid, c.threads, 0, s>>>(p);
    KPMGB_LAUNCHED();
    return KPMGB_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)c.threads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  KPMGB_CUDA(cudaLaunchKernelEx(&cfg, c.fn, p));
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

// Columns per step launch: kMaxCols, or fewer through KPMGB_COLS_PER_LAUNCH
// (a tuning knob: narrower launches give each lane group shorter rows).
int cols_per_launch() {
  static const int w = [] {
    const char* e = std::getenv("KPMGB_COLS_PER_LAUNCH");
    const int v = e ? std::atoi(e) : kMaxCols;
    return v >= 1 && v <= kMaxCols ? v : kMaxCols;
  }();
  return w;
}

// Automatic selection of the padded-row kernel for complex operators
// (KPMGB_PADDED_COMPLEX=1; off by default).
bool padded_complex() {
  static const bool on = [] {
    const char* e = std::getenv("KPMGB_PADDED_COMPLEX");
    return e && std::atoi(e) != 0;
  }();
  return on;
}

// Automatic selection of the complex row-streaming kernel
// (KPMGB_STREAMING_COMPLEX=0 turns it off).
const bool kStreamingComplex = [] {
  const char* e = std::getenv("KPMGB_STREAMING_COMPLEX");
  return !(e && std::atoi(e) == 0);
}();

int grid_for(KernelFn fn, int64_t NH, int lpr, int split = 1) {
  const int per_sm = blocks_per_sm(fn);
  const int64_t groups = kThreads / lpr;
  const int64_t tiles = (NH + groups - 1) / groups;
  return (int)std::max<int64_t>(
      1, std::min<int64_t>(tiles, (int64_t)per_sm * num_sms() / split));
}

// Grid of a packed step: resident blocks per SM times the SM count, capped by
// the row tiles.
int grid_packed(const PackedStep& ps, int64_t NH) {
  static std::mutex m;
  static std::unordered_map<const void*, int> cache;
  int per_sm = 1;
  {
    std::lock_guard<std::mutex> lk(m);
    auto it = cache.find((const void*)ps.fn);
    if (it != cache.end()) {
      per_sm = it->second;
    } else {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ps.fn, ps.threads, 0) !=
          cudaSuccess)
        per_sm = 1;
      per_sm = std::max(per_sm, 1);
      cudaGetLastError();
      cache.emplace((const void*)ps.fn, per_sm);
    }
  }
  const int64_t tiles = (NH + ps.rows_per_block - 1) / ps.rows_per_block;
  return (int)std::max<int64_t>(
      1, std::min<int64_t>(tiles, (int64_t)per_sm * num_sms() / ps.split));
}

}  // namespace

bool colpair_step_applies(const DeviceCSR& H, int NR, int dot) {
  return NR <= cols_per_launch() &&
         select_colpair_step(NR, dot, H.is_real != 0, H.ell_w, H.max_row_nnz, H.n).fn != nullptr;
}

void launch_columns(int64_t NH, int ncols, int precision, int dot, bool pairs, int* held, int* cpl) {
  *cpl = 1;
  if (pairs) {
    *held = ncols <= 2 ? ncols : ncols <= 4 ? 4 : (ncols + 7) / 8 * 8;
    return;
  }
  const Shape s = pick_shape(ncols, precision, dot, NH);
  const int width = s.lpr * s.cpl;
  *held = (ncols + width - 1) / width * width;
  *cpl = s.cpl;
}

bool packed_step_applies(const DeviceCSR& H, int NR, int dot) {
  return NR <= cols_per_launch() &&
         select_packed_step(NR, dot, H.is_real != 0, H.max_row_nnz, H.ell_w, H.n).fn != nullptr;
}

namespace {

// The kernel of the step `a` for a launch of ncols columns.
int choose_step(const StepArgs& a, int precision, int ncols, StepChoice* out) {
  const DeviceCSR& H = *a.H;
  auto take = [&](KernelFn fn, int lpr) {
    *out = StepChoice{fn, grid_for(fn, a.NH, lpr)};
    return KPMGB_OK;
  };
  const bool real = H.is_real != 0;
  // Calls in the standard layout.  Automatic selection for real operators with
  // 33..64 columns per launch (bra-ket moments): the row-streaming kernel when
  // rows hold at most 8 nonzeros, else the padded-row kernel; elsewhere the CSR
  // kernel (L2-resident 2D Anderson L = 64, 12 columns, 7.4 ms per call against
  // the padded rows' 8.3).
  if (a.colpair) {
    // the call keeps its vectors in the column-pair layout: only the
    // column-pair kernel reads them
    const PackedStep ps = precision == KPMGB_PREC_FF
                              ? select_colpair_step(ncols, a.dot, real, H.ell_w, H.max_row_nnz,
                                                    a.NH)
                              : PackedStep{};
    if (!ps.fn) return fail(KPMGB_ERR_CUDA, "internal: column-pair layout without its kernel");
    *out = StepChoice{ps.fn, grid_for(ps.fn, a.NH, kThreads / ps.rows_per_block, ps.split),
                      ps.threads, 0, ps.split};
    return KPMGB_OK;
  }
  if (a.paired) {
    // the call keeps its vectors in the paired layout: only the packed
    // kernel reads them
    const PackedStep ps = precision == KPMGB_PREC_FF
                              ? select_packed_step(ncols, a.dot, real, H.max_row_nnz, H.ell_w, a.NH)
                              : PackedStep{};
    if (!ps.fn) return fail(KPMGB_ERR_CUDA, "internal: paired layout without the packed kernel");
    *out = StepChoice{ps.fn, grid_packed(ps, a.NH), ps.threads, 0, ps.split};
    return KPMGB_OK;
  }
  if (a.variant == 11 && precision != KPMGB_PREC_FF)
    return fail(KPMGB_ERR_ARGUMENT, "the row-streaming kernel is float-float only");
  // the row-streaming kernels leave out Im<x|y> of the doubling dots (0 for a
  // Hermitian H)
  const bool streaming =
      a.variant == 11 || (a.variant == 0 && (H.hermitian || a.dot != DOT_DOUBLING));
  if (precision == KPMGB_PREC_FF && streaming) {
    if (KernelFn fr = select_kernel_ffr(ncols, a.dot, real, H.max_row_nnz, H.ell_w))
      return take(fr, 32);
    KernelFn fc = H.ell_w > 0 && (kStreamingComplex || a.variant == 11)
                      ? select_kernel_ffc(ncols, a.dot, real, H.ell_w, H.max_row_nnz)
                      : nullptr;
    if (fc) return take(fc, ffc_lanes(ncols));
    if (a.variant == 11)
      return fail(KPMGB_ERR_ARGUMENT,
                  "the row-streaming kernels serve float-float steps of real operators with "
                  "33..64 columns and rows of 5..8 nonzeros, and of complex operators with "
                  "9..32 columns and rows of 5..12 nonzeros");
  }
  const bool auto_padded =
      a.variant == 0 && H.ell_w > 0 && ((real && ncols > 32) || padded_complex());
  if (precision == KPMGB_PREC_FF && (a.variant == 9 || auto_padded)) {
    KernelFn fe = H.ell_w > 0 ? select_kernel_ffe(ncols, a.dot, real) : nullptr;
    if (fe) return take(fe, ffe_lanes(ncols));
    if (a.variant == 9)
      return fail(KPMGB_ERR_ARGUMENT, "the padded-row kernel serves float-float steps with 5..64 "
                                      "columns and rows of at most 16 nonzeros");
  }
  const Shape sh = shape_for(a, ncols, precision);
  const int width = sh.lpr * sh.cpl;
  out->fn = select_kernel(sh, precision, a.dot, real);
  out->split = (ncols + width - 1) / width;
  if (precision == KPMGB_PREC_FF && sh.cpl > 2) out->batch = 1;
  out->grid = grid_for(out->fn, a.NH, sh.lpr, out->split);
  if (a.max_grid > 0) out->grid = std::min(out->grid, a.max_grid);
  // The FP64 step of a complex operator is bound by each SM's FP64 pipe.  A
  // grid that leaves some of the resident slots free, but fewer than it needs,
  // gets its successor's first blocks all on the SMs with those slots when
  // they are launched early: such grids launch one after another (Haldane
  // 101x87, NR = 5: 18.5 us per step against 22.3; 150x80, NR = 11: 35.0
  // against 43.3), the others early (64x64, NR = 8: 2.7 us less per step).
  if (precision == KPMGB_PREC_FP64 && !real) out->slots = blocks_per_sm(out->fn) * num_sms();
  return KPMGB_OK;
}

int last_column(const StepArgs& a) { return a.c1 > 0 ? a.c1 : a.NR; }

int num_dots(int dot) { return dot == DOT_NONE ? 0 : (dot == DOT_LR1 ? 1 : 2); }

size_t partials_count(const StepArgs& a, const StepChoice& c, int ncols) {
  return (size_t)c.grid * num_dots(a.dot) * ncols;
}

// A block adds the per-block sums of one step for up to 32 of its entries
// (dot, column): the blocks in P interleaved parts of 4 accumulators each,
// then the parts, always in the same order.
struct FinishParams {
  const double2* partials;
  int64_t stride;  // double2 elements from step to step
  int G;           // blocks per step
  int nd, ncols, c0, ld;
  MomentArgs m;
};

__global__ void __launch_bounds__(256) k_finish_moments(FinishParams f) {
  __shared__ double2 part[256];
  const int ne = f.nd * f.ncols;
  const int e0 = blockIdx.y * 32;
  const int E = min(32, ne - e0);
  const int P = 256 / E;
  const int q = threadIdx.x / E, e = threadIdx.x % E;
  const double2* src = f.partials + (int64_t)blockIdx.x * f.stride + e0 + e;
  if (q < P) {
    double2 a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = make_double2(0.0, 0.0);
    for (int b = q; b < f.G; b += 4 * P) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (b + k * P < f.G) {
          const double2 v = src[(int64_t)(b + k * P) * ne];
          a[k].x += v.x;
          a[k].y += v.y;
        }
    }
    part[threadIdx.x] = make_double2((a[0].x + a[1].x) + (a[2].x + a[3].x),
                                     (a[0].y + a[1].y) + (a[2].y + a[3].y));
  }
  for (int w = 128; w > 0; w >>= 1) {
    __syncthreads();
    if (q < w && q + w < P) {
      part[threadIdx.x].x += part[threadIdx.x + w * E].x;
      part[threadIdx.x].y += part[threadIdx.x + w * E].y;
    }
  }
  if (q != 0) return;
  double2 s = part[e];
  const int k = (e0 + e) / f.ncols;
  const int cc = f.c0 + (e0 + e) % f.ncols;
  if (f.m.scale) {
    s.x *= f.m.scale[cc];
    s.y *= f.m.scale[cc];
  }
  if (f.m.mom == MOM_DOUBLING) {
    const double2 base = f.m.mu[(size_t)k * f.ld + cc];
    if (k == 0 && f.m.growth_limit > 0.0 && !(s.x <= f.m.growth_limit * base.x))
      atomicOr(f.m.status, (unsigned)STATUS_GROWTH);
    s.x = 2.0 * s.x - base.x;
    s.y = 2.0 * s.y - base.y;
  }
  f.m.mu[(size_t)(f.m.i0 + (int64_t)blockIdx.x * f.nd + k) * f.ld + cc] = s;
  if (!isfinite(s.x) || !isfinite(s.y)) atomicOr(f.m.status, (unsigned)STATUS_NONFINITE);
}

}  // namespace

int step_partials_bytes(const StepArgs& a, int precision, size_t* bytes) {
  *bytes = 0;
  const int W = cols_per_launch();
  for (int c0 = a.c0; c0 < last_column(a); c0 += W) {
    const int ncols = std::min(W, last_column(a) - c0);
    StepChoice c;
    KPMGB_TRY(choose_step(a, precision, ncols, &c));
    *bytes += partials_count(a, c, ncols) * sizeof(double2);
  }
  return KPMGB_OK;
}

namespace {

// Adds the per-block sums of nsteps steps like `a` (consecutive runs of
// step_partials_bytes at a.partials) in a fixed order and writes their moments.
int launch_finish_moments(const StepArgs& a, int precision, int nsteps, const MomentArgs& m,
                          cudaStream_t s) {
  size_t bytes = 0;
  KPMGB_TRY(step_partials_bytes(a, precision, &bytes));
  FinishParams f;
  f.partials = static_cast<const double2*>(a.partials);
  f.stride = (int64_t)(bytes / sizeof(double2));
  f.nd = num_dots(a.dot);
  f.ld = a.NR;
  f.m = m;
  const int W = cols_per_launch();
  for (int c0 = a.c0; c0 < last_column(a); c0 += W) {
    f.c0 = c0;
    f.ncols = std::min(W, last_column(a) - c0);
    StepChoice c;
    KPMGB_TRY(choose_step(a, precision, f.ncols, &c));
    f.G = c.grid;
    k_finish_moments<<<dim3((unsigned)nsteps, (unsigned)((f.nd * f.ncols + 31) / 32)), 256, 0,
                       s>>>(f);
    KPMGB_LAUNCHED();
    f.partials += partials_count(a, c, f.ncols);
  }
  return KPMGB_OK;
}

// The later steps of a recurrence: the doubling dots, or the one bra dot.
StepArgs later_step(StepArgs a, bool lr) {
  a.dot = lr ? DOT_LR1 : DOT_DOUBLING;
  a.alpha = 2.0;
  a.beta = -1.0;
  return a;
}

int64_t later_steps(int64_t NC, bool lr) { return lr ? NC - 2 : NC / 2 - 1; }

}  // namespace

int launch_steps(const StepArgs* steps, int n, int precision, cudaStream_t s) {
  for (int i = 0; i < n; ++i) {
    const StepArgs& a = steps[i];
    int e = 0;
    const double m = std::frexp(std::fabs(a.alpha), &e);
    if (!(m == 0.5) || !(a.beta == 0.0 || a.beta == -1.0))
      return fail(KPMGB_ERR_ARGUMENT,
                  "the recurrence step supports alpha = +-2^k and beta in {-1, 0}");
    if (precision == KPMGB_PREC_FF && !a.H->val_ff)
      return fail(KPMGB_ERR_ARGUMENT, "operator has no float-float values");
    if (a.dot != DOT_NONE && !a.partials)
      return fail(KPMGB_ERR_CUDA, "internal: a step with dots needs its partial sums");
  }
  const int W = cols_per_launch();
  const int end = last_column(steps[0]);
  double2* partials = static_cast<double2*>(steps[0].partials);  // steps with dots launch alone
  for (int c0 = steps[0].c0; c0 < end; c0 += W) {
    const int ncols = std::min(W, end - c0);
    StepChoice c;  // of the steps filled in so far
    KBatch batch;
    int held = 0;
    for (int i = 0; i < n; ++i) {
      const StepArgs& a = steps[i];
      const DeviceCSR& H = *a.H;
      StepChoice ci;
      KPMGB_TRY(choose_step(a, precision, ncols, &ci));
      if (held > 0 && (ci.fn != c.fn || ci.grid != c.grid || held >= c.batch)) {
        KPMGB_TRY(launch_step_kernel(c, held, s, batch));
        held = 0;
      }
      c = ci;
      KParams& p = batch.p[held++];
      p.rowptr = H.rowptr;
      p.col = H.col;
      p.val = precision == KPMGB_PREC_FF
                  ? H.val_ff
                  : (H.is_real ? (const void*)H.val_real : (const void*)H.val);
      p.NH = a.NH;
      p.ld = a.NR;
      p.c0 = c0;
      p.ncols = ncols;
      p.parts = c.split;
      p.x = a.x;
      p.z = a.z;
      p.y = a.y;
      p.bra = a.bra;
      p.alpha = a.alpha;
      p.partials = partials;
      p.blk = nullptr;
      p.vmax = a.vmax;
      p.ell_col = H.ell_col;
      p.ell_val = H.ell_val;
      p.ell_w = H.ell_w;
      p.alpha_f = (float)a.alpha;
      p.beta_mode = a.beta == 0.0 ? 0 : -1;
    }
    KPMGB_TRY(launch_step_kernel(c, held, s, batch));
    if (partials) partials += partials_count(steps[0], c, ncols);
  }
  return KPMGB_OK;
}

int launch_step(const StepArgs& a, int precision, cudaStream_t s) {
  return launch_steps(&a, 1, precision, s);
}

int launch_finish_sums(const double2* sums, int G, int nd, int NR, int64_t nsteps,
                       const MomentArgs& m, cudaStream_t s) {
  FinishParams f;
  f.partials = sums;
  f.stride = (int64_t)G * nd * NR;
  f.G = G;
  f.nd = nd;
  f.ncols = NR;
  f.c0 = 0;
  f.ld = NR;
  f.m = m;
  k_finish_moments<<<dim3((unsigned)nsteps, (unsigned)((nd * NR + 31) / 32)), 256, 0, s>>>(f);
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

int recurrence_scratch_bytes(const StepArgs& a0, int precision, int64_t NC, bool lr,
                             size_t* bytes, size_t* least) {
  // 32 MiB of block sums stay in L2 and cover 25 steps of the widest grids
  // and hundreds of the narrow ones, so that the finishing launch (a few us)
  // costs well under 1% of the steps it serves
  constexpr size_t kHeldBytes = size_t(32) << 20;
  StepArgs a = a0;
  a.dot = lr ? DOT_LR2 : DOT_DOUBLING;
  size_t first = 0, step = 0;
  KPMGB_TRY(step_partials_bytes(a, precision, &first));
  KPMGB_TRY(step_partials_bytes(later_step(a, lr), precision, &step));
  const size_t n = (size_t)std::max<int64_t>(1, later_steps(NC, lr));
  *bytes = std::max(first, step * std::max<size_t>(1, std::min(n, kHeldBytes / step)));
  if (least) {
    // one launch's columns at a time
    *least = 0;
    StepArgs b = later_step(a, lr);
    for (a.c0 = 0; a.c0 < a.NR; a.c0 = a.c1) {
      b.c0 = a.c0;
      a.c1 = b.c1 = std::min(a.c0 + cols_per_launch(), a.NR);
      KPMGB_TRY(step_partials_bytes(a, precision, &first));
      KPMGB_TRY(step_partials_bytes(b, precision, &step));
      *least = std::max(*least, std::max(first, step));
    }
  }
  return KPMGB_OK;
}

int launch_recurrence(StepArgs a, int precision, int64_t NC, bool lr, void* const (&slot)[2],
                      size_t held, MomentArgs m, cudaStream_t s) {
  // alpha_1 = H alpha_0 with mu_0, mu_1 (src/moment.jl:440-449, :521-527)
  a.dot = lr ? DOT_LR2 : DOT_DOUBLING;
  a.x = slot[0];
  a.z = nullptr;
  a.y = slot[1];
  a.alpha = 1.0;
  a.beta = 0.0;
  const double growth = m.growth_limit;
  m.mom = MOM_STORE;
  m.i0 = 0;
  m.growth_limit = 0.0;
  // a step and its moments at once, in parts of the columns whose sums fit
  auto step_alone = [&](StepArgs t) -> int {
    size_t bytes = 0;
    KPMGB_TRY(step_partials_bytes(t, precision, &bytes));
    const int W = bytes <= held ? t.NR : cols_per_launch();
    for (t.c0 = 0; t.c0 < t.NR; t.c0 = t.c1) {
      t.c1 = std::min(t.c0 + W, t.NR);
      KPMGB_TRY(launch_step(t, precision, s));
      KPMGB_TRY(launch_finish_moments(t, precision, 1, m, s));
    }
    return KPMGB_OK;
  };
  KPMGB_TRY(step_alone(a));
  // alpha_n = 2 H alpha_{n-1} - alpha_{n-2} in place: doubling moments
  // mu_{2n-2}, mu_{2n-1} (src/moment.jl:460-487), or mu_n = <psil|alpha_n>
  // (src/moment.jl:540-549)
  const int64_t later = later_steps(NC, lr);
  if (later < 1) return KPMGB_OK;
  StepArgs b = later_step(a, lr);
  char* const base = static_cast<char*>(a.partials);
  size_t step_bytes = 0;
  KPMGB_TRY(step_partials_bytes(b, precision, &step_bytes));
  const int64_t hold = std::max<int64_t>(1, std::min<int64_t>(later, (int64_t)(held / step_bytes)));
  m.mom = lr ? MOM_STORE : MOM_DOUBLING;
  m.i0 = 2;
  m.growth_limit = growth;
  int ip = 1;
  int64_t n = 0;
  for (int64_t i = 0; i < later; ++i) {
    b.partials = base + n * step_bytes;
    b.x = slot[ip];
    b.z = slot[ip ^ 1];
    b.y = slot[ip ^ 1];
    ip ^= 1;
    if (hold == 1) {
      KPMGB_TRY(step_alone(b));
      m.i0 += lr ? 1 : 2;
      continue;
    }
    KPMGB_TRY(launch_step(b, precision, s));
    if (++n == hold || i + 1 == later) {
      b.partials = base;
      KPMGB_TRY(launch_finish_moments(b, precision, (int)n, m, s));
      m.i0 += n * (lr ? 1 : 2);
      n = 0;
    }
  }
  return KPMGB_OK;
}

namespace {

// Moments of nsteps steps of every member from the sums of its blocks: one
// block per step and member, its blocks in P interleaved parts.
struct FinishMembers {
  const double2* partials;
  int64_t stride;  // double2 elements from step to step
  const int* first;
  int NR;
  int64_t NC;
  double2* mu;
  const double* scale;
  unsigned* status;
  int doubling;
  int64_t i0;
};

__global__ void __launch_bounds__(128) k_finish_members(FinishMembers f) {
  __shared__ double2 part[128];
  const int ne = 2 * f.NR;  // at most 64
  const int P = 128 / ne;
  const int q = threadIdx.x / ne, e = threadIdx.x % ne;
  const int b0 = f.first[blockIdx.y], b1 = f.first[blockIdx.y + 1];
  double2 a = make_double2(0.0, 0.0);
  if (q < P) {
    const double2* src = f.partials + (int64_t)blockIdx.x * f.stride + e;
    for (int b = b0 + q; b < b1; b += P) {
      const double2 v = src[(int64_t)b * ne];
      a.x += v.x;
      a.y += v.y;
    }
    part[threadIdx.x] = a;
  }
  __syncthreads();
  if (q != 0) return;
  for (int k = 1; k < P; ++k) {
    a.x += part[k * ne + e].x;
    a.y += part[k * ne + e].y;
  }
  const int k = e / f.NR, c = e % f.NR;
  if (f.scale) {
    a.x *= f.scale[c];
    a.y *= f.scale[c];
  }
  double2* mu = f.mu + (size_t)blockIdx.y * f.NC * f.NR;
  if (f.doubling) {
    const double2 base = mu[k * f.NR + c];
    a.x = 2.0 * a.x - base.x;
    a.y = 2.0 * a.y - base.y;
  }
  mu[(f.i0 + (int64_t)blockIdx.x * 2 + k) * f.NR + c] = a;
  if (!isfinite(a.x) || !isfinite(a.y)) atomicOr(f.status, (unsigned)STATUS_NONFINITE);
}

}  // namespace

bool packed_members_apply(const DeviceCSR& H, int NR) {
  return select_packed_members(NR, H.is_real != 0, H.max_row_nnz, H.ell_w, H.n).fn != nullptr;
}

int launch_member_recurrence(const DeviceCSR& H, int64_t NH, int NR, int64_t NC, void* slot0,
                             void* slot1, const MemberArgs& a, double2* mu, const double* scale,
                             unsigned* status, cudaStream_t s) {
  StepChoice c;
  const PackedStep ps = select_packed_members(NR, H.is_real != 0, H.max_row_nnz, H.ell_w, NH);
  c.fn = ps.fn;
  c.split = ps.split;
  if (!c.fn) return fail(KPMGB_ERR_CUDA, "internal: no packed step for these members");
  c.grid = a.nblk;
  void* const slot[2] = {slot0, slot1};
  KBatch batch;
  KParams& p = batch.p[0];
  p.rowptr = H.rowptr;
  p.col = H.col;
  p.val = H.val_ff;
  p.NH = NH;
  p.ld = NR;
  p.c0 = 0;
  p.ncols = NR;
  p.bra = nullptr;
  p.parts = c.split;
  p.blk = a.blk;
  p.vmax = nullptr;
  p.ell_col = H.ell_col;
  p.ell_val = H.ell_val;
  p.ell_w = H.ell_w;
  FinishMembers f;
  f.partials = static_cast<const double2*>(a.partials);
  f.stride = (int64_t)a.nblk * 2 * NR;
  f.first = a.first;
  f.NR = NR;
  f.NC = NC;
  f.mu = mu;
  f.scale = scale;
  f.status = status;
  const int64_t steps = NC / 2;
  const int64_t hold =
      std::max<int64_t>(1, (int64_t)(a.held / ((size_t)f.stride * sizeof(double2))));
  int64_t n = 0;
  f.i0 = 0;
  for (int64_t i = 0; i < steps; ++i) {
    // y = H x, then 2 H x - y in place; the first step's moments come before
    // those of the doubling identities that use them
    const bool first = i == 0;
    p.x = slot[i & 1];
    p.y = slot[(i & 1) ^ 1];
    p.z = first ? nullptr : p.y;
    p.alpha = first ? 1.0 : 2.0;
    p.alpha_f = first ? 1.f : 2.f;
    p.beta_mode = first ? 0 : -1;
    p.partials = static_cast<double2*>(a.partials) + n * f.stride;
    KPMGB_TRY(launch_step_kernel(c, 1, s, batch));
    if (++n == hold || first || i + 1 == steps) {
      f.doubling = first ? 0 : 1;
      for (int m0 = 0; m0 < a.nseg; m0 += 65535) {  // the grid's y limit
        FinishMembers g = f;
        g.first += m0;
        g.mu += (size_t)m0 * NC * NR;
        k_finish_members<<<dim3((unsigned)n, (unsigned)std::min(a.nseg - m0, 65535)), 128, 0,
                           s>>>(g);
        KPMGB_LAUNCHED();
      }
      f.i0 += 2 * n;
      n = 0;
    }
  }
  return KPMGB_OK;
}

int tune_step(const StepArgs& a0, int precision, DevBuf& partials, cudaStream_t s, int* variant,
              int* shape) {
  *variant = 1;
  *shape = 0;
  if (a0.NR > kMaxCols) return KPMGB_OK;  // several column batches: keep the default
  struct Cand {
    int variant, shape;
  };
  std::vector<Cand> cands;
  for (const Shape& c : candidate_shapes(a0.NR, precision, a0.dot, a0.NH)) cands.push_back({1, c.lpr * 10 + c.cpl});
  if (precision == KPMGB_PREC_FF && a0.H->ell_w > 0 &&
      select_kernel_ffe(a0.NR, a0.dot, a0.H->is_real != 0))
    cands.push_back({9, 0});
  if (precision == KPMGB_PREC_FF &&
      (select_kernel_ffr(a0.NR, a0.dot, a0.H->is_real != 0, a0.H->max_row_nnz, a0.H->ell_w) ||
       select_kernel_ffc(a0.NR, a0.dot, a0.H->is_real != 0, a0.H->ell_w, a0.H->max_row_nnz)))
    cands.push_back({11, 0});
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  KPMGB_CUDA(cudaEventCreate(&e0));
  cudaError_t ce = cudaEventCreate(&e1);
  if (ce != cudaSuccess) {
    cudaEventDestroy(e0);
    KPMGB_CUDA(ce);
  }
  float best = 0.f;
  int rc = KPMGB_OK;
  for (const Cand& c : cands) {
    StepArgs a = a0;
    a.variant = c.variant;
    a.shape = c.shape;
    size_t bytes = 0;
    if (step_partials_bytes(a, precision, &bytes) != KPMGB_OK ||
        partials.ensure(std::max(bytes, partials.bytes)) != KPMGB_OK) {
      clear_error();
      continue;
    }
    a.partials = partials.ptr;
    if (launch_step(a, precision, s) != KPMGB_OK) {
      clear_error();
      continue;
    }
    cudaEventRecord(e0, s);
    for (int r = 0; r < 3 && rc == KPMGB_OK; ++r) rc = launch_step(a, precision, s);
    cudaEventRecord(e1, s);
    if (rc != KPMGB_OK) break;
    if (cudaEventSynchronize(e1) != cudaSuccess) {
      rc = fail(KPMGB_ERR_CUDA, "autotuning: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (best == 0.f || ms < best) {
      best = ms;
      *variant = c.variant;
      *shape = c.shape;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

// ------------------------------------------------------------ block loading
namespace {

// Per-column squared norms of a column-major block (one block per column,
// fixed-order reduction).
__global__ void __launch_bounds__(256) k_colnorm2(const double2* __restrict__ psi, int64_t NH,
                                                  double* out) {
  const int c = blockIdx.x;
  const double2* col = psi + (int64_t)c * NH;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < NH; i += 256) {
    const double2 v = col[i];
    s = fma(v.x, v.x, s);
    s = fma(v.y, v.y, s);
  }
  __shared__ double red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double nrm = sqrt(red[0]);
    int e = 0;
    if (nrm > 0.0 && isfinite(nrm)) frexp(nrm, &e);
    // stored column = psi * 2^-e (norm in [0.5, 1)); moments carry 2^e
    out[c] = ldexp(1.0, e);
  }
}

// Column-major NH x NR -> row-major, FP64 (scale ignored) or float-float with
// the column scale 1/col_scale applied (an exact power of two).
template <bool FF>
__global__ void __launch_bounds__(256) k_transpose_in(const double2* __restrict__ psi, void* out,
                                                      int64_t NH, int NR,
                                                      const double* __restrict__ col_scale,
                                                      int layout) {
  __shared__ double2 tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (int k = ty; k < 32; k += 8) {
    const int c = c0 + k;
    const int64_t r = r0 + tx;
    double2 v = make_double2(0.0, 0.0);
    if (c < NR && r < NH) v = psi[(int64_t)c * NH + r];
    tile[k][tx] = v;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int64_t r = r0 + k;
    const int c = c0 + tx;
    // column pairs: the missing second column of an odd NR is stored as 0
    if (c < NR + (FF && layout == VEC_COLPAIR ? NR & 1 : 0) && r < NH) {
      const double2 v = tile[tx][k];
      if constexpr (FF) {
        const double f = c < NR ? 1.0 / col_scale[c] : 0.0;
        const float2 re = ff::split_double(v.x * f);
        const float2 im = ff::split_double(v.y * f);
        if (layout == VEC_COLPAIR) {
          const int half = (NR + 1) / 2, q = c % half, side = c / half;
          float* f = static_cast<float*>(out) + (r * half + q) * 8 + side;
          f[0] = re.x;
          f[2] = re.y;
          f[4] = im.x;
          f[6] = im.y;
        } else {
          static_cast<float4*>(out)[r * NR + c] = layout == VEC_PAIRED
                                                      ? make_float4(re.x, im.x, re.y, im.y)
                                                      : make_float4(re.x, re.y, im.x, im.y);
        }
      } else {
        static_cast<double2*>(out)[r * NR + c] = v;
      }
    }
  }
}

// All columns take the largest factor; the block factor is also stored at s[n].
__global__ void k_uniform_scale(double* s, int n) {
  double m = s[0];
  for (int i = 1; i < n; ++i) m = fmax(m, s[i]);
  for (int i = 0; i < n; ++i) s[i] = m;
  s[n] = m;
}

__global__ void k_scale_product(const double* a, const double* b, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] * b[i];
}

__global__ void k_copy2(const double2* src, double2* dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

}  // namespace

int launch_load_block(const void* psi, void* slot, int64_t NH, int NR, int precision,
                      double* col_scale, bool uniform, cudaStream_t s, int layout) {
  if (layout == VEC_COLPAIR && precision != KPMGB_PREC_FF)
    return fail(KPMGB_ERR_CUDA, "internal: column-pair layout needs float-float");
  const bool ff = precision == KPMGB_PREC_FF;
  if (ff) {
    k_colnorm2<<<NR, 256, 0, s>>>(static_cast<const double2*>(psi), NH, col_scale);
    KPMGB_LAUNCHED();
    if (uniform) {
      k_uniform_scale<<<1, 1, 0, s>>>(col_scale, NR);
      KPMGB_LAUNCHED();
    }
  }
  const int cols = layout == VEC_COLPAIR ? NR + (NR & 1) : NR;
  dim3 grid((unsigned)((NH + 31) / 32), (unsigned)((cols + 31) / 32));
  if (ff)
    k_transpose_in<true><<<grid, 256, 0, s>>>(static_cast<const double2*>(psi), slot, NH, NR,
                                              col_scale, layout);
  else
    k_transpose_in<false><<<grid, 256, 0, s>>>(static_cast<const double2*>(psi), slot, NH, NR,
                                               nullptr, VEC_STD);
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

int launch_scale_product(const double* sa, const double* sb, double* out, int NR,
                         cudaStream_t s) {
  k_scale_product<<<(NR + 255) / 256, 256, 0, s>>>(sa, sb, out, NR);
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

int launch_copy_moments(const double2* src, double2* dst, int64_t count, cudaStream_t s) {
  const int blocks = (int)std::min<int64_t>((count + 255) / 256, 1024);
  k_copy2<<<std::max(blocks, 1), 256, 0, s>>>(src, dst, count);
  KPMGB_LAUNCHED();
  return KPMGB_OK;
}

}  // namespace kpmgb
