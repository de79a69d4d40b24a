// Host-side plan of the kpm_2d contractions (mu += R L^H): tile shapes, K
// splits, K ranges and scratch sizes, and the block sizes of a kpm_2d call
// within its device budget.  Plain C++.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace kpmgb {

constexpr int TC_M = 128;  // A rows per tile

// Digit planes S per operand, B rows N per tile, K' elements KT per k-tile (a
// pipeline stage), k-tiles CHUNK per exact chunk, STAGES in shared memory.
template <int S, int N, int KT_, int CHUNK_, int STAGES_, int64_t MAXK>
struct PlaneCfg {
  static constexpr int kSlices = S;
  static constexpr int kN = N;
  static constexpr int KT = KT_;
  static constexpr int kChunk = CHUNK_;
  static constexpr int kStages = STAGES_;
  static constexpr uint32_t kATile = TC_M * KT * 2;  // one plane
  static constexpr uint32_t kBTile = N * KT * 2;
  static constexpr uint32_t kAStage = kATile * S;
  static constexpr uint32_t kBStage = kBTile * S;
  static constexpr uint32_t kStage = kAStage + kBStage;
  static constexpr int64_t kMaxKt = MAXK / KT;  // k-tiles per split: int64 headroom
  static constexpr int kAcc = S <= 5 ? 1 : 2;    // int64 accumulators per output
  // a row's entries are integers of scale 2^(kBits - e): |N| <= 2^kBits
  static constexpr int kBits = S == 5 ? 39 : 62;
  // value of plane 0's unit: 2^(e - kLead)
  static constexpr int kLead = kBits - 8 * (S - 1);
  static_assert(N * S <= 256 && (N * S) % 16 == 0 && N % 16 == 0,
                "one MMA covers up to S B planes");
  static_assert(KT % 16 == 0, "K steps of 16");
};
// Five digits (the split contraction): 40 KiB + 15 KiB per stage.
using Planes5 = PlaneCfg<5, 48, 32, 8, 4, (int64_t)1 << 24>;
// Eight digits (the double-precision contraction): 32 KiB + 8 KiB per stage.
using Planes8 = PlaneCfg<8, 32, 16, 8, 5, (int64_t)1 << 20>;

struct TcPlan {
  int mtiles, ntiles, nsplit;
  int64_t ktiles, kt_per_split;
  size_t a_bytes, b_bytes, exp_bytes, part_bytes;
};

template <class C>
TcPlan plan_for(int64_t K, int nr, int nl, int sms) {
  TcPlan pl;
  pl.mtiles = (nr + TC_M - 1) / TC_M;
  pl.ntiles = (2 * nl + C::kN - 1) / C::kN;
  pl.ktiles = (2 * K + C::KT - 1) / C::KT;
  const int64_t tiles = (int64_t)pl.mtiles * pl.ntiles;
  const int64_t S = sms;  // one CTA per SM (shared memory)
  const int64_t kmax = std::max<int64_t>(1, pl.ktiles / (4 * C::kChunk));
  int64_t want = std::max<int64_t>(1, (2 * S + tiles - 1) / tiles);
  want = std::min<int64_t>(want, kmax);
  // K splits: the count in [want, 4 want] (at most 8 S + tiles CTAs) whose
  // grid fills its last wave best, i.e. the least waves per unit of work
  // ceil(n tiles / S) / n; e.g. 64 tiles on 152 SMs: 19 splits (8 full
  // waves) instead of 5 (2.1 waves run as 3)
  int64_t best = want;
  double best_cost = 1e300;
  for (int64_t n = want; n <= std::min<int64_t>(4 * want, kmax); ++n) {
    if (n * tiles > 8 * S + tiles) break;
    const double cost = (double)((n * tiles + S - 1) / S) / (double)n;
    if (cost < best_cost * (1.0 - 1e-9)) {
      best_cost = cost;
      best = n;
    }
  }
  want = std::max(best, (pl.ktiles + C::kMaxKt - 1) / C::kMaxKt);
  pl.kt_per_split = (pl.ktiles + want - 1) / want;
  pl.kt_per_split = (pl.kt_per_split + C::kChunk - 1) / C::kChunk * C::kChunk;
  pl.kt_per_split = std::min(pl.kt_per_split, C::kMaxKt);
  pl.nsplit = (int)((pl.ktiles + pl.kt_per_split - 1) / pl.kt_per_split);
  pl.a_bytes = (size_t)pl.mtiles * pl.ktiles * C::kAStage;
  pl.b_bytes = (size_t)pl.ntiles * pl.ktiles * C::kBStage;
  pl.exp_bytes = ((size_t)(nr + nl) * sizeof(int) + 255) & ~size_t(255);
  pl.part_bytes = (size_t)pl.nsplit * nr * 2 * nl * sizeof(double);
  return pl;
}

// Partials of a plan, bounded over its sub-blocks: the split count times the
// tiles stays within 8 SMs + tiles and the split count within the K tiles of
// four chunks each, or it is the minimum that keeps a split within C::kMaxKt.
template <class C>
size_t part_bound_bytes(const TcPlan& pl, int sms) {
  const int64_t tiles = (int64_t)pl.mtiles * pl.ntiles;
  const int64_t nmin = (pl.ktiles + C::kMaxKt - 1) / C::kMaxKt;
  const int64_t kmax = std::max<int64_t>(1, pl.ktiles / (4 * C::kChunk));
  return (size_t)std::max<int64_t>(std::min<int64_t>(8 * sms + tiles, kmax * tiles), nmin * tiles) *
         TC_M * C::kN * sizeof(double);
}

inline size_t contract_align256(size_t b) { return (b + 255) & ~size_t(255); }

// ------------------------------------------------ split contraction (Planes5)
// The largest plan over sub-blocks nr' <= nr, nl' <= nl is the full block's
// (plane sizes grow with nr, nl; partials within part_bound_bytes).
inline size_t split_scratch_bytes(int64_t K, int nr, int nl, int sms) {
  const TcPlan pl = plan_for<Planes5>(K, nr, nl, sms);
  return pl.a_bytes + pl.b_bytes + 2 * pl.exp_bytes +
         std::max(pl.part_bytes, part_bound_bytes<Planes5>(pl, sms)) + 1024;
}

// ------------------------------------------------------------- FP64 kernel
constexpr int kSimtTile = 32;
// The double-precision contraction's device word at the start of its scratch
// (nonzero: its vectors need the FP64 kernel), padded to the planes' alignment.
constexpr size_t kContractGateBytes = 1024;

inline int64_t simt_tiles(int nr, int nl) {
  return (int64_t)((nr + kSimtTile - 1) / kSimtTile) * ((nl + kSimtTile - 1) / kSimtTile);
}

inline int simt_slices(int64_t K, int nr, int nl, int sms) {
  const int64_t tiles = simt_tiles(nr, nl);
  const int64_t want = (4LL * sms + tiles - 1) / tiles;
  const int64_t maxs = std::max<int64_t>(1, K / 1024);
  return (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, maxs), 64));
}

// Bound over every sub-block nr' <= nr, nl' <= nl that a launch may use:
// slices * nr' * nl' <= (4 * SMs / tiles' + 1) * tiles' * tile^2.
inline size_t simt_scratch_bytes(int64_t K, int nr, int nl, int sms) {
  const size_t bound = (4 * (size_t)sms + (size_t)simt_tiles(nr, nl)) * kSimtTile * kSimtTile;
  return std::max(bound, (size_t)simt_slices(K, nr, nl, sms) * nr * nl) * 16 + kContractGateBytes;
}

// ------------------------------------------------- eight planes (Planes8)
constexpr size_t kPlaneBytes = size_t(2) << 30;
constexpr int kStatChunk = 8192;      // complex elements per block of the statistics
constexpr size_t kVecStatBytes = 16;  // one block's statistics of a vector
constexpr int64_t kRangeChunk = Planes8::kChunk * Planes8::KT / 2;  // complex elements
// Chunks of the smallest K range: with 16, launches decide (Haldane 128x128, 4
// columns, 256 moments, 0.1 GiB: 1118 ms, FP64 kernel 422).
constexpr int64_t kMinChunks = 64;

// Scratch of the digit planes of an nr x nl block whose K elements are taken
// in ranges of `range`.  Every part grows with nr and nl, so a call sizes its
// scratch for its largest block and keeps one range for all of them.
struct Layout8 {
  TcPlan pl;
  int64_t range;
  int chunks;  // statistics blocks per vector
  size_t b, a, expB, expA, stat, gate, part, bytes;
};

inline Layout8 layout8(int64_t K, int nr, int nl, int64_t range, int sms) {
  Layout8 l;
  l.range = range;
  l.pl = plan_for<Planes8>(range, nr, nl, sms);
  l.chunks = (int)((K + kStatChunk - 1) / kStatChunk);
  l.gate = 0;
  l.b = kContractGateBytes;
  l.expB = l.b + contract_align256(l.pl.b_bytes);
  l.a = l.expB + contract_align256((size_t)nl * sizeof(int));
  l.expA = l.a + contract_align256(l.pl.a_bytes);
  l.stat = l.expA + contract_align256((size_t)nr * sizeof(int));
  l.part = l.stat + contract_align256((size_t)(nr + nl) * l.chunks * kVecStatBytes);
  l.bytes = l.part + std::max(l.pl.part_bytes, part_bound_bytes<Planes8>(l.pl, sms));
  return l;
}

// Complex elements per K range of blocks of at most nr x nl: planes of the size
// of the vectors themselves, but at least 64 MiB and at most kPlaneBytes, in
// whole exact chunks, no fewer than kMinChunks of them; 0 where those do not fit into
// `limit` bytes of scratch (the FP64 kernel takes the call).
inline int64_t contract_range(int64_t K, int nr, int nl, int sms, size_t limit) {
  const Layout8 one = layout8(K, nr, nl, kRangeChunk, sms);
  const size_t per_chunk = one.pl.a_bytes + one.pl.b_bytes;
  if (limit < one.bytes) return 0;
  const size_t whole = (size_t)((K + kRangeChunk - 1) / kRangeChunk) * per_chunk;
  const size_t most = std::min<size_t>(
      kPlaneBytes,
      std::max<size_t>({(size_t)64 << 20, (size_t)K * (nr + nl) * 16, whole / 8}));
  // what the other parts leave: those of one chunk first, then those of the
  // range that this allows (they grow with it)
  int64_t chunks = 1;
  for (int pass = 0; pass < 2; ++pass) {
    const Layout8 l = layout8(K, nr, nl, chunks * kRangeChunk, sms);
    const size_t other = l.bytes - l.pl.a_bytes - l.pl.b_bytes;
    if (limit < other) return 0;
    chunks = std::max<int64_t>((int64_t)(std::min(most, limit - other) / per_chunk), kMinChunks);
  }
  const int64_t range = chunks * kRangeChunk;
  // equal ranges: the tiles of a short last one would leave SMs idle
  const int64_t n = (K + range - 1) / range;
  const int64_t equal =
      std::min(K, ((K + n - 1) / n + kRangeChunk - 1) / kRangeChunk * kRangeChunk);
  return layout8(K, nr, nl, equal, sms).bytes <= limit ? equal : 0;
}

// ---------------------------------------------------------- kpm_2d blocks
struct Kpm2dBlocks {
  int64_t KL = 0, KR = 0;  // left and right blocks (0: the budget holds none)
  int64_t range = 0;       // K range of the digit planes (0: the FP64 kernel)
  size_t scratch = 0;      // bytes of contraction scratch
};

// Scratch of the contraction of KR x KL blocks.
inline size_t contract_scratch_bytes(int64_t K, int nr, int nl, bool split, int64_t range, int sms) {
  if (split) return split_scratch_bytes(K, nr, nl, sms);
  const size_t simt = simt_scratch_bytes(K, nr, nl, sms);
  return range > 0 ? std::max(simt, layout8(K, nr, nl, range, sms).bytes) : simt;
}

// Block sizes of a kpm_2d call of K complex elements per vector and NC moments
// a side: explicit sizes are honoured (results are blocking invariant);
// otherwise both chains stay resident when the budget allows it with the FP64
// kernel's scratch (src/moment.jl:759-810 for the reference's rule).  The digit
// planes take what the budget has left beside the blocks.  A blocked call
// gives a quarter of its budget to them (more where their smallest form needs
// it, less where they want less) if that costs no more than a third of the left
// block: Haldane 256x256, 8 columns, 256 moments in 1 GiB 971 ms, a sixteenth
// 1142, the FP64 kernel with the whole left block 2208; in 4 GiB 365, 480 and
// 1163; 128x128, 4 columns in 0.2 GiB 150, 268 and 268.  With both sizes
// explicit the budget bounds nothing.
inline Kpm2dBlocks kpm2d_blocks(int64_t K, int64_t NC, int64_t arr_size, int64_t right_block,
                                size_t budget, bool split, int sms) {
  Kpm2dBlocks b;
  const size_t block = (size_t)K * 16;
  const bool fixed = arr_size > 0 && right_block > 0;
  b.KL = arr_size;
  b.KR = right_block;
  if (!fixed) {
    const int64_t kr = std::min(b.KR ? b.KR : NC, NC);
    const size_t full = (size_t)(NC + (b.KR ? b.KR : NC) + 4) * block +
                        contract_scratch_bytes(K, (int)kr, (int)NC, split, 0, sms);
    if (full <= budget) {
      if (!b.KR) b.KR = NC;
      if (!b.KL) b.KL = NC;
    } else {
      if (!b.KR) b.KR = std::min<int64_t>(NC, 16);
      if (!b.KL) {
        const int64_t base = (b.KR + 7) * (int64_t)block;
        const int64_t per_left = (int64_t)block + b.KR * 16;
        const int64_t kl = ((int64_t)budget - base) / per_left;
        if (kl < 2) return Kpm2dBlocks{};
        b.KL = std::min<int64_t>(kl, NC);
        if (!split) {
          const int nr = (int)std::min(b.KR, NC), nl = (int)b.KL;
          auto bytes = [&](int64_t range) { return layout8(K, nr, nl, range, sms).bytes; };
          const size_t keep = std::max(bytes(std::min(K, kMinChunks * kRangeChunk)),
                                       std::min(bytes(contract_range(K, nr, nl, sms, SIZE_MAX)),
                                                budget / 4));
          const int64_t less =
              keep < budget ? (int64_t)((budget - keep) / block) - b.KR - 4 : 0;
          if (less < b.KL && less >= 2 && 3 * less >= 2 * b.KL) b.KL = less;
        }
      }
    }
  }
  const int nl = (int)std::min<int64_t>(b.KL, NC), nr = (int)std::min<int64_t>(b.KR, NC);
  if (!split) {
    const size_t held = (size_t)(nl + nr + 4) * block;
    b.range = contract_range(K, nr, nl, sms, fixed ? SIZE_MAX : budget > held ? budget - held : 0);
  }
  b.scratch = contract_scratch_bytes(K, nr, nl, split, b.range, sms);
  return b;
}

}  // namespace kpmgb
