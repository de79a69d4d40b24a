// Test driver for the host-side plan of the kpm_2d contractions
// (kpmgb_contract_plan.h).  Every input line is one call,
//   K NC arr_size right_block budget split sms
// (sizes 0: automatic); the output line is
//   KL KR range scratch largest fp64
// with `largest` the scratch that the call's blocks need at most (full and
// last left block, full and last right block) and `fp64` the FP64 kernel's alone.
#include <algorithm>
#include <cstdio>

#include "kpmgb_contract_plan.h"

int main() {
  long long K, NC, arr, right, budget;
  int split, sms;
  while (std::scanf("%lld %lld %lld %lld %lld %d %d", &K, &NC, &arr, &right, &budget, &split,
                    &sms) == 7) {
    const kpmgb::Kpm2dBlocks b =
        kpmgb::kpm2d_blocks(K, NC, arr, right, (size_t)budget, split != 0, sms);
    size_t largest = 0, fp64 = 0;
    if (b.KL > 0) {
      fp64 = kpmgb::contract_scratch_bytes(K, (int)std::min<long long>(b.KR, NC),
                                           (int)std::min<long long>(b.KL, NC), split != 0, 0, sms);
      for (long long nl : {std::min<long long>(b.KL, NC), NC % b.KL})
        for (long long nr : {std::min<long long>(b.KR, NC), NC % b.KR})
          if (nl > 0 && nr > 0)
            largest = std::max(largest, kpmgb::contract_scratch_bytes(K, (int)nr, (int)nl,
                                                                      split != 0, b.range, sms));
    }
    std::printf("%lld %lld %lld %zu %zu %zu\n", (long long)b.KL, (long long)b.KR, (long long)b.range,
                b.scratch, largest, fp64);
  }
  return 0;
}
