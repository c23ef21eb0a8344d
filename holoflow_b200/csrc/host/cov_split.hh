// Split of the Gram matrices of a call over CTAs (host only: no CUDA in here).
#pragma once

#include <algorithm>
#include <cstdint>

namespace hf {

// CTAs per window of a call of `nwin` windows of `ntiles` pixel tiles: about two per SM over the whole
// call, at least one tile each.
inline int64_t cov_split(int sms, int64_t ntiles, int nwin) {
  return std::max<int64_t>(1, std::min<int64_t>((2LL * sms + nwin - 1) / nwin, ntiles));
}

// No call of 1 .. max_windows windows takes more CTAs than this: what a workspace made once for all of
// them has to hold.  The windows of a call times cov_split do not grow with the windows: at 148 SMs, 37
// windows of 64 tiles take 296 CTAs, 36 take 324.
inline int64_t cov_split_most(int sms, int64_t ntiles, int max_windows) {
  return std::min<int64_t>(2LL * sms + max_windows - 1, ntiles * max_windows);
}

} // namespace hf
