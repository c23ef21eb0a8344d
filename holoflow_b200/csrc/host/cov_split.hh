// Split of the Gram matrices of a call over CTAs (host only: no CUDA in here).
#pragma once

#include <algorithm>
#include <cstdint>

namespace hf {

// CTAs per window of a call of `nwin` windows of `ntiles` pixel tiles: two per SM over the whole call and
// no more, at least one tile each.  (Rounded up, 16 windows took 304 CTAs where 296 run at once, and so a
// second wave: 16 windows of 128 x 16384 8-bit pixels 318 us, 213 here.)
inline int64_t cov_split(int sms, int64_t ntiles, int nwin) {
  return std::max<int64_t>(1, std::min<int64_t>(2LL * sms / nwin, ntiles));
}

// No call of 1 .. max_windows windows takes more CTAs than this: what a workspace made once for all of
// them has to hold.  The windows of a call times cov_split do not grow with the windows: at 148 SMs, 33
// windows of 9 tiles take 264 CTAs, 32 take 288.
inline int64_t cov_split_most(int sms, int64_t ntiles, int max_windows) {
  return std::min<int64_t>(std::max<int64_t>(2LL * sms, max_windows), ntiles * max_windows);
}

} // namespace hf
