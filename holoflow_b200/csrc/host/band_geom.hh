// Tile geometry of the FP32 band DFT (host only: no CUDA in here).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace hf {

constexpr int    kBandPX   = 4;   // pixels per thread
constexpr int    kBandThr  = 128; // threads per CTA
constexpr size_t kBandSmem = 220 * 1024;

// Bins per thread (even, at most 14), bin groups side by side, bins with the last group filled up, tiles
// of samples in shared memory (2: the next one streams in while one is summed) and the launch's shared
// memory.
struct BandGeom {
  int    NB, KG, nzpad, stages;
  size_t smem;
};

// A window of T frames of num / den bytes per sample and nz bins; smem > kBandSmem where no tile fits.
inline BandGeom band_geom(int T, int nz, int num, int den) {
  const int k  = (nz + 13) / 14; // bin groups
  BandGeom  g{};
  g.NB    = std::max(4, ((nz + k - 1) / k + 1) / 2 * 2);
  g.nzpad = (nz + g.NB - 1) / g.NB * g.NB;
  const auto bytes = [&](int KG, int stages) {
    return (size_t)stages * T * (kBandThr * kBandPX / KG) * num / den + (size_t)(T + 1) * g.nzpad * 8 + (size_t)T * 8;
  };
  // the fewest groups side by side (the largest tile) that leave three CTAs per SM, else the most; one
  // stage where two do not fit (28 bins of T = 256 float frames, 65536 pixels: 132 us, 1975 with a thread
  // per pixel; two stages just fit 65 bins of T = 128: 137 us against 2322)
  g.stages = 2;
  for (g.KG = 1; g.KG < 4 && bytes(g.KG, 2) > 74 * 1024;)
    g.KG *= 2;
  if (bytes(g.KG, 2) > kBandSmem)
    g.stages = 1;
  g.smem = bytes(g.KG, g.stages);
  return g;
}

} // namespace hf
