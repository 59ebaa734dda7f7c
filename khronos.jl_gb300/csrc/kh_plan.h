// How the step kernels split a grid among CTAs: z planes per CTA.  Plain functions
// of the grid and of how many CTAs the GPU holds at once (slots).
#pragma once

#include <algorithm>
#include <cmath>

namespace kh {

inline long long plan_tiles(int nx, int ny, int tile_x, int tile_y) {
  return (long long)((nx + tile_x - 1) / tile_x) * ((ny + tile_y - 1) / tile_y);
}

// General TMA-staged kernel (kh_tma.cu), which reads one curl-source plane more than
// it updates: 10 planes (a measured optimum on 128- and 256-plane grids: that halo
// plane against enough CTAs to balance the SMs), fewer when the launch would not fill
// two rounds of resident CTAs.  At the reduced-state kernel's depths, µs a step: FP32
// 160×160×96 with the CPU-path semantics 93.8, 89.5 at these; FP64 256×256×128 with σ 656
// and 634, 160×160×96 periodic with χ3 383 and 363.
inline int general_zplanes(int nz, long long tiles, int slots) {
  const long long fill = tiles * nz / (2LL * std::max(1, slots));
  return int(std::min<long long>(nz, std::max(2LL, std::min<long long>(10, fill))));
}

// CTAs that a launch can have along z.
constexpr int kMaxGridZ = 65535;

inline int reduced_zplanes_by_cost(int nz, long long tiles, int slots, bool fp64) {
  // FP64 is bound by arithmetic: the shallowest chunks balance best (240×144×96, 32
  // steps: 12.26 / 12.40 / 12.50 / 12.52 / 13.0 ms at 2 / 3 / 4 / 5 / 10 planes).
  if (fp64) return std::min(2, nz);
  // A plane costs a CTA about 1.4 µs whatever else runs, its start about three
  // planes; more rounds of CTAs cost less than their number (the SMs overlap them).
  // The optimum of that grows with the square root of the rounds at one plane per
  // CTA (320×192×128, 96 steps: 15.66 / 15.35 / 15.04 / 15.04 / 15.12 / 15.36 ms at 3 /
  // 4 / 5 / 6 / 7 / 10 planes; 200×200×64: 23.97 / 23.58 / 22.96 / 23.07 / 23.40 at 3 - 7).
  const double rounds = double(tiles) * nz / double(slots);
  auto ctas = [&](int z) { return tiles * ((nz + z - 1) / z); };
  const int best = int(std::max(2.0, std::min(7.0, std::floor(1.25 * std::sqrt(rounds) + 0.5))));
  const double many = (best + 3) * (1.15 + 0.3 * double(ctas(best)) / double(slots));
  // … unless all CTAs (but a few of the last, shorter ones) are resident at once at
  // a depth that costs clearly less (96³, 64 steps: 3.87 ms at 5 planes, 4.05 at 2;
  // 181×97×75, where it does not: 6.09 ms at 3 planes, 6.72 at 7).
  for (int z = 1; z <= 10; ++z) {
    const double r = double(ctas(z)) / double(slots);
    if (r > 1.06) continue;
    if ((z + 3) * (r > 1.0 ? 1.1 : 1.0) < 0.925 * many) return std::min(z, nz);
    break;
  }
  return std::min(best, nz);
}

// Reduced-state kernel (kh_lean.cu).
inline int reduced_zplanes(int nz, long long tiles, int slots, bool fp64) {
  return std::max(reduced_zplanes_by_cost(nz, tiles, slots, fp64), (nz + kMaxGridZ - 1) / kMaxGridZ);
}

}  // namespace kh
