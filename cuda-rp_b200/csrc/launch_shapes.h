// Launch shapes of the marching grid passes, as functions of the grid and the GPU.
#pragma once
#include <algorithm>
#include <climits>

namespace crp {

// Largest launch extent along y and z.
constexpr long kMaxGridYZ = 65535;

// Rows per chunk of the 2-D marching passes: of the numbers up to half the tuned one, that
// whose blocks (`warps` chunks each) take the least time in full waves of the `slots` blocks
// that the GPU holds, a chunk's start counted as two rows.  Per FDTD pass with 2, 3, 4, 6
// and 8 rows (us, the rule's choice in brackets): 600 x 701 12.8, [11.1], 12.7, 14.8, 16.1;
// 1001 x 1531 29.0, 27.0, [25.9], 26.1, 27.6; 1024 x 2048 with bubbles 43.7, 39.6, [40.7],
// 41.1, 47.0; 256 x 512 takes 11.7 with [1] and 13.0 with 2.
inline int march_rows(long Y, long strips, int tuned, int warps, long slots) {
  int best = 1;
  long least = LONG_MAX;
  for (int r = std::max(1, tuned / 2); r >= 1; r--) {
    const long chunks = (Y + r - 1) / r, blocks = strips * ((chunks + warps - 1) / warps);
    const long t = (blocks + slots - 1) / slots * (r + 2);
    if (t < least) least = t, best = r;
  }
  return best;
}

// Planes per chunk of the 3-D marching passes: up to 16 (256^3: 398 us, 425 with 32, 402
// with 8), fewer where that would leave less than two waves of the two blocks per SM that
// the GPU holds, more where the chunks would not fit a launch.  blocks: of one chunk.
inline int march3_planes(long Z, long blocks, int sms) {
  long planes = 16;
  while (planes > 2 && blocks * ((Z + planes - 1) / planes) < 4L * sms) planes /= 2;
  while ((Z + planes - 1) / planes > kMaxGridYZ) planes *= 2;
  return (int)planes;
}

}  // namespace crp
