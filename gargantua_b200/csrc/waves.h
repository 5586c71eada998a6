// How the server's waves use the device's places: plain C++, no CUDA.
#pragma once

#include <cstdint>

namespace gg {

// Blocks of a Kerr kernel's grid that leave their places to the FP64 pass of
// the part before, where a request is marched in two waves. The pass needs
// one place for each 32 of its rays at a time and is done long before the
// wave if it gets a few: 1 in 550 (256 steps) to 670 (4096) of the first
// part's rays at every size. Lone requests, mean of three views, with 0, 20,
// 40, 60 and 100 places: 640x360 at 4096 steps 2074, 2043, 2042, 2083, 2044
// us; 960x540 at 256 1949, 1780, 1782, 1781, 1779; 1280x720 at 256 3067,
// 2922, 2826, 2859, 2889; 1920x1080 at 4096 7208, 6982, 6429, 6364, 6421;
// 2560x1440 at 4096 11686, 11553, 10825, 10862, 10971. Small requests do not
// miss 40 places, large ones gain nothing from more. Never more than an
// eighth of the grid: the rays need the rest.
constexpr uint32_t spare_blocks(uint32_t grid) { return grid / 8u < 40u ? grid / 8u : 40u; }

}  // namespace gg
