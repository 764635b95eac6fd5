// wc_lanes.h — the slots of the lane passes and who takes them: how many there are, and when a lane takes two targets.
#pragma once
#include <cstdint>

namespace wc {

// The slots of the lane passes. Padded: every cell's particles start at a multiple of 4 and the
// places up to the next multiple hold PAD_POSITION in x, y and z, so that four consecutive slots
// are one aligned 16-byte load per coordinate and never belong to two cells. Packed: the sorted slots themselves; the
// passes mask the places of a load that lie outside a row of cells. The padded slots' total (known on the device,
// after the scan) decides: padded while it fits the capacity of 1.5 slots per particle. The dam breaks of 1,000 to
// 1,048,576 particles take 1.01 to 1.26 per particle over 2,000 steps, the reference's scene 1.07 to 1.11. In dilute
// states most of a cell's places would be padding, which every neighbour tests: with one particle per cell a step
// of 660,000 takes 195 us padded and 135 packed, of 2.5 M 645 and 455 (147 and 459 before there was padding).
// PAD_POSITION lies far beyond any kernel radius, with a finite squared distance (a padding place contributes
// 0 x finite = 0 to every sum, where an infinite one would contribute 0 x infinity).
constexpr float PAD_POSITION = 3e18f;
inline uint32_t slot_capacity(uint64_t n) { return (uint32_t)((n + n / 2u + 7u) & ~7ull) + 8u; }

// Whether the lane density pass over n particles takes the pairs of padded slots, which share every candidate load and
// loop step, or one target per lane, on `warps` resident warps: pairs halve the warps, so they need half a wave of pairs to
// lose nothing. A step in us, one target / pairs, at 4,864 warps (155,648 particles), alone and overlapped with those of two
// other streams: 130,000 69.6 / 71.7; 150,000 86.0 / 86.8 and 51.2 / 52.0; 165,000 85.0 / 84.2 and 53.5 / 50.6;
// 290,000 119.8 / 104.2 and 82.7 / 77.4; 365,000 147.8 / 148.6 and 107.8 / 102.3; 500,000 170.8 / 174.0 and
// 139.7 / 128.3; 560,000 184.9 / 177.6 and 152.6 / 138.7; 1,048,576 286.7 / 272.4.
inline bool lane_pairs(uint32_t n, uint32_t warps) { return n >= 32u * warps; }

// The same for the judge's passes, whose pairs leave a place for three quarters of `warps` (a rollout of two cycles in us,
// one / pairs: 150,000 639 / 647, 180,000 724 / 676, 230,000 774 / 728, 262,144 781 / 780, 300,000 849 / 877, 350,000
// 907 / 922, 380,000 918 / 910, 420,000 938 / 932, 700,000 1,257 / 1,202): not where a third of a second wave follows.
inline bool judge_pairs(uint32_t n, uint32_t warps) {
    const float waves = 1.05f * (float)n / (48.f * (float)warps);  // with the padding of a usual state
    return lane_pairs(n, warps) && !(waves > 1.3f && waves < 1.7f);
}

}  // namespace wc
