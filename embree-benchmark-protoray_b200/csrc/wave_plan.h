// How the paths of a render call are divided into waves and their camera rays
// traced (host code without CUDA).
#pragma once
#include <algorithm>

namespace prt_b200 {

// Items (pixels of all passes, rounded up to tiles) of one launch: its 32-bit
// counter also takes the requests of every lane past the end.
constexpr long long kMaxItems = 1LL << 30;

// Items of one pass of a frame: its 8x8 tiles.  A frame of more than kMaxFrameItems
// (one pixel wide or high) has no wave small enough for the counter.
constexpr long long kMaxFrameItems = (1LL << 31) - (1 << 20);
inline long long frame_items(int width, int height)
{
    return (long long)((width + 7) / 8) * ((height + 7) / 8) * 64;
}

// Paths of a wave: the setting (prt_tune::pathsPerWave), 0: the automatic size.
inline long long wave_paths(int setting, long long automatic)
{
    return std::min(setting > 0 ? (long long)setting : automatic, kMaxItems);
}

// Passes of a wave of at most `paths` paths, and the waves of `spp` passes.
inline int wave_passes(long long paths, long long perPass, int spp)
{
    return (int)std::max<long long>(1, std::min<long long>(spp, paths / perPass));
}
inline int wave_count(int spp, int passes) { return (int)(((long long)spp + passes - 1) / passes); }

// prt_tune::primaryPackets.
constexpr int kPrimaryAuto = 0, kPrimaryPackets = 1, kPrimaryIntervals = 2, kPrimaryLanes = 3;

// Without a setting, large waves of many passes take packets, which then span few
// pixels; smaller ones end in the longest packet.  A 1080p frame of 16 passes (two
// waves of 16.6M paths), per lane -> packets: 82K triangles 6.30 -> 5.87 ms, 1.38M
// 23.2 -> 21.5, 10.24M 16.7 -> 15.2, 2M in 2000 spheres 10.1 -> 9.9.  At 7.4M paths the
// last is 5% slower with packets, at 1.6M 40%.
// All waves of a call take what its full ones take: the last one runs beside the
// bounces of another chain, so its longest packet is not exposed (1080p, 12 passes
// as 8 and 4, 1.38M triangles: the 4 per lane 17.1 ms, as packets 16.3).
// Batches likewise, by their passes on average: 32 requests (156M paths) 28.0 -> 24.8 ms.
constexpr long long kPacketPaths = 81920;   // per SM
constexpr int kPacketPasses = 8;

// How a wave of `paths` paths over `pixels` pixels traces its camera rays: per lane
// (0) or as packets (kPrimaryPackets, kPrimaryIntervals).
inline int primary_packets(int setting, int numSMs, long long paths, long long pixels)
{
    if (setting == kPrimaryLanes) return 0;
    if (setting != kPrimaryAuto) return setting;
    return paths >= kPacketPaths * numSMs && paths >= kPacketPasses * pixels ? kPrimaryPackets : 0;
}

} // namespace prt_b200
