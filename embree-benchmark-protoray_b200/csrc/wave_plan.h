// How the paths of a render call are divided into waves (host code without CUDA).
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

} // namespace prt_b200
