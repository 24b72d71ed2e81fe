// What a launch's size alone decides: which form may store its samples, and in how many parts. Host arithmetic without
// CUDA, so that the sizes no test can render are checked all the same (tests/test_launch_plan.py).
#pragma once

#include <algorithm>
#include <cstdint>

namespace rtb
{
// A launch's stored samples (16 bytes each in float, 24 in double): at most 2 GiB, but for a wavefront's launch of one
// chunk, which is not divided
constexpr int64_t sample_budget_bytes = int64_t{2} << 30;
// A slot, and a path of the pool kernel, keeps its sample's number in 32 bits
constexpr bool samples_numbered(int64_t samples) { return samples < (int64_t{1} << 32); }

// Whether the pool kernel may take a bare small scene's launch (the persistent kernel renders it otherwise, whose scratch
// is 24 bytes a pixel and chunk): its samples fit the budget, so they are numbered too
constexpr bool bare_samples_fit(int64_t samples) { return samples <= sample_budget_bytes / 16; }

// What a samples buffer of `held` samples grows to for a launch of `count`: twice its size, so that launches of growing
// size reallocate a few times, but not beyond the budget for that
constexpr int64_t grown_samples(int64_t count, int64_t held)
{
    return std::max(count, std::min(2 * held, sample_budget_bytes / 16));
}

// A double launch's samples in bands of whole tiles (32 pixels of the padded image) one after another, each band with all
// of the launch's passes: a pixel's samples are added in one order whatever the bands. The pixels of a band, every band
// but the last: all of them where they fit the budget, else an even share that does (a tile at least).
constexpr int64_t band_pixels(int64_t padded_pixels, int64_t passes)
{
    const int64_t tiles = padded_pixels / 32;
    const int64_t most = std::max<int64_t>(1, sample_budget_bytes / (24 * 32 * passes));
    const int64_t bands = (tiles + most - 1) / most;
    return (tiles + bands - 1) / bands * 32;
}
} // namespace rtb
