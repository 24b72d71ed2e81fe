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

// What a pool launch of an unknown view is taken to render a second, in samples: a first launch of that many seldom takes
// longer than asked for, and a short render is one launch, not a chunk to measure the speed and the rest (each launch ends
// with its last paths). A path is taken to be as long as it may, or 50 segments: measured on the B200, in segments a
// second, a closed white room of flat walls 33 G in float and 19 G in double, the same with 400 spheres 3.7 and 2.8 G,
// the 1.3M-triangle mesh 2.0 G, the second book's final scene 4.0 and 2.2 G; so the slowest, closed in, take at most 2.5
// times as long as asked for, whatever the depth.
constexpr double first_launch_speed(int max_depth, bool f64)
{
    return (f64 ? 3e9 : 5e9) / std::max(50, max_depth);
}

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
