"""What a launch's size alone decides (raytracing_b200/csrc/launch_plan.h), compiled here with g++ and checked over sizes
that no test can render.

* A path keeps its sample's number in 32 bits: a bare scene's launch that the pool kernel takes, and every band of a
  double launch, has fewer than 2^32 samples, whatever the image (up to 2^31 pixels) and the passes; a wavefront's launch
  of 2^32 samples or more is refused.
* The stored samples of either stay within 2 GiB, a buffer grown by doubling too.
* A first launch of an unknown view is planned by its paths' longest, so its length in time does not grow with the depth.
* A double launch's bands are whole tiles, cover the image, and are one where the samples fit.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent

CHECK = r"""
#include <cstdio>
#include <random>
#include "launch_plan.h"

int main()
{
    using namespace rtb;
    std::mt19937_64 gen(11);
    long long wrong = 0, checked = 0, refused = 0, banded = 0, whole = 0;
    auto check = [&](int64_t width, int64_t height, int64_t passes) {
        ++checked;
        const int64_t padded = (width + 7) / 8 * ((height + 3) / 4) * 32;
        const int64_t samples = padded * passes;
        wrong += bare_samples_fit(samples) && !(samples_numbered(samples) && samples * 16 <= (int64_t{2} << 30));
        wrong += !bare_samples_fit(samples) && samples * 16 <= (int64_t{2} << 30);
        wrong += samples_numbered(samples) != (samples < 4294967296ll);
        refused += !samples_numbered(samples);
        if (passes * 24 * 32 > (int64_t{2} << 30)) { return; } // a tile alone is beyond the budget: no launch is planned so
        const int64_t band = band_pixels(padded, passes);
        wrong += band < 32 || band % 32 != 0 || band > padded || band * passes * 24 > (int64_t{2} << 30);
        wrong += !samples_numbered(band * passes);
        int64_t covered = 0;
        for (int64_t first = 0; first < padded; first += band) { covered += std::min(band, padded - first); }
        wrong += covered != padded;
        wrong += samples * 24 <= (int64_t{2} << 30) && band != padded;
        wrong += samples * 24 > (int64_t{2} << 30) && band == padded;
        (band < padded ? banded : whole) += 1;
    };
    for (int i = 0; i < 20000; ++i)
    {
        // a buffer grown from launch to launch: it holds the launch, and more than 2 GiB only where the launch does
        int64_t held = 0;
        for (int k = 0; k < 8; ++k)
        {
            const int64_t count = 1 + static_cast<int64_t>(gen() >> (24 + gen() % 30));
            held = count > held ? grown_samples(count, held) : held;
            wrong += held < count;
            if (count * 16 > (int64_t{2} << 30)) { break; }
            wrong += held * 16 > (int64_t{2} << 30);
        }
    }
    for (int64_t p : {1, 2, 15, 16, 32, 4096})
    {
        for (int64_t w : {1, 8, 9, 256, 1920, 3840, 7680, 16383, 16384, 16400, 30000, 46300})
        {
            for (int64_t h : {1, 3, 4, 5, 1080, 2160, 16384, 16400, 46300}) { check(w, h, p); }
        }
    }
    for (int i = 0; i < 20000; ++i)
    {
        const int64_t w = 1 + static_cast<int64_t>(gen() % 46300), h = 1 + static_cast<int64_t>(gen() % 46300);
        check(w, h, 1 + static_cast<int64_t>(gen() % 64));
    }
    for (const bool f64 : {false, true})
    {
        // a first launch's segments a second never above what the slowest measured scenes make, times 2.5
        for (int depth : {0, 1, 50, 51, 1000, 10000, 2147483647})
        {
            wrong += first_launch_speed(depth, f64) * std::max(depth, 1) > (f64 ? 2.2e9 : 2.0e9) * 2.5;
        }
        wrong += first_launch_speed(50, f64) != first_launch_speed(1, f64) || first_launch_speed(5000, f64) * 100 != first_launch_speed(50, f64);
    }
    std::printf("%lld %lld %lld %lld %lld\n", checked, wrong, refused, banded, whole);
    return wrong == 0 ? 0 : 1;
}
"""


def test_every_launchs_samples_are_numbered_and_within_the_budget(tmp_path):
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no g++")
    source = tmp_path / "check.cpp"
    source.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([compiler, "-std=c++20", "-O2", "-I", str(REPO / "raytracing_b200" / "csrc"), str(source), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    checked, wrong, refused, banded, whole = map(int, r.stdout.split())
    assert r.returncode == 0 and wrong == 0
    assert checked > 20000 and refused > 100 and banded > 1000 and whole > 100
