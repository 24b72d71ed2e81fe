// A session's renders by the pool kernel (pool_kernel.cuh): the kernels' instantiations and their launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ggx_energy_table.h"
#include "kernels.cuh"
#include "philox.cuh"
#include "rounding.cuh"
#include "rt_b200.h"

namespace rtb
{
namespace
{
using rounds = rounds_session;
#include "path.cuh"
#include "pool_kernel.cuh"

__global__ void pool_prepare_kernel(unsigned long long* work_counter) { *work_counter = 0ull; }

pool_program program_for(const scene_view& scene, bool quality)
{
    const bool flat = scene.flat != 0;
    const bool features = has_features(scene);
    if (!wavefront_suits(scene))
    {
        return bare_pool_program();
    }
    if (quality)
    {
        return quality_pool_program(features, flat, scene.prim_count > scene.triangle_base);
    }
    if (flat)
    {
        return features ? pool_program_of<false, true, true, false>() : pool_program_of<false, false, true, false>();
    }
    return features ? pool_program_of<false, true, false, false>() : pool_program_of<false, false, false, false>();
}
} // namespace

cudaError_t prepare_pool(unsigned long long* work_counter, cudaStream_t stream)
{
    pool_prepare_kernel<<<1, 1, 0, stream>>>(work_counter);
    return cudaGetLastError();
}

cudaError_t pool_program_attributes(const pool_program& program, kernel_attributes& out)
{
    const auto* const kernel = reinterpret_cast<const void*>(program.kernel);
    if (const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, program.shared);
        e != cudaSuccess)
    {
        return e;
    }
    return function_attributes(kernel, out, program.shared);
}

// A launch of fewer samples than lanes spreads them over the warps, so that every multiprocessor takes part
pool_launch pool_launch_of(int64_t sample_count, int grid)
{
    constexpr int64_t block_warps = render_block / 32;
    const int64_t warps = grid * block_warps;
    const int64_t claim = std::clamp<int64_t>((sample_count + warps - 1) / warps, 1, 32);
    const int64_t blocks = std::min<int64_t>(grid, (sample_count + claim * block_warps - 1) / (claim * block_warps));
    return {static_cast<int32_t>(claim), static_cast<unsigned>(std::max<int64_t>(blocks, 1))};
}

cudaError_t launch_pool(const launch_params& p, bool quality, float4* samples, int64_t sample_count, int grid,
                        cudaStream_t stream)
{
    const pool_launch l = pool_launch_of(sample_count, grid);
    const pool_run run{samples, sample_count, l.claim, 0};
    if (const cudaError_t e = prepare_pool(p.work_counter, stream); e != cudaSuccess)
    {
        return e;
    }
    const pool_program program = program_for(p.scene, quality);
    program.kernel<<<l.blocks, render_block, static_cast<size_t>(program.shared), stream>>>(p, run, wave_batch{});
    return cudaGetLastError();
}

cudaError_t pool_attributes(const scene_view& scene, bool quality, kernel_attributes& out)
{
    const pool_program program = program_for(scene, quality);
    return pool_program_attributes(program, out);
}
} // namespace rtb
