// A batch's groups of books' jobs by the pool kernel, each sample with its job's scene and
// camera; the roundings are a session's, so a job's image is its session's.
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

pool_program batch_program(bool flat, bool features)
{
    if (flat)
    {
        return features ? pool_program_of<false, true, true, true>() : pool_program_of<false, false, true, true>();
    }
    return features ? pool_program_of<false, true, false, true>() : pool_program_of<false, false, false, true>();
}
} // namespace

cudaError_t launch_pool_batch(const wave_batch& w, bool flat, bool features, float4* samples, int64_t sample_count, int grid,
                              cudaStream_t stream)
{
    const pool_launch l = pool_launch_of(sample_count, grid);
    const pool_run run{samples, sample_count, l.claim, 0};
    if (const cudaError_t e = prepare_pool(w.work_counter, stream); e != cudaSuccess)
    {
        return e;
    }
    const pool_program program = batch_program(flat, features);
    program.kernel<<<l.blocks, render_block, static_cast<size_t>(program.shared), stream>>>(launch_params{}, run, w);
    return cudaGetLastError();
}

cudaError_t pool_batch_attributes(bool flat, bool features, kernel_attributes& out)
{
    const pool_program program = batch_program(flat, features);
    return pool_program_attributes(program, out);
}
} // namespace rtb
