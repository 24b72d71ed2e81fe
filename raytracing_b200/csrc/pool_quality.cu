// A session's renders under NEE/MIS by the pool kernel (pool_kernel.cuh). Compact code: with the random numbers and the
// large spheres' quadratic called, cornell-mis 400x400 x 64 takes 6.65 ms instead of 7.62 on the B200, weekend under MIS
// 2.18 instead of 2.23, the final scene 7.31 instead of 8.02, smoke 1.95 instead of 1.89. (sincospif or atan2f called
// too gave more on one scene and lost as much on another; the books' kernels, whose code fits, lost 3 to 4%.)
#include <cuda_runtime.h>

#include <cstdint>

#include "ggx_energy_table.h"
#include "kernels.cuh"
#include "philox.cuh"
#include "rounding.cuh"
#include "rt_b200.h"

#define RTB_COMPACT_CODE

namespace rtb
{
namespace
{
using rounds = rounds_session;
#include "path.cuh"
#include "pool_kernel.cuh"
} // namespace

pool_program quality_pool_program(bool features, bool flat, bool mesh)
{
    if (features)
    {
        return flat ? pool_program_of<true, true, true, false>() : pool_program_of<true, true, false, false>();
    }
    if (flat)
    {
        return pool_program_of<true, false, true, false>();
    }
    return mesh ? pool_program_of<true, false, false, false, true>() : pool_program_of<true, false, false, false>();
}
} // namespace rtb
