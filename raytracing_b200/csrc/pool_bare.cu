// The bare small scenes' renders (flat-searched, no lights, textures, smoke or environment) by the pool kernel, with the
// roundings of the persistent kernel that otherwise renders them.
#include <cuda_runtime.h>

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
using rounds = rounds_bare;
#include "path.cuh"
#include "pool_kernel.cuh"
} // namespace

pool_program bare_pool_program() { return pool_program_of<false, false, true, false>(); }
} // namespace rtb
