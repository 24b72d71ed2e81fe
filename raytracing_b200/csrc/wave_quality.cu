// The wavefront's shade kernel of a session under NEE/MIS without the second book's features (wave_shade.cuh). Its code
// outgrows the instruction cache (on the mesh a warp waits for instructions more than for memory), so compact code
// (path.cuh), and seven resident blocks instead of six to wait side by side: the 1.3M-triangle mesh 1920x1080 x 32 16.9
// -> 15.4 ms of its 45 on the B200, cornell-mis 600x600 x 64 19.7 -> 18.2 (six blocks 16.3 and 19.2, eight 15.4 and 18.3;
// inlined code 15.7 and 18.6 at best). A block's slots sorted by what they shade, through shared memory: 16.3 and 19.2.
#include <cuda_runtime.h>

#include <cstdint>

#include "ggx_energy_table.h"
#include "kernels.cuh"
#include "philox.cuh"
#include "rounding.cuh"
#include "rt_b200.h"

#define RTB_COMPACT_CODE
#define RTB_WAVE_SHADE_MIN_BLOCKS 7

namespace rtb
{
namespace
{
using rounds = rounds_session;
#include "path.cuh"
#include "wave_shade.cuh"
} // namespace

wave_shade_function quality_shade_kernel() { return wave_shade_kernel<true, false, false>; }
} // namespace rtb
