// The path-tracing kernels for sm_100a.
//
// One persistent kernel renders a launch: a grid of (multiprocessors x resident blocks) threads, each of which takes
// work items (a pixel and a chunk of its passes) from a global counter, traces their samples one after another, and
// starts the next sample the moment one ends (path regeneration), so a warp's lanes stay busy however uneven the
// paths are. The lanes that need new work in an iteration claim it together: a ballot over the warp, one atomicAdd
// by its leader for the whole batch, and each lane's item from the prefix count of the ballot below it. Each item's
// sum goes to its own slot of a partials buffer, and a second kernel adds the slots to the pixels' sums in chunk
// order, so the image does not depend on which thread rendered what.
//
// The estimators are the reference's: the books' strategies (src/gpu/camera.cuh:304-437 diffuse_bounce, trace_ray;
// material.cuh:84-126 scatter; lights.cuh:49-227 the lights list) and the quality kernel's NEE with MIS
// (quality_path.cuh:61-188, light_sampler.cuh:40-103, lamps.cuh:81-146, mis.cuh:30-62). What differs is the B200 form:
// a 64-byte node holding both children's boxes, a flat search for small scenes, counter-based random numbers that
// depend only on (seed, pixel, pass, depth, dimension), work items instead of one thread per pixel, and FP64 only for
// a large sphere's quadratic and for the per-pixel sums.
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "ggx_energy_table.h"
#include "kernels.cuh"
#include "philox.cuh"
#include "rounding.cuh"
#include "rt_b200.h"

namespace rtb
{
namespace
{
using rounds = rounds_compiler;
#include "path.cuh"
#include "wave_shade.cuh"

// FEATURES: the scene has moving spheres, textures other than solid colors, or smoke (the counting build always
// compiles them in)
template <bool QUALITY, bool COUNT, bool FLAT, bool FEATURES>
__global__ void __launch_bounds__(render_block, render_min_blocks<QUALITY, FLAT, FEATURES>())
    render_kernel(const __grid_constant__ launch_params P)
{
    __shared__ unsigned long long block_rays;
    __shared__ unsigned long long block_shadow_rays;
    if (threadIdx.x == 0)
    {
        block_rays = 0;
        block_shadow_rays = 0;
    }
    __syncthreads();

    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    const camera_params& cam = P.cam;

    uint32_t rays = 0;
    uint32_t shadow_rays = 0;
    fetch_counts counts;
    bool need = true;
    bool start = false;
    int px = 0, py = 0;
    int64_t pass = 0, pass_end = 0;
    int64_t slot = 0;
    double acc_r = 0.0, acc_g = 0.0, acc_b = 0.0;
    sampler rng{};
    rng.job = P.job;
    path_state ps{};

    while (true)
    {
        // Claim work for the lanes that need it: one atomic per warp
        const unsigned active = __activemask();
        const unsigned needing = __ballot_sync(active, need);
        if (needing != 0u)
        {
            const int leader = __ffs(static_cast<int>(needing)) - 1;
            unsigned long long base = 0;
            if (static_cast<int>(lane) == leader)
            {
                base = atomicAdd(P.work_counter, static_cast<unsigned long long>(__popc(needing)));
            }
            base = __shfl_sync(active, base, leader);
            if (need)
            {
                const unsigned long long item = base + static_cast<unsigned long long>(__popc(needing & lanes_below));
                if (item >= static_cast<unsigned long long>(P.total_items))
                {
                    break; // no work left for this lane
                }
                const sample_place at = place_of(static_cast<int64_t>(item), cam, 0);
                const int64_t k = at.pass; // the item's chunk within the launch
                const int q = static_cast<int>(static_cast<int64_t>(item) - k * P.padded_pixels);
                px = at.x;
                py = at.y;
                if (px >= cam.width || py >= cam.height)
                {
                    continue; // a lane of a tile that hangs over the image's edge: nothing to render
                }
                const int64_t chunk_first = (P.first_chunk + k) * P.chunk;
                pass = chunk_first > P.pass_begin ? chunk_first : P.pass_begin;
                const int64_t chunk_end = chunk_first + P.chunk;
                pass_end = chunk_end < P.pass_end ? chunk_end : P.pass_end;
                slot = k * P.padded_pixels + q;
                acc_r = acc_g = acc_b = 0.0;
                rng.pixel = static_cast<uint32_t>(py) * static_cast<uint32_t>(cam.width) + static_cast<uint32_t>(px);
                need = false;
                start = true;
            }
        }
        if (start)
        {
            // A new sample: pass n is pass n % k^2 of round n / k^2, whose numbers come from seed + round * 2^32
            const int64_t round = round_of(pass, cam);
            const int in_round = static_cast<int>(pass - round * P.round_passes);
            const uint64_t key = P.seed + (static_cast<uint64_t>(round) << 32);
            rng.key = make_uint2(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32));
            rng.pass = static_cast<uint32_t>(in_round);
            const float4 u = rng.draw(0, 0);
            int s_i, s_j;
            stratum_of(cam, in_round, s_i, s_j);
            camera_ray(cam, px, py, s_i, s_j, u, ps.o, ps.d);
            // the moment in the shutter, in a scene where something moves (camera.ixx get_ray's ray time)
            ps.time = FEATURES && P.scene.has_motion ? rng.draw(0, block_time).x : 0.0f;
            ps.throughput = make_float3(1.0f, 1.0f, 1.0f);
            ps.radiance = make_float3(0.0f, 0.0f, 0.0f);
            ps.bsdf_pdf = 0.0f;
            ps.specular = true;
            ps.rays_left = cam.max_depth;
            ps.depth = 0;
            ps.from = -1;
            ps.inward = false;
            start = false;
        }

        // One segment: the closest event (a surface, or a particle of smoke before it), then the vertex's shading
        constexpr int search = FLAT ? search_flat : search_tree;
        hit_info h;
        traverse<false, COUNT, search, FEATURES>(P.scene, ps.o, ps.d, ps.time, infinity_f, ps.from, ps.inward, -1,
                                                 h, &counts);
        ++rays;
        ++ps.depth;
        if (FEATURES && P.scene.medium_count > 0)
        {
            media_event(P.scene, ps.o, ps.d, ps.time, rng, ps.depth, h);
        }
        float3 sample;
        const step_result r =
            QUALITY ? shade_quality<COUNT, search, FEATURES>(P.scene, cam, rng, ps, h, sample, shadow_rays, &counts)
                    : shade_books<FEATURES>(P.scene, cam, rng, ps, h, sample);
        if (r == step_result::done)
        {
            acc_r += without_nan(sample.x);
            acc_g += without_nan(sample.y);
            acc_b += without_nan(sample.z);
            if (++pass == pass_end)
            {
                double* out = P.partials + 3 * slot;
                out[0] = acc_r;
                out[1] = acc_g;
                out[2] = acc_b;
                need = true;
            }
            else
            {
                start = true;
            }
        }
    }
    if (COUNT)
    {
        atomicAdd(P.counters + 2, static_cast<unsigned long long>(counts.nodes));
        atomicAdd(P.counters + 3, static_cast<unsigned long long>(counts.spheres));
        atomicAdd(P.counters + 4, static_cast<unsigned long long>(counts.quads));
        atomicAdd(P.counters + 5, static_cast<unsigned long long>(counts.triangles));
    }
    atomicAdd(&block_rays, static_cast<unsigned long long>(rays));
    if (QUALITY)
    {
        atomicAdd(&block_shadow_rays, static_cast<unsigned long long>(shadow_rays));
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        atomicAdd(P.counters, block_rays);
        if (QUALITY)
        {
            atomicAdd(P.counters + 1, block_shadow_rays);
        }
    }
}

// Adds each pixel's chunk partials to its sums, in chunk order (the sums are plain doubles in HBM, 24 bytes a pixel)
__global__ void reduce_kernel(const reduce_params P)
{
    const int x = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    const int y = static_cast<int>(blockIdx.y);
    if (x >= P.width || y >= P.height)
    {
        return;
    }
    const int q = ((y >> 2) * P.tiles_x + (x >> 3)) * 32 + ((y & 3) << 3) + (x & 7);
    double* sum = P.sums + 3 * (static_cast<int64_t>(y) * P.width + x);
    double r = sum[0], g = sum[1], b = sum[2];
    for (int k = 0; k < P.chunks; ++k)
    {
        const double* part = P.partials + 3 * (static_cast<int64_t>(k) * P.padded_pixels + q);
        r += part[0];
        g += part[1];
        b += part[2];
    }
    sum[0] = r;
    sum[1] = g;
    sum[2] = b;
}

// ---- batched launches: many jobs (requests), each its own scene, camera and passes, in one persistent kernel ------

// The same loop as render_kernel, with the job of each work item looked up in the job table: the jobs' items follow
// each other in one item space, so the persistent threads pull work from every job at once, and a small job's tail
// fills with another's work. Each job may use either integrator. The jobs of flat scenes come first in the table and
// the item space, and each search has its own launch (FLAT: items [0, flat_items) of jobs [0, flat_jobs); otherwise
// the rest), compiled as render_kernel's for that search, so a job renders the same bits as its plain render.
template <bool FLAT, bool FEATURES>
__global__ void __launch_bounds__(render_block, render_min_blocks<true, FLAT, FEATURES>())
    render_batch_kernel(const batch_params P)
{
    constexpr int search = FLAT ? search_flat : search_tree;
    constexpr int group = batch_group(FLAT, FEATURES);
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    const int64_t item_begin = P.header->group_items[group];
    const int64_t total_items = P.header->group_items[group + 1];
    const int job_first = P.header->group_jobs[group];
    const int job_end = P.header->group_jobs[group + 1];
    unsigned long long* const work_counter = P.work_counter + group;

    uint32_t rays = 0;
    uint32_t shadow_rays = 0;
    bool need = true;
    bool start = false;
    int px = 0, py = 0;
    int64_t pass = 0, pass_end = 0;
    int64_t slot = 0;
    double acc_r = 0.0, acc_g = 0.0, acc_b = 0.0;
    const batch_job* J = nullptr;
    sampler rng{};
    path_state ps{};

    while (true)
    {
        const unsigned active = __activemask();
        const unsigned needing = __ballot_sync(active, need);
        if (needing != 0u)
        {
            const int leader = __ffs(static_cast<int>(needing)) - 1;
            unsigned long long base = 0;
            if (static_cast<int>(lane) == leader)
            {
                base = atomicAdd(work_counter, static_cast<unsigned long long>(__popc(needing)));
            }
            base = __shfl_sync(active, base, leader);
            if (need)
            {
                const auto item = item_begin + static_cast<int64_t>(base + __popc(needing & lanes_below));
                if (item >= total_items)
                {
                    break;
                }
                J = P.jobs + find_job<job_items>(P.jobs, job_first, job_end, item);
                const int64_t local = item - J->item_begin;
                const sample_place at = place_of(local, J->cam, 0);
                const int64_t k = at.pass; // the item's chunk within the step
                const int q = static_cast<int>(local - k * J->padded_pixels);
                px = at.x;
                py = at.y;
                if (px >= J->cam.width || py >= J->cam.height)
                {
                    continue;
                }
                const int64_t chunk_first = (J->first_chunk + k) * J->chunk;
                pass = chunk_first > J->pass_begin ? chunk_first : J->pass_begin;
                const int64_t chunk_end = chunk_first + J->chunk;
                pass_end = chunk_end < J->pass_end ? chunk_end : J->pass_end;
                slot = k * J->padded_pixels + q;
                acc_r = acc_g = acc_b = 0.0;
                rng.pixel = static_cast<uint32_t>(py) * static_cast<uint32_t>(J->cam.width) + static_cast<uint32_t>(px);
                rng.job = J->job;
                rays = 0;
                shadow_rays = 0;
                need = false;
                start = true;
            }
        }
        const camera_params& cam = J->cam;
        if (start)
        {
            const int64_t round = round_of(pass, cam);
            const int in_round = static_cast<int>(pass - round * J->round_passes);
            const uint64_t key = J->seed + (static_cast<uint64_t>(round) << 32);
            rng.key = make_uint2(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32));
            rng.pass = static_cast<uint32_t>(in_round);
            const float4 u = rng.draw(0, 0);
            int s_i, s_j;
            stratum_of(cam, in_round, s_i, s_j);
            camera_ray(cam, px, py, s_i, s_j, u, ps.o, ps.d);
            ps.time = FEATURES && J->scene.has_motion ? rng.draw(0, block_time).x : 0.0f;
            ps.throughput = make_float3(1.0f, 1.0f, 1.0f);
            ps.radiance = make_float3(0.0f, 0.0f, 0.0f);
            ps.bsdf_pdf = 0.0f;
            ps.specular = true;
            ps.rays_left = cam.max_depth;
            ps.depth = 0;
            ps.from = -1;
            ps.inward = false;
            start = false;
        }
        hit_info h;
        traverse<false, false, search, FEATURES>(J->scene, ps.o, ps.d, ps.time, infinity_f, ps.from, ps.inward, -1,
                                                 h);
        ++rays;
        ++ps.depth;
        if (FEATURES && J->scene.medium_count > 0)
        {
            media_event(J->scene, ps.o, ps.d, ps.time, rng, ps.depth, h);
        }
        float3 sample;
        const step_result r =
            J->quality
                ? shade_quality<false, search, FEATURES>(J->scene, cam, rng, ps, h, sample, shadow_rays, nullptr)
                : shade_books<FEATURES>(J->scene, cam, rng, ps, h, sample);
        if (r == step_result::done)
        {
            acc_r += without_nan(sample.x);
            acc_g += without_nan(sample.y);
            acc_b += without_nan(sample.z);
            if (++pass == pass_end)
            {
                double* out = J->partials + 3 * slot;
                out[0] = acc_r;
                out[1] = acc_g;
                out[2] = acc_b;
                atomicAdd(J->counters, static_cast<unsigned long long>(rays));
                if (shadow_rays)
                {
                    atomicAdd(J->counters + 1, static_cast<unsigned long long>(shadow_rays));
                }
                need = true;
            }
            else
            {
                start = true;
            }
        }
    }
}

// Every job's pixels, in one grid-stride pass: each pixel's chunk partials added to its job's sums in chunk order
__global__ void reduce_batch_kernel(const batch_params P)
{
    const int64_t total = P.header->total_pixels;
    const int job_count = P.header->job_count;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const batch_job& J = P.jobs[find_job<job_pixels>(P.jobs, 0, job_count, i)];
        const int64_t local = i - J.pixel_begin;
        const int y = static_cast<int>(local / J.cam.width);
        const int x = static_cast<int>(local - static_cast<int64_t>(y) * J.cam.width);
        const int q = ((y >> 2) * J.tiles_x + (x >> 3)) * 32 + ((y & 3) << 3) + (x & 7) - J.first_pixel;
        double* sum = J.sums + 3 * local;
        double r = sum[0], g = sum[1], b = sum[2];
        for (int k = 0; k < J.chunks; ++k)
        {
            const double* part = J.partials + 3 * (static_cast<int64_t>(k) * J.padded_pixels + q);
            r += part[0];
            g += part[1];
            b += part[2];
        }
        sum[0] = r;
        sum[1] = g;
        sum[2] = b;
    }
}

template <bool WIDE>
__global__ void closest_hits_kernel(const scene_view S, const float* origins, const float* directions, int64_t count,
                                    const int32_t* prim_source, int32_t* ids, float* ts)
{
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count)
    {
        return;
    }
    const float3 o = make_float3(origins[3 * i], origins[3 * i + 1], origins[3 * i + 2]);
    const float3 d = make_float3(directions[3 * i], directions[3 * i + 1], directions[3 * i + 2]);
    hit_info h;
    if constexpr (WIDE)
    {
        closest_hit_wide(S, o, d, h);
    }
    else
    {
        traverse<false>(S, o, d, 0.0f, infinity_f, -1, false, -1, h);
    }
    ids[i] = h.id >= 0 ? prim_source[h.id] : -1;
    ts[i] = h.id >= 0 ? h.t : infinity_f;
}

__global__ void camera_rays_kernel(const camera_params cam, uint64_t seed, int64_t pass, int32_t round_passes,
                                   float* origins, float* directions)
{
    const int x = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    const int y = static_cast<int>(blockIdx.y);
    if (x >= cam.width || y >= cam.height)
    {
        return;
    }
    const int64_t round = pass / round_passes;
    const int in_round = static_cast<int>(pass - round * round_passes);
    const uint64_t key = seed + (static_cast<uint64_t>(round) << 32);
    sampler rng{make_uint2(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32)),
                static_cast<uint32_t>(y) * static_cast<uint32_t>(cam.width) + static_cast<uint32_t>(x),
                static_cast<uint32_t>(in_round), 0u};
    float3 o, d;
    camera_ray(cam, x, y, in_round % cam.sqrt_spp, in_round / cam.sqrt_spp, rng.draw(0, 0), o, d);
    const int64_t i = static_cast<int64_t>(y) * cam.width + x;
    origins[3 * i] = o.x;
    origins[3 * i + 1] = o.y;
    origins[3 * i + 2] = o.z;
    directions[3 * i] = d.x;
    directions[3 * i + 1] = d.y;
    directions[3 * i + 2] = d.z;
}

// ---- the wavefront form: resident path slots, a shade kernel and a trace kernel ----------------------------------
// In the persistent kernel a warp walks the tree for all its lanes' rays together, and a lane whose ray left the
// scene at the root waits for the lane whose ray goes deepest: on the mesh and the sphere grids a walk step runs with
// 4 to 10 of 32 lanes. Here the walk is a kernel of its own whose lanes take a new ray as soon as theirs is answered
// (Aila and Laine's persistent while-while with replacement of finished rays, HPG 2009 and its 2012 addendum), and the
// paths between walks live in HBM as slots. A slot goes through the same steps, in the same order and with the same
// arithmetic, as a persistent kernel's lane: the images are the persistent kernel's.
// The query at position q of the queue: the shade step's next rays and shadow rays fill it from the bottom (`lower`
// of them), its new samples' camera rays from the top down. A primary query (pixel, pass in its round, the RNG's key) is
// made into its camera ray here, the persistent kernel's start of a sample with the same random numbers, and the ray
// goes into its slot's first two rows, which the shade step that meets its hit reads.
template <bool FEATURES, bool BATCH>
__device__ __forceinline__ void wave_camera_query(const wave_buffers& B, const wave_batch& W, const scene_view& S0,
                                                  unsigned q, unsigned lower, float4& qo, float4& qd, int4& qm)
{
    const unsigned k = q < lower ? q : 2u * static_cast<unsigned>(B.slot_count) - 1u - (q - lower);
    qo = stream_load(B.query_o + k);
    qd = stream_load(B.query_d + k);
    qm = stream_load(B.query_meta + k);
    if (qm.y & wave_query_primary)
    {
        const batch_job* J = BATCH ? W.jobs + (qm.y >> 3) : nullptr;
        const camera_params& cam = BATCH ? J->cam : B.cam;
        const scene_view& S = BATCH ? J->scene : S0;
        const int px = __float_as_int(qo.x), py = __float_as_int(qo.y), round_pass = __float_as_int(qo.z);
        sampler rng;
        rng.key = make_uint2(__float_as_uint(qd.x), __float_as_uint(qd.y));
        rng.pixel = static_cast<uint32_t>(py) * static_cast<uint32_t>(cam.width) + static_cast<uint32_t>(px);
        rng.pass = static_cast<uint32_t>(round_pass);
        rng.job = BATCH ? J->job : B.job;
        float3 o, d;
        int s_i, s_j;
        stratum_of(cam, round_pass, s_i, s_j);
        camera_ray(cam, px, py, s_i, s_j, rng.draw(0, 0), o, d);
        const float time = FEATURES && S.has_motion ? rng.draw(0, block_time).x : 0.0f;
        float4* rows = static_cast<float4*>(B.slots);
        stream_store(rows + qm.w, make_float4(o.x, o.y, o.z, time));
        stream_store(rows + B.slot_count + qm.w, make_float4(d.x, d.y, d.z, 0.0f)); // bsdf_pdf 0 at the camera
        qo = make_float4(o.x, o.y, o.z, time);
        qd = make_float4(d.x, d.y, d.z, infinity_f);
        qm.y &= ~wave_query_primary;
    }
}

// The trace kernel's resident blocks per multiprocessor (64 registers at 8) and the number of lanes still walking
// under which a warp stops to give its idle lanes new queries (the addendum's 20 of 32)
#ifndef RTB_TRACE_MIN_BLOCKS
#define RTB_TRACE_MIN_BLOCKS RTB_TRACE_MIN_BLOCKS_DEFAULT
#endif
#ifndef RTB_REFILL_LANES
#define RTB_REFILL_LANES 20
#endif

// The queued queries' walks through the tree: closest hits for the paths' next rays, any hit for shadow rays (the
// persistent kernel's traverse, the same leaf tests and self-intersection rules). WIDE: the tree four wide, a node's
// hit children visited nearest first (a four-key sorting network); otherwise the binary tree in the persistent
// kernel's node order. BATCH: each query walks its own job's scene (the job in its flags); otherwise the launch's
// scene S0. The walks are counted into `counters` when it is given.
template <bool FEATURES, bool BATCH, bool WIDE, int MINB = RTB_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(render_block, MINB)
    wave_trace_kernel(const __grid_constant__ scene_view S0, const __grid_constant__ wave_buffers B,
                      const __grid_constant__ wave_batch W, unsigned long long* counters)
{
    __shared__ unsigned block_walks[2]; // the block's closest-hit and shadow queries: the path segments and shadow rays
    if (threadIdx.x < 2)
    {
        block_walks[threadIdx.x] = 0;
    }
    __syncthreads();
    const unsigned lower = B.control[0];
    const unsigned count = lower + B.control[2];
    unsigned walks[2] = {0, 0};
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    int2 stack[WIDE ? wide_stack : max_bvh_depth];
    int sp = 0;
    int link = traversal_done;
    int leaf = 0;
    bool has_query = false;
    bool drained = false; // the warp found the queue empty: no idle lane can take a query any more
    float3 o = make_float3(0.0f, 0.0f, 0.0f);
    float3 d = o, inv = o, os = o;
    float time = 0.0f;
    float inverse_a = 0.0f;
    int from = -1, skip = -1, slot = 0;
    bool inward = false, shadow = false;
    hit_info hit{-1, 0.0f, false};
    // the scene the lane's query walks: its job's, or the launch's (a __grid_constant__ parameter, read in place)
    const scene_view* job_scene = BATCH ? &W.jobs[W.job_first].scene : &S0;
    const auto scene = [&]() -> const scene_view& { return *job_scene; };
    // the lane's tree, read from its scene once a query (a batch's scene is in global memory, where every read of it
    // in the walk would wait on L1 behind the stack's stores)
    const bvh_node* tree_nodes = scene().nodes;
    const bvh4_node* tree_wide = scene().wide_nodes;
    const auto pop = [&]() -> int {
        while (sp > 0)
        {
            const int2 e = stack[--sp];
            if (shadow || __int_as_float(e.y) < hit.t)
            {
                return e.x;
            }
        }
        return traversal_done;
    };
    // Warp-synchronous: every lane runs every loop, with nothing to do once its query is answered and the queue is
    // empty, so that each ballot sees the whole warp and the refill rule holds as written
    while (true)
    {
        const bool answered = has_query && link == traversal_done && leaf == 0;
        if (answered)
        {
            if (shadow)
            {
                stream_store(B.shadow_result + slot, hit.id >= 0 ? 1 : 0);
            }
            else
            {
                stream_store(B.ext_result + slot, make_int4(hit.id, __float_as_int(hit.t), hit.front ? 1 : 0, 0));
            }
            has_query = false;
        }
        // New queries for the idle lanes: one atomic per warp
        const unsigned idle = __ballot_sync(full_warp, !has_query);
        if (idle != 0u && !drained)
        {
            const int leader = __ffs(static_cast<int>(idle)) - 1;
            unsigned base = 0;
            if (static_cast<int>(lane) == leader)
            {
                base = atomicAdd(B.control + 1, static_cast<unsigned>(__popc(idle)));
            }
            base = __shfl_sync(full_warp, base, leader);
            drained = base + static_cast<unsigned>(__popc(idle)) >= count;
            const unsigned q = base + static_cast<unsigned>(__popc(idle & lanes_below));
            if (!has_query && q < count)
            {
                float4 qo, qd;
                int4 qm;
                wave_camera_query<FEATURES, BATCH>(B, W, S0, q, lower, qo, qd, qm);
                o = make_float3(qo.x, qo.y, qo.z);
                time = qo.w;
                d = make_float3(qd.x, qd.y, qd.z);
                hit.id = -1;
                hit.t = qd.w;
                hit.front = false;
                from = qm.x;
                inward = (qm.y & 1) != 0;
                shadow = (qm.y & 2) != 0;
                skip = qm.z;
                slot = qm.w;
                if constexpr (BATCH)
                {
                    job_scene = &W.jobs[qm.y >> 3].scene;
                    tree_nodes = scene().nodes;
                    tree_wide = scene().wide_nodes;
                }
                ++walks[shadow ? 1 : 0];
                inverse_a = 1.0f / length_squared(d);
                inv = make_float3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
                os = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
                sp = 0;
                leaf = 0;
                link = scene().node_count == 0 ? traversal_done : 0;
                has_query = true;
                if (BATCH && scene().flat != 0)
                {
                    // a flat-searched scene beside tree-searched ones (a stream run): its query answered here by the
                    // flat search, the same hits its session's flat trace kernel finds
                    flat_search_call<FEATURES>(scene(), o, d, time, from, inward, skip, shadow, hit);
                    link = traversal_done;
                }
            }
        }
        if (__ballot_sync(full_warp, has_query) == 0u)
        {
            break; // the queue is empty and every lane's query answered
        }
        // The walks, until fewer than RTB_REFILL_LANES lanes are still walking (or none, once the queue is empty)
        while (true)
        {
            // inner nodes: a lane descends, setting aside the first leaf it meets, until every descending lane holds one
            while (true)
            {
                const bool descending = has_query && link >= 0;
                if (!__any_sync(full_warp, descending))
                {
                    break;
                }
                if (WIDE && descending)
                {
                    const float4* np = reinterpret_cast<const float4*>(tree_wide + link);
                    const float4 lx = __ldg(np), hx = __ldg(np + 1);
                    const float4 ly = __ldg(np + 2), hy = __ldg(np + 3);
                    const float4 lz = __ldg(np + 4), hz = __ldg(np + 5);
                    const int4 nl = __ldg(reinterpret_cast<const int4*>(np + 6));
                    // each child's entry distance, or infinity where the ray misses it (or the slot is unused)
                    const auto entry = [&](float lox, float hix, float loy, float hiy, float loz, float hiz,
                                           int child) -> float {
                        const float a0 = fmaf(lox, inv.x, -os.x), a1 = fmaf(hix, inv.x, -os.x);
                        const float b0 = fmaf(loy, inv.y, -os.y), b1 = fmaf(hiy, inv.y, -os.y);
                        const float c0 = fmaf(loz, inv.z, -os.z), c1 = fmaf(hiz, inv.z, -os.z);
                        const float enter = fmaxf(fmaxf(fminf(a0, a1), fminf(b0, b1)), fmaxf(fminf(c0, c1), t_min));
                        const float exit = fminf(fminf(fmaxf(a0, a1), fmaxf(b0, b1)), fminf(fmaxf(c0, c1), hit.t));
                        return enter <= exit && child != traversal_done ? enter : infinity_f;
                    };
                    float k0 = entry(lx.x, hx.x, ly.x, hy.x, lz.x, hz.x, nl.x);
                    float k1 = entry(lx.y, hx.y, ly.y, hy.y, lz.y, hz.y, nl.y);
                    float k2 = entry(lx.z, hx.z, ly.z, hy.z, lz.z, hz.z, nl.z);
                    float k3 = entry(lx.w, hx.w, ly.w, hy.w, lz.w, hz.w, nl.w);
                    int l0 = nl.x, l1 = nl.y, l2 = nl.z, l3 = nl.w;
                    const auto order = [](float& ka, int& la, float& kb, int& lb) {
                        if (kb < ka)
                        {
                            const float k = ka;
                            ka = kb;
                            kb = k;
                            const int l = la;
                            la = lb;
                            lb = l;
                        }
                    };
                    order(k0, l0, k1, l1);
                    order(k2, l2, k3, l3);
                    order(k0, l0, k2, l2);
                    order(k1, l1, k3, l3);
                    order(k1, l1, k2, l2);
                    if (k0 == infinity_f)
                    {
                        link = pop();
                    }
                    else
                    {
                        // the far ones wait on the stack, farthest deepest; the nearest is next
                        if (k3 != infinity_f)
                        {
                            stack[sp++] = make_int2(l3, __float_as_int(k3));
                        }
                        if (k2 != infinity_f)
                        {
                            stack[sp++] = make_int2(l2, __float_as_int(k2));
                        }
                        if (k1 != infinity_f)
                        {
                            stack[sp++] = make_int2(l1, __float_as_int(k1));
                        }
                        link = l0;
                    }
                    if (link < 0 && link != traversal_done && leaf == 0)
                    {
                        leaf = link;
                        link = pop();
                    }
                }
                else if (descending)
                {
                    const float4* np = reinterpret_cast<const float4*>(tree_nodes + link);
                    const float4 nx = __ldg(np);
                    const float4 ny = __ldg(np + 1);
                    const float4 nz = __ldg(np + 2);
                    const int2 nl = __ldg(reinterpret_cast<const int2*>(np + 3));
                    const float a0 = fmaf(nx.x, inv.x, -os.x), a1 = fmaf(nx.y, inv.x, -os.x);
                    const float b0 = fmaf(ny.x, inv.y, -os.y), b1 = fmaf(ny.y, inv.y, -os.y);
                    const float c0 = fmaf(nz.x, inv.z, -os.z), c1 = fmaf(nz.y, inv.z, -os.z);
                    const float enter0 = fmaxf(fmaxf(fminf(a0, a1), fminf(b0, b1)), fmaxf(fminf(c0, c1), t_min));
                    const float exit0 = fminf(fminf(fmaxf(a0, a1), fmaxf(b0, b1)), fminf(fmaxf(c0, c1), hit.t));
                    const float a2 = fmaf(nx.z, inv.x, -os.x), a3 = fmaf(nx.w, inv.x, -os.x);
                    const float b2 = fmaf(ny.z, inv.y, -os.y), b3 = fmaf(ny.w, inv.y, -os.y);
                    const float c2 = fmaf(nz.z, inv.z, -os.z), c3 = fmaf(nz.w, inv.z, -os.z);
                    const float enter1 = fmaxf(fmaxf(fminf(a2, a3), fminf(b2, b3)), fmaxf(fminf(c2, c3), t_min));
                    const float exit1 = fminf(fminf(fmaxf(a2, a3), fmaxf(b2, b3)), fminf(fmaxf(c2, c3), hit.t));
                    const bool h0 = enter0 <= exit0;
                    const bool h1 = enter1 <= exit1;
                    if (h0 && h1)
                    {
                        const bool second_first = enter1 < enter0;
                        link = second_first ? nl.y : nl.x;
                        stack[sp++] =
                            make_int2(second_first ? nl.x : nl.y, __float_as_int(second_first ? enter0 : enter1));
                    }
                    else if (h0 || h1)
                    {
                        link = h0 ? nl.x : nl.y;
                    }
                    else
                    {
                        link = pop();
                    }
                    if (link < 0 && link != traversal_done && leaf == 0)
                    {
                        leaf = link;
                        link = pop();
                    }
                }
                if (!__any_sync(full_warp, has_query && link >= 0 && leaf == 0))
                {
                    break; // every lane still descending holds a leaf: test them together
                }
            }
            // leaves
            while (true)
            {
                const bool testing = has_query && leaf < 0;
                if (!__any_sync(full_warp, testing))
                {
                    break;
                }
                if (testing)
                {
                    if (test_leaf<false, false, FEATURES>(scene(), leaf, o, d, time, inverse_a, from, inward, skip,
                                                          hit, nullptr, shadow))
                    {
                        hit.id = 1; // a shadow ray's blocker: answered
                        leaf = 0;
                        link = traversal_done;
                    }
                    else
                    {
                        leaf = 0;
                        if (link < 0 && link != traversal_done)
                        {
                            leaf = link;
                            link = pop();
                        }
                    }
                }
            }
            const unsigned walking = __ballot_sync(full_warp, has_query && !(link == traversal_done && leaf == 0));
            if (walking == 0u || (!drained && __popc(walking) < RTB_REFILL_LANES))
            {
                break;
            }
        }
    }
    atomicAdd(&block_walks[0], walks[0]);
    atomicAdd(&block_walks[1], walks[1]);
    __syncthreads();
    if (counters != nullptr && threadIdx.x < 2 && block_walks[threadIdx.x] != 0u)
    {
        atomicAdd(counters + threadIdx.x, static_cast<unsigned long long>(block_walks[threadIdx.x]));
    }
}

// The queued queries of a flat-searched scene: one query per thread at a time (grid-stride), every lane the same
// loop over the same records, no tree, no stack, no refill. BATCH: each query searches its job's scene (W's table; a
// warp's lanes may loop over different scenes), its walks counted where the shade kernel queued it.
template <bool FEATURES, bool BATCH, int MINB = RTB_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(render_block, MINB)
    wave_flat_trace_kernel(const __grid_constant__ scene_view S, const __grid_constant__ wave_buffers B,
                           const __grid_constant__ wave_batch W, unsigned long long* counters)
{
    __shared__ unsigned block_walks[2];
    if (threadIdx.x < 2)
    {
        block_walks[threadIdx.x] = 0;
    }
    __syncthreads();
    const unsigned count = B.control[0];
    unsigned walks[2] = {0, 0};
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x)
    {
        const float4 qo = stream_load(B.query_o + q);
        const float4 qd = stream_load(B.query_d + q);
        const int4 qm = stream_load(B.query_meta + q);
        const bool shadow = (qm.y & 2) != 0;
        hit_info hit{-1, qd.w, false};
        const scene_view* scene = &S;
        if constexpr (BATCH)
        {
            scene = &W.jobs[qm.y >> 3].scene;
        }
        flat_search<FEATURES>(*scene, make_float3(qo.x, qo.y, qo.z), make_float3(qd.x, qd.y, qd.z), qo.w, qm.x,
                              (qm.y & 1) != 0, qm.z, shadow, hit);
        if (shadow)
        {
            stream_store(B.shadow_result + qm.w, hit.id >= 0 ? 1 : 0);
        }
        else
        {
            stream_store(B.ext_result + qm.w, make_int4(hit.id, __float_as_int(hit.t), hit.front ? 1 : 0, 0));
        }
        ++walks[shadow ? 1 : 0];
    }
    atomicAdd(&block_walks[0], walks[0]);
    atomicAdd(&block_walks[1], walks[1]);
    __syncthreads();
    if (counters != nullptr && threadIdx.x < 2 && block_walks[threadIdx.x] != 0u)
    {
        atomicAdd(counters + threadIdx.x, static_cast<unsigned long long>(block_walks[threadIdx.x]));
    }
}

// The wavefront's samples into the image's sums: each chunk's samples added in pass order into its partial, the
// partials in chunk order into the sums, as the persistent kernel's lanes and reduce_kernel add them
__global__ void wave_reduce_kernel(const reduce_params R, const float4* samples, int64_t pass_begin, int64_t pass_end,
                                   int32_t chunk)
{
    const int x = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    const int y = static_cast<int>(blockIdx.y);
    if (x >= R.width || y >= R.height)
    {
        return;
    }
    const int q = ((y >> 2) * R.tiles_x + (x >> 3)) * 32 + ((y & 3) << 3) + (x & 7);
    double* sum = R.sums + 3 * (static_cast<int64_t>(y) * R.width + x);
    double r = sum[0], g = sum[1], b = sum[2];
    int64_t pass = pass_begin;
    while (pass < pass_end)
    {
        const int64_t chunk_end = (pass / chunk + 1) * chunk;
        const int64_t end = chunk_end < pass_end ? chunk_end : pass_end;
        double pr = 0.0, pg = 0.0, pb = 0.0;
        for (; pass < end; ++pass)
        {
            const float4 s = samples[(pass - pass_begin) * R.padded_pixels + q];
            pr += without_nan(s.x);
            pg += without_nan(s.y);
            pb += without_nan(s.z);
        }
        r += pr;
        g += pg;
        b += pb;
    }
    sum[0] = r;
    sum[1] = g;
    sum[2] = b;
}

// A stream run's finished segments into their requests' images (stream_reduce_item): one thread per pixel of an
// item; the segment's samples of that pixel, pass after pass, into the request's chunk accumulator, which goes into
// the sums after a chunk's last pass, after the first pass (the first frame) and at the target. A pixel's passes
// arrive in order (the host reduces a request's segments one after another), so a pixel's sums are the session's
// chunk partials added in chunk order, up to the first frame's split of the first chunk.
__global__ void stream_reduce_kernel(const stream_reduce_item* items, int32_t count, int64_t total_pixels)
{
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total_pixels;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        int lo = 0, hi = count - 1;
        while (lo < hi)
        {
            const int mid = (lo + hi + 1) >> 1;
            if (items[mid].pixel_begin <= i)
            {
                lo = mid;
            }
            else
            {
                hi = mid - 1;
            }
        }
        const stream_reduce_item& it = items[lo];
        const int64_t pixel = i - it.pixel_begin;
        const int y = static_cast<int>(pixel / it.width);
        const int x = static_cast<int>(pixel - static_cast<int64_t>(y) * it.width);
        const int q = ((y >> 2) * it.tiles_x + (x >> 3)) * 32 + ((y & 3) << 3) + (x & 7);
        // the passes whose sample of this pixel lies in [local_begin, local_end)
        const int64_t padded = it.padded_pixels;
        int64_t pass = (it.local_begin - q + padded - 1) / padded;
        pass = pass < 0 ? 0 : pass;
        double* acc = it.acc + 3 * pixel;
        double* sum = it.sums + 3 * pixel;
        double ar = acc[0], ag = acc[1], ab = acc[2];
        for (int64_t local = pass * padded + q; local < it.local_end; local += padded, ++pass)
        {
            const float4 v = it.values[local - it.local_begin];
            ar += without_nan(v.x);
            ag += without_nan(v.y);
            ab += without_nan(v.z);
            const int64_t done = pass + 1;
            if (done % it.chunk == 0 || done == 1 || done == it.target)
            {
                sum[0] += ar;
                sum[1] += ag;
                sum[2] += ab;
                ar = ag = ab = 0.0;
            }
        }
        acc[0] = ar;
        acc[1] = ag;
        acc[2] = ab;
    }
}


// A wavefront group's samples into its jobs' chunk partials, laid out as the persistent batch kernel writes them: each
// work item (chunk, pixel) the sum of its passes' samples in pass order; items of pixels over the image's edge skipped
__global__ void wave_batch_partials_kernel(const wave_batch W, const float4* samples)
{
    for (int64_t i = W.item_first + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < W.item_end;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const batch_job& J = W.jobs[find_job<job_items>(W.jobs, W.job_first, W.job_end, i)];
        const int64_t local = i - J.item_begin;
        const int64_t k = local / J.padded_pixels;
        const int q = static_cast<int>(local - k * J.padded_pixels);
        const int tile = (J.first_pixel + q) >> 5;
        const int l = q & 31;
        if ((tile % J.tiles_x) * 8 + (l & 7) >= J.cam.width || (tile / J.tiles_x) * 4 + (l >> 3) >= J.cam.height)
        {
            continue;
        }
        const int64_t chunk_first = (J.first_chunk + k) * J.chunk;
        const int64_t begin = chunk_first > J.pass_begin ? chunk_first : J.pass_begin;
        const int64_t end = chunk_first + J.chunk < J.pass_end ? chunk_first + J.chunk : J.pass_end;
        double r = 0.0, g = 0.0, b = 0.0;
        for (int64_t pass = begin; pass < end; ++pass)
        {
            const float4 s = samples[J.sample_begin + (pass - J.pass_begin) * J.padded_pixels + q];
            r += without_nan(s.x);
            g += without_nan(s.y);
            b += without_nan(s.z);
        }
        double* out = J.partials + 3 * local;
        out[0] = r;
        out[1] = g;
        out[2] = b;
    }
}
} // namespace

namespace
{
using render_function = void (*)(launch_params);

template <bool QUALITY, bool FLAT>
render_function render_kernel_of(bool counting, bool features)
{
    if (counting)
    {
        return render_kernel<QUALITY, true, FLAT, true>;
    }
    return features ? render_kernel<QUALITY, false, FLAT, true> : render_kernel<QUALITY, false, FLAT, false>;
}

// The render kernel for an integrator, the counting build or not, a flat or a tree search, and a scene with or
// without the second book's features
render_function render_kernel_for(bool quality, bool counting, bool flat, bool features)
{
    if (quality)
    {
        return flat ? render_kernel_of<true, true>(counting, features)
                    : render_kernel_of<true, false>(counting, features);
    }
    return flat ? render_kernel_of<false, true>(counting, features) : render_kernel_of<false, false>(counting, features);
}
} // namespace

cudaError_t launch_render(const launch_params& p, bool quality, bool counting, int grid, cudaStream_t stream)
{
    render_kernel_for(quality, counting, p.scene.flat != 0, has_features(p.scene))<<<grid, render_block, 0, stream>>>(
        p);
    return cudaGetLastError();
}

namespace
{
using batch_function = void (*)(batch_params);

batch_function batch_kernel_of(int group)
{
    switch (group)
    {
    case 0:
        return render_batch_kernel<true, false>;
    case 1:
        return render_batch_kernel<true, true>;
    case 2:
        return render_batch_kernel<false, false>;
    default:
        return render_batch_kernel<false, true>;
    }
}
} // namespace

cudaError_t launch_batch(const batch_params& p, const int* grids, int first_group, int end_group, cudaStream_t stream)
{
    for (int g = first_group; g < end_group; ++g)
    {
        batch_kernel_of(g)<<<grids[g], render_block, 0, stream>>>(p);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
        {
            return e;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_batch_reduce(const batch_params& p, int grid, cudaStream_t stream)
{
    reduce_batch_kernel<<<grid, 256, 0, stream>>>(p);
    return cudaGetLastError();
}

// Two attribute queries for the device: cudaGetDeviceProperties would fill every field of its description, a cost each
// session paid. A kernel's attributes are asked for once a device: sessions and servers are made often, and the
// queries take some 50 us a kernel.
cudaError_t function_attributes(const void* kernel, kernel_attributes& out, int shared)
{
    static std::mutex mutex;
    static auto* known = new std::map<std::pair<const void*, int>, kernel_attributes>();
    cudaFuncAttributes a{};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess)
    {
        const std::lock_guard<std::mutex> lock(mutex);
        if (const auto it = known->find({kernel, device}); it != known->end())
        {
            out = it->second;
            return cudaSuccess;
        }
        e = cudaFuncGetAttributes(&a, kernel);
    }
    int blocks = 0;
    if (e == cudaSuccess)
    {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, render_block, static_cast<size_t>(shared));
    }
    int multiprocessors = 0;
    int max_threads = 0;
    if (e == cudaSuccess)
    {
        e = cudaDeviceGetAttribute(&multiprocessors, cudaDevAttrMultiProcessorCount, device);
    }
    if (e == cudaSuccess)
    {
        e = cudaDeviceGetAttribute(&max_threads, cudaDevAttrMaxThreadsPerMultiProcessor, device);
    }
    if (e != cudaSuccess)
    {
        return e;
    }
    out.registers = a.numRegs;
    out.local_bytes = static_cast<int>(a.localSizeBytes);
    out.blocks_per_sm = blocks;
    out.threads_per_block = render_block;
    out.max_threads_per_sm = max_threads;
    out.multiprocessors = multiprocessors;
    const std::lock_guard<std::mutex> lock(mutex);
    (*known)[{kernel, device}] = out;
    return cudaSuccess;
}

namespace
{
template <class Kernel>
cudaError_t attributes_of(Kernel kernel, kernel_attributes& out)
{
    return function_attributes(reinterpret_cast<const void*>(kernel), out);
}
} // namespace

cudaError_t batch_attributes(int group, kernel_attributes& out) { return attributes_of(batch_kernel_of(group), out); }

cudaError_t launch_reduce(const reduce_params& p, cudaStream_t stream)
{
    const dim3 block(128, 1);
    const dim3 grid(static_cast<unsigned>((p.width + 127) / 128), static_cast<unsigned>(p.height));
    reduce_kernel<<<grid, block, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t render_attributes(const scene_view& scene, bool quality, kernel_attributes& out)
{
    return attributes_of(render_kernel_for(quality, false, scene.flat != 0, has_features(scene)), out);
}

cudaError_t launch_closest_hits(const scene_view& s, const float* origins, const float* directions, int64_t count,
                                const int32_t* prim_source, int32_t* ids, float* ts, cudaStream_t stream)
{
    if (count <= 0)
    {
        return cudaSuccess;
    }
    const int block = 128;
    const auto grid = static_cast<unsigned>((count + block - 1) / block);
    // the tree four wide where there is one (half the dependent steps of the binary walk); a flat scene's primitives in turn
    const bool wide = s.flat == 0 && s.node_count > 0 && s.wide_nodes != nullptr;
    (wide ? closest_hits_kernel<true> : closest_hits_kernel<false>)<<<grid, block, 0, stream>>>(
        s, origins, directions, count, prim_source, ids, ts);
    return cudaGetLastError();
}

size_t wave_slot_bytes() { return (wave_rows + wave_shadow_rows) * sizeof(float4); }

cudaError_t clear_wave_slots(const wave_buffers& b, cudaStream_t stream)
{
    // the other rows are written when a slot's first sample starts
    return cudaMemsetAsync(static_cast<float4*>(b.slots) + int64_t{wave_flags_row} * b.slot_count, 0,
                           static_cast<size_t>(b.slot_count) * sizeof(float4), stream);
}

namespace
{
using wave_trace_function = void (*)(scene_view, wave_buffers, wave_batch, unsigned long long*);

template <bool BATCH>
wave_trace_function wave_trace_variant(bool features, bool wide)
{
    if (wide)
    {
        return features ? wave_trace_kernel<true, BATCH, true> : wave_trace_kernel<false, BATCH, true>;
    }
    return features ? wave_trace_kernel<true, BATCH, false> : wave_trace_kernel<false, BATCH, false>;
}

wave_shade_function wave_shade_of(bool quality, bool features)
{
    if (quality)
    {
        return features ? wave_shade_kernel<true, true, false> : quality_shade_kernel();
    }
    return features ? wave_shade_kernel<false, true, false> : wave_shade_kernel<false, false, false>;
}

// A session's walk at one of the register caps the autotuner chooses between: the default blocks per multiprocessor
// (64 registers a thread at 8 blocks of 128) or fewer blocks with more registers (80 at 6)
wave_trace_function wave_trace_of(bool features, bool wide, int min_blocks = RTB_TRACE_MIN_BLOCKS)
{
    if (min_blocks == wave_trace_roomy_blocks)
    {
        if (wide)
        {
            return features ? wave_trace_kernel<true, false, true, wave_trace_roomy_blocks>
                            : wave_trace_kernel<false, false, true, wave_trace_roomy_blocks>;
        }
        return features ? wave_trace_kernel<true, false, false, wave_trace_roomy_blocks>
                        : wave_trace_kernel<false, false, false, wave_trace_roomy_blocks>;
    }
    return wave_trace_variant<false>(features, wide);
}

template <bool BATCH>
wave_trace_function wave_flat_trace_of(bool features, int min_blocks = RTB_TRACE_MIN_BLOCKS)
{
    if (!BATCH && min_blocks == wave_trace_roomy_blocks)
    {
        return features ? wave_flat_trace_kernel<true, false, wave_trace_roomy_blocks>
                        : wave_flat_trace_kernel<false, false, wave_trace_roomy_blocks>;
    }
    return features ? wave_flat_trace_kernel<true, BATCH> : wave_flat_trace_kernel<false, BATCH>;
}
} // namespace

// marks (when given): three events recorded before the shade kernel, between the two kernels and after the trace
// kernel, for per-kernel timing
cudaError_t launch_wave_step(const launch_params& p, bool quality, const wave_buffers& slots, const wave_shape& shape,
                             cudaStream_t stream, const cudaEvent_t* marks, bool draining)
{
    const int trace_grid = shape.trace_grid;
    const int shade_block = shape.shade_block > 0 ? shape.shade_block : render_block;
    wave_buffers b = slots; // with the launch's camera and RNG job, for the camera rays the trace kernel makes
    b.cam = p.cam;
    b.job = p.job;
    b.draining = draining ? 1 : 0;
    cudaError_t e = cudaMemsetAsync(b.control, 0, 3 * sizeof(unsigned), stream);
    if (e != cudaSuccess)
    {
        return e;
    }
    const bool features = has_features(p.scene);
    if (marks)
    {
        cudaEventRecord(marks[0], stream);
    }
    wave_shade_of(quality, features)<<<b.slot_count / shade_block, shade_block, 0, stream>>>(p, b, wave_batch{});
    e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        return e;
    }
    if (marks)
    {
        cudaEventRecord(marks[1], stream);
    }
    if (p.scene.flat != 0)
    {
        wave_flat_trace_of<false>(features, shape.trace_min_blocks)<<<trace_grid, render_block, 0, stream>>>(
            p.scene, b, wave_batch{}, p.counters);
    }
    else
    {
        wave_trace_of(features, p.scene.wide_nodes != nullptr, shape.trace_min_blocks)<<<trace_grid, render_block, 0,
                                                                                          stream>>>(
            p.scene, b, wave_batch{}, p.counters);
    }
    e = cudaGetLastError();
    if (marks && e == cudaSuccess)
    {
        cudaEventRecord(marks[2], stream);
    }
    return e;
}

cudaError_t launch_wave_batch_step(const wave_batch& w, bool flat, bool features, bool wide, bool quality,
                                   const wave_buffers& b, int trace_grid, cudaStream_t stream, bool draining)
{
    cudaError_t e = cudaMemsetAsync(b.control, 0, 3 * sizeof(unsigned), stream);
    if (e != cudaSuccess)
    {
        return e;
    }
    const launch_params none{};
    const auto shade = quality ? (features ? wave_shade_kernel<true, true, true> : wave_shade_kernel<true, false, true>)
                               : (features ? wave_shade_kernel<false, true, true> : wave_shade_kernel<false, false, true>);
    wave_buffers bd = b;
    bd.draining = draining ? 1 : 0;
    shade<<<b.slot_count / render_block, render_block, 0, stream>>>(none, bd, w);
    e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        return e;
    }
    const wave_trace_function trace = flat ? wave_flat_trace_of<true>(features) : wave_trace_variant<true>(features, wide);
    trace<<<trace_grid, render_block, 0, stream>>>(scene_view{}, bd, w, nullptr);
    return cudaGetLastError();
}

cudaError_t preload_wave_batch()
{
    cudaFuncAttributes a{};
    const void* kernels[] = {reinterpret_cast<const void*>(wave_shade_kernel<false, false, true>),
                             reinterpret_cast<const void*>(wave_shade_kernel<false, true, true>),
                             reinterpret_cast<const void*>(wave_shade_kernel<true, false, true>),
                             reinterpret_cast<const void*>(wave_shade_kernel<true, true, true>),
                             reinterpret_cast<const void*>(wave_trace_variant<true>(false, false)),
                             reinterpret_cast<const void*>(wave_trace_variant<true>(false, true)),
                             reinterpret_cast<const void*>(wave_trace_variant<true>(true, false)),
                             reinterpret_cast<const void*>(wave_trace_variant<true>(true, true)),
                             reinterpret_cast<const void*>(wave_flat_trace_of<true>(false)),
                             reinterpret_cast<const void*>(wave_flat_trace_of<true>(true)),
                             reinterpret_cast<const void*>(wave_batch_partials_kernel)};
    for (const void* k : kernels)
    {
        const cudaError_t e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess)
        {
            return e;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_stream_reduce(const stream_reduce_item* items, int32_t count, int64_t total_pixels,
                                 cudaStream_t stream)
{
    if (count <= 0 || total_pixels <= 0)
    {
        return cudaSuccess;
    }
    const int64_t wanted = (total_pixels + 255) / 256;
    const int64_t blocks = wanted < 148 * 16 ? wanted : 148 * 16;
    stream_reduce_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(items, count, total_pixels);
    return cudaGetLastError();
}

cudaError_t launch_wave_batch_partials(const wave_batch& w, const wave_buffers& b, cudaStream_t stream)
{
    if (w.item_end <= w.item_first)
    {
        return cudaSuccess;
    }
    const int64_t blocks = std::min<int64_t>((w.item_end - w.item_first + 255) / 256, 148 * 16);
    wave_batch_partials_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(w, b.samples);
    return cudaGetLastError();
}

cudaError_t launch_wave_reduce(const reduce_params& r, const wave_buffers& b, int64_t pass_begin, int64_t pass_end,
                               int32_t chunk, cudaStream_t stream)
{
    const dim3 block(128, 1);
    const dim3 grid(static_cast<unsigned>((r.width + 127) / 128), static_cast<unsigned>(r.height));
    wave_reduce_kernel<<<grid, block, 0, stream>>>(r, b.samples, pass_begin, pass_end, chunk);
    return cudaGetLastError();
}

cudaError_t wave_attributes(const scene_view& scene, bool quality, kernel_attributes& shade, kernel_attributes& trace,
                            int trace_min_blocks)
{
    const bool features = has_features(scene);
    const cudaError_t e = attributes_of(wave_shade_of(quality, features), shade);
    if (e != cudaSuccess)
    {
        return e;
    }
    // the session's trace kernel of the scene's search at the given register cap
    if (scene.flat != 0)
    {
        return attributes_of(wave_flat_trace_of<false>(features, trace_min_blocks), trace);
    }
    return attributes_of(wave_trace_of(features, scene.wide_nodes != nullptr, trace_min_blocks), trace);
}

cudaError_t launch_camera_rays(const camera_params& cam, uint64_t seed, int64_t pass, int32_t round_passes,
                               float* origins, float* directions, cudaStream_t stream)
{
    const dim3 block(128, 1);
    const dim3 grid(static_cast<unsigned>((cam.width + 127) / 128), static_cast<unsigned>(cam.height));
    camera_rays_kernel<<<grid, block, 0, stream>>>(cam, seed, pass, round_passes, origins, directions);
    return cudaGetLastError();
}
} // namespace rtb
