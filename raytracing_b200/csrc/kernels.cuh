// The launch interface between the host code (session.cpp) and the kernels (kernels.cu).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "device_types.h"

namespace rtb
{
// One launch of the persistent render kernel: passes [pass_begin, pass_end) of every pixel of one view, cut into
// work items (pixel, chunk of passes). Chunks are aligned to absolute multiples of `chunk` passes, so an image of N
// passes is the same bit for bit however its passes were grouped into launches, as long as launches start and end
// on chunk boundaries.
struct launch_params
{
    scene_view scene;
    camera_params cam;
    uint64_t seed;          // round r of strata draws with seed + r * 2^32 (renderer.h:564-584)
    int64_t pass_begin;
    int64_t pass_end;
    int64_t first_chunk;    // pass_begin / chunk
    int32_t chunk;          // passes per work item
    int32_t chunks;         // work items per pixel in this launch
    int32_t tiles_x;        // the image in tiles of 8 x 4 pixels, a warp's worth
    int32_t padded_pixels;  // tiles * 32
    int64_t total_items;    // chunks * padded_pixels
    int32_t round_passes;   // sqrt_spp^2
    uint32_t job;           // a request's id in the RNG counter (0 for a plain render)
    unsigned long long* work_counter;
    double* partials;       // chunks * padded_pixels * 3
    unsigned long long* counters; // [0] path segments, [1] shadow rays; the counting build also [2] node fetches,
                                  // [3] sphere, [4] quad, [5] triangle tests
};

struct reduce_params
{
    const double* partials;
    double* sums;           // width * height * 3
    int32_t width, height;
    int32_t tiles_x;
    int32_t padded_pixels;
    int32_t chunks;
};

// One job of a batched launch: a resident scene's view, its camera, and the passes this step renders of it. Its work
// items are numbered from item_begin in the batch's item space, its pixels from pixel_begin in the batch's pixel
// space (for the reduction); partials is its own slice of the batch's partials arena. A job of a group the wavefront
// renders numbers its samples from sample_begin in its group's sample space. A job rendered in bands (the pool kernel's
// alone) has in this step padded_pixels of the padded image from first_pixel on, with its camera's divisor and its items
// to match, one chunk of passes, and its partials from that pixel on; the pixels come into the reduction with its last.
struct alignas(16) batch_job
{
    scene_view scene;
    camera_params cam;
    uint64_t seed;
    int64_t pass_begin;
    int64_t pass_end;
    int64_t first_chunk;
    int64_t item_begin;
    int64_t pixel_begin;
    int64_t sample_begin;
    double* partials;
    double* sums;                 // width * height * 3, this job's
    unsigned long long* counters; // [0] segments, [1] shadow rays, this job's, accumulated
    int32_t chunk;
    int32_t chunks;
    int32_t tiles_x;
    int32_t padded_pixels;
    int32_t round_passes;
    int32_t quality;
    uint32_t job;                 // the RNG counter's job field
    int32_t first_pixel;
    // A stream run's segment (the server's continuous wavefront): its samples are [sample_begin, sample_begin +
    // pass-major count) of the run's sample space, numbered within the request from local_begin; their values go to
    // values[local - local_begin] and each finished one is counted in *done
    float4* values;
    unsigned long long* done;
    int64_t local_begin;
};

// Whether a scene has any of the second book's features (moving spheres, textures other than solid colors, smoke):
// its kernels are compiled with their code, the others without
RTB_HD inline bool has_features(const scene_view& s) { return s.has_motion != 0 || s.has_textures != 0 || s.medium_count > 0; }

// Whether the wavefront's steps render a scene faster than the persistent kernel (a session's AUTO takes the pool kernel
// before either, pool_suits): every tree-searched scene (its walks diverge: the mesh 3.2 times and the sphere scenes
// 1.2-2 times as fast) and a flat-searched scene whose shading is heavy (lights or lamps, the second book's features, an
// environment: the glass Cornell box 10-16% faster, the marble spheres 55%); not the bare small flat scenes (five spheres
// or five quads under the sky), whose paths are one or two cheap segments that cannot pay for the slots' traffic (40%
// slower).
inline bool wavefront_suits(const scene_view& v)
{
    const bool heavy = v.light_count > 0 || v.lamp_count > 0 || has_features(v) || v.has_environment;
    return v.node_count > 0 && (v.flat == 0 || heavy);
}

// The jobs come in twelve groups: the scenes of each search (flat, tree) without and with the second book's features,
// in each form. Four are rendered each by its own launch of the persistent kernel compiled for it (batch_group), four
// each by its own run of the wavefront's steps (wave_batch_group), as wavefront_suits says; and four by the pool kernel
// (pool_batch_group: the books' jobs of tree-searched scenes, and in the continuous server's refinement, whose images
// follow a session's roundings, of flat ones).
constexpr int persistent_groups = 4;
constexpr int batch_groups = 12;
RTB_HD constexpr int batch_group(bool flat, bool features) { return (flat ? 0 : 2) + (features ? 1 : 0); }
RTB_HD constexpr int wave_batch_group(bool flat, bool features) { return persistent_groups + batch_group(flat, features); }
RTB_HD constexpr int pool_batch_group(bool flat, bool features)
{
    return 2 * persistent_groups + batch_group(flat, features);
}

struct batch_header
{
    int64_t total_pixels;
    int64_t group_items[batch_groups + 1]; // group g's items are [group_items[g], group_items[g + 1])
    int32_t group_jobs[batch_groups + 1];  // and its jobs [group_jobs[g], group_jobs[g + 1])
    int32_t job_count;
    int32_t pad0;
};

struct batch_params
{
    const batch_job* jobs;
    const batch_header* header;
    unsigned long long* work_counter; // one per group's launch
};

// The batch engine's groups of tree-searched jobs in the wavefront form: the jobs [job_first, job_end) of the table,
// their samples numbered from 0 (job j's from jobs[j].sample_begin) up to the wave_buffers' sample_count
struct wave_batch
{
    const batch_job* jobs;
    int32_t job_first;
    int32_t job_end;
    int64_t item_first; // the group's work items [item_first, item_end) in the batch's item space
    int64_t item_end;
    unsigned long long* work_counter; // the group's samples taken so far (zero at the start)
    // A stream run (the server's continuous wavefront; null in a batch's run): samples are claimed up to *published,
    // a claim beyond it waits in its slot until the host publishes that far; the jobs are segments in a ring of
    // job_mask + 1 entries, the window window[0] .. window[1] counted without wrapping (in device memory with the
    // limit, so that one captured graph of steps serves every group)
    const unsigned long long* published;
    int32_t job_mask;
    int32_t pad0;
    const int32_t* window;
    const int64_t* starts; // each ring entry's first sample (its sample_begin), compact for the claims' search
};

// The stream run's reduction: each item a segment's samples added, pixel by pixel in pass order, into its request's
// chunk accumulator, which goes into the request's sums at every chunk's end, after the first pass (the first frame)
// and at the target, as a session adds its chunk partials
struct stream_reduce_item
{
    const float4* values;
    double* sums;
    double* acc;
    int64_t local_begin; // the segment's samples [local_begin, local_end) of the request's pass-major numbering
    int64_t local_end;
    int64_t pixel_begin; // the item's pixels in the launch's pixel space
    int64_t target;
    int32_t padded_pixels;
    int32_t tiles_x;
    int32_t width;
    int32_t height;
    int32_t chunk;       // passes a chunk (16)
    int32_t pad0;
};
cudaError_t launch_stream_reduce(const stream_reduce_item* items, int32_t count, int64_t total_pixels,
                                 cudaStream_t stream);

// The kernels' static properties for kernel_info
struct kernel_attributes
{
    int registers;
    int local_bytes;
    int blocks_per_sm;
    int threads_per_block;
    int max_threads_per_sm;
    int multiprocessors;
};

// A kernel's registers, local memory and resident blocks (with `shared` bytes of dynamic shared memory a block), and the
// device's multiprocessors
cudaError_t function_attributes(const void* kernel, kernel_attributes& out, int shared = 0);

constexpr int render_block = 128;

cudaError_t launch_render(const launch_params& p, bool quality, bool counting, int grid, cudaStream_t stream);
cudaError_t launch_reduce(const reduce_params& p, cudaStream_t stream);
// The batched step: the persistent kernel of groups [first_group, end_group) over their jobs' items (grids[g]
// blocks each), and the reduction of every job's pixels
cudaError_t launch_batch(const batch_params& p, const int* grids, int first_group, int end_group, cudaStream_t stream);
cudaError_t launch_batch_reduce(const batch_params& p, int grid, cudaStream_t stream);
cudaError_t batch_attributes(int group, kernel_attributes& out);
// The attributes of the render kernel that launch_render picks for the scene and integrator
cudaError_t render_attributes(const scene_view& scene, bool quality, kernel_attributes& out);

// The wavefront form of a launch, for scenes searched through the tree: `slot_count` resident paths, each the state a
// lane of the persistent kernel keeps in registers (its sample, path and pending shadow ray), advanced by steps of two
// kernels. The shade kernel (one thread per slot) takes the last step's hits, shades, stores finished samples, claims
// new ones and queues each slot's next ray and shadow ray; the trace kernel (persistent) walks the queued rays, each
// lane taking the next query as soon as its own is answered. A step that queues nothing ends the launch, and the
// reduction adds the samples into the sums chunk by chunk, in pass order.
struct wave_buffers
{
    void* slots;            // slot_count slots of wave_slot_bytes() each, cleared before a launch
    int32_t slot_count;     // a multiple of render_block
    float4* samples;        // sample_count: (pass - pass_begin) * padded_pixels + tile slot -> the sample's value
    int64_t sample_count;   // (pass_end - pass_begin) * padded_pixels
    float4* query_o;        // 2 * slot_count queries: origin, time
    float4* query_d;        // direction, t_max
    int4* query_meta;       // from, flags (1 inward, 2 shadow, 4 a camera ray to make; the job << 3), skip, slot
    int4* ext_result;       // per slot: the next ray's hit (id, t's bits, front)
    int32_t* shadow_result; // per slot: 1 if the shadow ray was blocked
    // [0] next rays and shadow rays the last shade step queued (from the bottom), [1] queries the trace kernel took,
    // [2] camera rays it queued (from the top down; tree-searched scenes only); [3] a stream run's error flag (a claim
    // outside the window of segments it was given), never cleared by a step
    unsigned* control;
    camera_params cam;      // a session's launch: its camera and RNG job field (a batch: each job's, in its table)
    uint32_t job;
    int32_t draining;       // every sample is claimed: the shade kernel reads a slot's rows only if it has work
};
size_t wave_slot_bytes();
// Every slot without a sample (its flags row zeroed), before a launch's first step
cudaError_t clear_wave_slots(const wave_buffers& b, cudaStream_t stream);
using wave_shade_function = void (*)(launch_params, wave_buffers, wave_batch);
// A session's shade kernel under NEE/MIS without the second book's features (wave_quality.cu)
wave_shade_function quality_shade_kernel();

// How a session's wavefront step is launched (the autotuner's choice): the trace kernel's grid and register cap (its
// minimum resident blocks per multiprocessor: RTB_TRACE_MIN_BLOCKS or wave_trace_roomy_blocks), the shade kernel's
// block size (64 or 128 threads)
constexpr int wave_trace_roomy_blocks = 6;
#ifndef RTB_TRACE_MIN_BLOCKS_DEFAULT
#define RTB_TRACE_MIN_BLOCKS_DEFAULT 8
#endif
struct wave_shape
{
    int trace_grid;
    int shade_block;
    int trace_min_blocks;
};
// One step: clears the queue, the shade kernel over the slots, the trace kernel (shape.trace_grid blocks) over the queue
cudaError_t launch_wave_step(const launch_params& p, bool quality, const wave_buffers& b, const wave_shape& shape,
                             cudaStream_t stream, const cudaEvent_t* marks = nullptr, bool draining = false);
// The samples of passes [pass_begin, pass_end) into the sums (chunk partials in pass order, added in chunk order)
cudaError_t launch_wave_reduce(const reduce_params& r, const wave_buffers& b, int64_t pass_begin, int64_t pass_end,
                               int32_t chunk, cudaStream_t stream);
// The same for a group of batch jobs (flat: the group's scenes are searched flat; features: its kernels compile the
// second book's features; wide: every job's tree is four wide; quality: some job uses the NEE/MIS integrator, which
// the shade kernel then picks per job, where a group of books' jobs only gets a kernel without that code), and the
// group's samples into its jobs' chunk partials (then the batch's reduction adds them into the sums)
cudaError_t launch_wave_batch_step(const wave_batch& w, bool flat, bool features, bool wide, bool quality,
                                   const wave_buffers& b, int trace_grid, cudaStream_t stream,
                                   bool draining = false);
cudaError_t launch_wave_batch_partials(const wave_batch& w, const wave_buffers& b, cudaStream_t stream);
// Loads the batch wavefront's kernels (every variant) now, so that no step pays for loading them
cudaError_t preload_wave_batch();
// The shade kernel's and the trace kernel's attributes for the scene and integrator
// The shade kernel's and the session's trace kernel's attributes (the trace kernel of the scene's search, at the given
// register cap)
cudaError_t wave_attributes(const scene_view& scene, bool quality, kernel_attributes& shade, kernel_attributes& trace,
                            int trace_min_blocks = RTB_TRACE_MIN_BLOCKS_DEFAULT);

// A launch of the pool kernel (the wavefront within a warp): each warp keeps its paths in shared memory and walks,
// shades and starts them a warp's worth at a time. The samples' values go to `samples` as the wavefront's do.
struct pool_run
{
    float4* samples;
    int64_t sample_count;
    int32_t claim; // samples a warp claims at a time, 1..32
    int32_t pad0;
};
// Whether a session's AUTO renders a scene by the pool kernel: one searched flat, or through a tree four wide; nor a bare
// small scene under NEE/MIS, nor an empty one. (The bare small scenes lost 40% in the wavefront's steps: quads 397x401 x
// 100 2.02 ms in the persistent kernel, 0.96 here; materials 800x450 x 64 6.77 and 2.82.) With triangles, only under
// NEE/MIS without the second book's features, the kernel whose image is checked against the steps'.
inline bool pool_suits(const scene_view& v, bool quality)
{
    const bool searched = v.node_count > 0 && (v.flat != 0 || v.wide_nodes != nullptr);
    const bool triangles = v.prim_count > v.triangle_base;
    return searched && (wavefront_suits(v) || !quality) && (!triangles || (quality && !has_features(v)));
}
// The launches it renders: all, but with triangles those of up to 2^20 samples per unit of depth, and with volumes beside
// a tree 2^22. (The line follows the smaller mesh, where the steps are ahead above it; the larger crosses later, and a
// launch of it between the two, as at depth 50 with 66M, is 10 to 20% slower in the steps that the rule gives it to. The
// crossing moves with the mesh's size, which the rule does not read.) A mesh's shading (rough metal, coat, environment) waits for its instructions beside the walks', which the
// steps' shade kernel does less; the steps wait at each depth for their last walks. The mesh of 1,280 triangles at depth 6
// with 3.7M samples 2.42 ms here and 2.44 in the steps, with 14.7M 9.1 and 8.0, at depth 50 with 14.7M 11.2 and 16.2, with
// 66M 38.8 and 36.9; that of 1.3M at depth 6 with 7.4M 6.1 and 6.9, with 29M 20.7 and 19.3, at depth 50 with 66M 50 and
// 60. The second book's final scene at depth 2 with 1.4M 0.67 and 0.95, with 23M 9.3 and 8.9, at depth 50 with 23M 23.4
// and 28.6.
inline int64_t pool_most_samples(const scene_view& v, int max_depth)
{
    const int64_t depth = max_depth < 64 ? max_depth : 64;
    const bool triangles = v.prim_count > v.triangle_base;
    const bool volumes = v.medium_count > 0 && v.flat == 0;
    return triangles ? depth << 20 : volumes ? depth << 22 : INT64_MAX;
}
// A bare small scene's single pass of up to this many samples is the persistent kernel's: each of its lanes takes one
// sample, and there is no samples buffer to reduce (quads 64x64 35 us there and 39 here, 236x650 50 and 56, materials
// 64x64 80 and 87; above, and with more passes, which a lane takes in turn, the pool kernel: quads 1280x720 96 and 95,
// two passes of materials 811x274 208 and 167)
constexpr int64_t pool_least_bare_samples = int64_t{1} << 18;
using pool_function = void (*)(launch_params, pool_run, wave_batch);
struct pool_program
{
    pool_function kernel;
    int shared; // dynamic shared memory, bytes a block
};
// The kernel's attributes; and its shared memory allowed on the current device, before its first launch there
cudaError_t pool_program_attributes(const pool_program& program, kernel_attributes& out);
pool_program quality_pool_program(bool features, bool flat, bool mesh); // under NEE/MIS (pool_quality.cu)
pool_program bare_pool_program(); // a scene that does not suit the wavefront (pool_bare.cu)
// Claims, renders and writes out every sample of the launch (`grid` blocks fill the GPU; a small launch takes fewer)
cudaError_t launch_pool(const launch_params& p, bool quality, float4* samples, int64_t sample_count, int grid,
                        cudaStream_t stream);
cudaError_t pool_attributes(const scene_view& scene, bool quality, kernel_attributes& out);
// The same for a batch's group of books' jobs, searched flat or through trees four wide (w's jobs, their samples
// numbered from 0)
cudaError_t launch_pool_batch(const wave_batch& w, bool flat, bool features, float4* samples, int64_t sample_count, int grid,
                              cudaStream_t stream);
cudaError_t pool_batch_attributes(bool flat, bool features, kernel_attributes& out);
// The work counter cleared before a launch, and the launch's shape for its samples
struct pool_launch
{
    int32_t claim;
    unsigned blocks;
};
cudaError_t prepare_pool(unsigned long long* work_counter, cudaStream_t stream);
pool_launch pool_launch_of(int64_t sample_count, int grid);

// The books' integrator in double (precision::float64; renderer.h:402-409, all_books_kernel<double>,
// renderer.cu:445-451): the samples of launch_params' passes and pixels by a pool kernel in double, their values added
// into the sums by launch_reduce_f64 as launch_wave_reduce adds a float launch's. Its own random numbers: 53-bit
// uniforms.
struct launch_params_f64
{
    scene_view_f64 scene;
    camera_d cam;
    uint64_t seed;
    int64_t pass_begin;
    int64_t pass_end;
    int64_t sample_count;   // (pass_end - pass_begin) * band_pixels
    int32_t chunk;
    int32_t tiles_x;
    int32_t first_pixel;    // the band of the padded image's pixels this launch renders, whole tiles
    int32_t band_pixels;
    int32_t round_passes;
    int32_t claim;          // set by the launch
    int32_t pad0;
    unsigned long long* work_counter;
    double* samples;              // 3 a sample
    unsigned long long* counters; // [0] path segments
    unsigned long long* tied;     // not 0: a path of the view so far met several primitives at one distance
};
// (`kernels` grows by those launched)
cudaError_t launch_render_f64(const launch_params_f64& p, int grid, cudaStream_t stream, int32_t& kernels);
cudaError_t launch_reduce_f64(const launch_params_f64& p, double* sums, cudaStream_t stream);
cudaError_t render_f64_attributes(const scene_view_f64& scene, kernel_attributes& out);

// Parity hooks: closest hits of given rays (source ids through prim_source), and the camera rays of one pass
cudaError_t launch_closest_hits(const scene_view& s, const float* origins, const float* directions, int64_t count,
                                const int32_t* prim_source, int32_t* ids, float* ts, cudaStream_t stream);
cudaError_t launch_camera_rays(const camera_params& cam, uint64_t seed, int64_t pass, int32_t round_passes,
                               float* origins, float* directions, cudaStream_t stream);
} // namespace rtb
