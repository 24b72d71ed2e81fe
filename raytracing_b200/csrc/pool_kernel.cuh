// The pool kernel: the wavefront within a warp. Included after path.cuh by each source that compiles it.
//
// A persistent warp keeps 64 or 96 paths in shared memory and, in turn, walks rays (32 lanes, each with a path of its own),
// shades answered paths and starts new samples, each phase with as full a warp as the lists hold; a path is never bound
// to a lane between phases. What it replaces: the wavefront's steps keep up to 3 x 2^20 paths in HBM and run two kernels
// a step over all of them, so every segment paid 160 to 224 bytes of HBM traffic and a round through a queue, and every
// launch ended with a drain of a path's length of nearly empty steps (a 400x225, 32-pass cover render spent 4.4 ms in
// 128 steps for 1.3 ms of work). Against the one-lane-one-path persistent kernel, shading and searches run with full
// warps. Bound by instruction issue, with the lanes that materials and walks of uneven depth leave idle.
// Measured on the B200, GPU time, against the steps (images equal bit for bit): glass 600x600 x 1024 173 -> 96 ms,
// cornell-mis x 256 109 -> 58, weekend 400x225 x 32 4.36 -> 1.27, one pass of weekend at 256x256 1.35 -> 0.25,
// final 400x400 x 100 19.9 -> 17.0, smoke 300x300 x 64 5.8 -> 1.9, checker 400x225 x 64 4.9 -> 0.85.

// A path's record in shared memory, as words of a structure of arrays ([word][path]): a warp's reads of a word touch
// consecutive banks but for the paths' order
template <bool QUALITY, bool FEATURES, bool BATCH>
struct pool_record
{
    static constexpr int o = 0;          // origin
    static constexpr int d = 3;          // direction
    static constexpr int throughput = 6;
    static constexpr int pixel = 9;      // the random numbers' counter and key: pixel, pass in its round, key's high word
    static constexpr int pass = 10;
    static constexpr int key = 11;
    static constexpr int sample = 12;    // the sample's number in the launch (a batch: within its job)
    static constexpr int meta = 13;      // depth << 6 and the flags below
    static constexpr int from = 14;      // the primitive the ray leaves
    static constexpr int hit_t = 15;     // the walk's answer
    static constexpr int hit = 16;       // id << 1 | front, or -1
    static constexpr int time = 17;
    static constexpr int job = time + (FEATURES ? 1 : 0);
    static constexpr int radiance = job + (BATCH ? 1 : 0);
    static constexpr int pdf = radiance + 3;
    static constexpr int shadow_d = pdf + 1;
    static constexpr int shadow_t = shadow_d + 3;
    static constexpr int light = shadow_t + 1; // what the shadow ray brings if nothing blocks it
    static constexpr int skip = light + 3;
    static constexpr int words = QUALITY ? skip + 1 : radiance;
};
constexpr uint32_t pool_inward = 1u;        // the ray starts inside the surface it leaves
constexpr uint32_t pool_specular = 2u;
constexpr uint32_t pool_ext = 4u;           // the path goes on: its next ray is to be walked
constexpr uint32_t pool_shadow = 8u;        // a shadow ray is to be walked (before the next ray)
constexpr uint32_t pool_shadow_inward = 16u;
constexpr uint32_t pool_blocked = 32u;      // the shadow ray's answer, where the shading needs it (smoke)

// A kernel's shape, swept on the B200 for each kind of scene: the resident blocks, which cap its registers; a warp's paths
// (twice its lanes, so that while up to 32 of them walk, enough others wait for a full warp's shading); and the lists
// its answered paths wait in, by what their shading runs (shade_ends ...), so that a warp shades like with like: three
// lists want more paths, whose shared memory a flat scene can spare. GPU times of each rule's line:
// * flat scenes {8 blocks, 64 paths, 1 list} -> {7, 96, 3}: glass 600x600 x 64 7.13 -> 6.19 ms; {8, 96, 3} 6.30, {6, 128,
//   3} 6.57, {7, 96, 2} 6.91. With the second book's features {6, 64, 1} -> {6, 96, 3}: smoke 1.67 -> 1.57.
// * bare flat scenes {8, 64, 1} -> {8, 96, 2}: quads 0.92 -> 0.87, materials 1.41 -> 1.34.
// * the books' trees keep one list: three cost weekend 3.03 -> 3.14 and its 256x256 first frame 0.237 -> 0.277 (fewer
//   lanes a phase); 8 blocks against 7: 6.32 -> 6.18; with the features 6 against 5: final 11.25 -> 10.4. A batch, whose
//   jobs' scenes and cameras take registers: 7 (16 cover jobs 20.7, 19.8, 19.0, 19.7 ms at 5, 6, 7, 8).
// * NEE/MIS one list too (cornell-mis 6.65; three 7.4): flat 6 blocks (5: +4%), trees and features 5 (6 spills: +8%).
// * a mesh under NEE/MIS {5, 64, 1} -> {4, 96, 3, 12}: the 1.3M triangles at 1280x720 x 16 14.9 -> 10.8; {5, 80, 3} 11.3,
//   {6, 64, 3} 11.5, {3, 128, 3} 12.2, {2, 192, 3} 14.9; walks broken off at 20 lanes 10.9.
struct pool_shape
{
    int blocks;  // resident per multiprocessor
    int paths;   // a warp's
    int classes; // lists of answered paths
    int refill;  // the lanes still walking under which a warp stops its walks to give the others something to do
};

template <bool QUALITY, bool FEATURES, bool FLAT, bool BATCH, bool MESH>
RTB_HD constexpr pool_shape pool_shape_of()
{
    if (MESH)
    {
        return {4, 96, 3, 12};
    }
    if (QUALITY)
    {
        return {FLAT && !FEATURES ? 6 : 5, 64, 1, 20};
    }
    if (FLAT && !BATCH)
    {
        if (rounds::bare)
        {
            return {8, 96, 2, 20};
        }
        return {FEATURES ? 6 : 7, 96, 3, 20};
    }
    if (BATCH)
    {
        return {FEATURES ? 5 : 7, 64, 1, 20};
    }
    return {FEATURES ? 6 : 8, 64, 1, 20};
}

template <bool QUALITY, bool FEATURES, bool FLAT, bool BATCH, bool MESH = false>
__global__ void __launch_bounds__(render_block, pool_shape_of<QUALITY, FEATURES, FLAT, BATCH, MESH>().blocks)
    pool_kernel(const __grid_constant__ launch_params P, const __grid_constant__ pool_run R,
                const __grid_constant__ wave_batch W)
{
    using record = pool_record<QUALITY, FEATURES, BATCH>;
    constexpr int pool_paths = pool_shape_of<QUALITY, FEATURES, FLAT, BATCH, MESH>().paths;
    constexpr int shade_classes = pool_shape_of<QUALITY, FEATURES, FLAT, BATCH, MESH>().classes;
    constexpr int refill = pool_shape_of<QUALITY, FEATURES, FLAT, BATCH, MESH>().refill;
    constexpr int warps = render_block / 32;
    extern __shared__ uint32_t pool_memory[];
    auto& records = *reinterpret_cast<uint32_t(*)[warps][record::words][pool_paths]>(pool_memory);
    auto& lists = *reinterpret_cast<uint8_t(*)[warps][2 + shade_classes][pool_paths]>(pool_memory + warps * record::words * pool_paths);
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    const int warp = static_cast<int>(threadIdx.x >> 5);
    uint32_t(*const rec)[pool_paths] = records[warp];
    uint8_t* const walk_list = lists[warp][0];  // paths with a ray to walk
    uint8_t* const free_list = lists[warp][1];  // records without a sample
    uint8_t* const shade_list = lists[warp][2]; // paths with an answer to shade, a list for each class of vertex
    const auto put3 = [&](int word, int p, float3 v) {
        rec[word][p] = __float_as_uint(v.x);
        rec[word + 1][p] = __float_as_uint(v.y);
        rec[word + 2][p] = __float_as_uint(v.z);
    };
    const auto get3 = [&](int word, int p) {
        return make_float3(__uint_as_float(rec[word][p]), __uint_as_float(rec[word + 1][p]),
                           __uint_as_float(rec[word + 2][p]));
    };
    // The lanes for which `which` holds append their path to a list; its new length
    const auto push = [&](uint8_t* list, int count, bool which, int p) -> int {
        const unsigned lanes = __ballot_sync(full_warp, which);
        if (which)
        {
            list[count + __popc(lanes & lanes_below)] = static_cast<uint8_t>(p);
        }
        return count + __popc(lanes);
    };
    for (int p = static_cast<int>(lane); p < pool_paths; p += 32)
    {
        free_list[p] = static_cast<uint8_t>(p);
    }
    int walk_count = 0;
    int shade_count[shade_classes] = {};
    int free_count = pool_paths;
    const auto limit = static_cast<unsigned long long>(R.sample_count);
    bool dry = limit == 0ull; // every sample of the launch is claimed
    uint32_t rays = 0, shadow_rays = 0;
    __syncwarp();

    // The lane's walk (tree-searched scenes): the path it walks for (-1: none) and the walk's state
    int slot = -1;
    bool shadow = false;
    int link = traversal_done;
    int leaf = 0;
    int sp = 0;
    hit_info hit{-1, 0.0f, false};
    int2 stack[FLAT ? 1 : wide_stack];

    // The lanes for which `which` holds append their path to its class's list
    const auto to_shade_lists = [&](bool which, int shade_class, int p) {
#pragma unroll
        for (int c = 0; c < shade_classes; ++c)
        {
            shade_count[c] = push(shade_list + c * pool_paths, shade_count[c], which && shade_class == c, p);
        }
    };
    const auto fullest = [&]() -> int {
        int best = 0;
#pragma unroll
        for (int c = 1; c < shade_classes; ++c)
        {
            best = shade_count[c] > shade_count[best] ? c : best;
        }
        return best;
    };
    const auto waiting = [&]() -> int {
        int n = 0;
#pragma unroll
        for (int c = 0; c < shade_classes; ++c)
        {
            n += shade_count[c];
        }
        return n;
    };
    const auto class_of = [&](const scene_view& S, int id) -> int {
        const int c = id < 0 ? shade_ends : __ldg(S.prim_class + id);
        return c < shade_classes ? c : shade_classes - 1;
    };

    const auto job_of = [&](int p) -> const batch_job* { return BATCH ? W.jobs + rec[record::job][p] : nullptr; };

    while (true)
    {
        enum class phase
        {
            walk,
            start,
            shade,
            end
        } next;
        float3 o = make_float3(0.0f, 0.0f, 0.0f);
        float3 d = o;
        float time = 0.0f;
        int from = -1, skip = -1;
        bool inward = false;
        if constexpr (!FLAT)
        {
            // The answered walks: a shadow ray's light is added (or lost), then its path's next ray is walked by the
            // same lane; a next ray's hit goes to the shading
            const bool answered = slot >= 0 && link == traversal_done && leaf == 0;
            bool fresh = false;
            bool to_shade = false, to_free = false;
            int shade_class = 0;
            const int was = slot;
            if (answered)
            {
                if (QUALITY && shadow)
                {
                    uint32_t meta = rec[record::meta][slot];
                    if constexpr (FEATURES)
                    {
                        meta |= hit.id >= 0 ? pool_blocked : 0u;
                    }
                    else
                    {
                        meta &= ~pool_shadow;
                        if (hit.id < 0)
                        {
                            put3(record::radiance, slot, get3(record::radiance, slot) + get3(record::light, slot));
                        }
                    }
                    rec[record::meta][slot] = meta;
                    shadow = false;
                    if (meta & pool_ext)
                    {
                        fresh = true;
                    }
                    else if (FEATURES)
                    {
                        to_shade = true;
                        slot = -1;
                    }
                    else
                    {
                        const float3 sample = get3(record::radiance, slot);
                        const batch_job* J = job_of(slot);
                        stream_store(R.samples + (BATCH ? J->sample_begin : 0) + rec[record::sample][slot],
                                     make_float4(sample.x, sample.y, sample.z, 0.0f));
                        to_free = true;
                        slot = -1;
                    }
                }
                else
                {
                    rec[record::hit_t][slot] = __float_as_uint(hit.t);
                    rec[record::hit][slot] = hit.id < 0 ? 0xffffffffu
                                                        : (static_cast<uint32_t>(hit.id) << 1) | (hit.front ? 1u : 0u);
                    to_shade = true;
                    shade_class = class_of(BATCH ? job_of(slot)->scene : P.scene, hit.id);
                    slot = -1;
                }
            }
            to_shade_lists(to_shade, shade_class, was);
            if (QUALITY && !FEATURES)
            {
                free_count = push(free_list, free_count, to_free, was);
            }
            // New rays for the idle lanes
            const unsigned idle = __ballot_sync(full_warp, slot < 0);
            const int taken = min(__popc(idle), walk_count);
            const int rank = __popc(idle & lanes_below);
            __syncwarp();
            if (slot < 0 && rank < taken)
            {
                slot = walk_list[walk_count - 1 - rank];
                fresh = true;
                shadow = QUALITY && (rec[record::meta][slot] & pool_shadow) != 0u;
            }
            walk_count -= taken;
            if (fresh)
            {
                hit = {-1, QUALITY && shadow ? __uint_as_float(rec[record::shadow_t][slot]) : infinity_f, false};
                sp = 0;
                leaf = 0;
                const scene_view& S = BATCH ? job_of(slot)->scene : P.scene;
                link = S.node_count == 0 ? traversal_done : 0;
            }
            const int walking = __popc(__ballot_sync(full_warp, slot >= 0));
            const int startable = dry ? 0 : free_count;
            // Few walks left and no ray to refill the lanes with: shade or start, whichever has the fuller warp
            const bool few = walking < refill && walking * 8 < (walking + waiting() + startable) * 5;
            if (walk_count == 0 && few)
            {
                next = startable > shade_count[fullest()] ? phase::start : phase::shade;
            }
            else
            {
                next = walking > 0 ? phase::walk : phase::end;
            }
        }
        else
        {
            const int startable = dry ? 0 : free_count;
            const int shadeable = shade_count[fullest()];
            if (walk_count >= 32 || (walk_count >= startable && walk_count >= shadeable))
            {
                next = walk_count > 0 ? phase::walk : phase::end;
            }
            else
            {
                next = startable > shadeable ? phase::start : phase::shade;
            }
        }
        if (next == phase::end)
        {
            break;
        }
        if (next == phase::walk)
        {
            if constexpr (FLAT)
            {
                const int taken = min(32, walk_count);
                const bool mine = static_cast<int>(lane) < taken;
                const int p = mine ? walk_list[walk_count - taken + static_cast<int>(lane)] : 0;
                walk_count -= taken;
                bool to_shade = false, to_free = false;
                int shade_class = 0;
                if (mine)
                {
                    const batch_job* J = job_of(p);
                    const scene_view& S = BATCH ? J->scene : P.scene;
                    uint32_t meta = rec[record::meta][p];
                    o = get3(record::o, p);
                    time = FEATURES ? __uint_as_float(rec[record::time][p]) : 0.0f;
                    from = static_cast<int>(rec[record::from][p]);
#pragma unroll 1
                    for (int k = QUALITY ? 0 : 1; k < 2; ++k)
                    {
                        // the shadow ray first, then the next ray
                        const bool any = QUALITY && k == 0;
                        if ((meta & (any ? pool_shadow : pool_ext)) == 0u)
                        {
                            continue;
                        }
                        d = get3(QUALITY && any ? record::shadow_d : record::d, p);
                        hit_info h{-1, QUALITY && any ? __uint_as_float(rec[record::shadow_t][p]) : infinity_f, false};
                        flat_search<FEATURES>(S, o, d, time, from,
                                              (meta & (any ? pool_shadow_inward : pool_inward)) != 0u,
                                              QUALITY && any ? static_cast<int>(rec[record::skip][p]) : -1, any, h);
                        if (!any)
                        {
                            rec[record::hit_t][p] = __float_as_uint(h.t);
                            rec[record::hit][p] = h.id < 0 ? 0xffffffffu
                                                           : (static_cast<uint32_t>(h.id) << 1) | (h.front ? 1u : 0u);
                            shade_class = class_of(S, h.id);
                        }
                        else if (FEATURES)
                        {
                            meta |= h.id >= 0 ? pool_blocked : 0u;
                        }
                        else
                        {
                            meta &= ~pool_shadow;
                            if (h.id < 0)
                            {
                                put3(record::radiance, p, get3(record::radiance, p) + get3(record::light, p));
                            }
                        }
                    }
                    to_shade = true;
                    if (QUALITY)
                    {
                        rec[record::meta][p] = meta;
                        if (!FEATURES && (meta & pool_ext) == 0u)
                        {
                            const float3 sample = get3(record::radiance, p);
                            stream_store(R.samples + (BATCH ? J->sample_begin : 0) + rec[record::sample][p],
                                         make_float4(sample.x, sample.y, sample.z, 0.0f));
                            to_shade = false;
                            to_free = true;
                        }
                    }
                }
                to_shade_lists(to_shade, shade_class, p);
                if (QUALITY && !FEATURES)
                {
                    free_count = push(free_list, free_count, to_free, p);
                }
            }
            else
            {
                // The walks: the trace kernel's, until too few lanes walk or all are answered
                const scene_view& S = BATCH && slot >= 0 ? job_of(slot)->scene : (BATCH ? W.jobs[W.job_first].scene : P.scene);
                const bvh4_node* const tree = S.wide_nodes;
                float inverse_a = 0.0f;
                wide_ray ray{};
                if (slot >= 0)
                {
                    const uint32_t meta = rec[record::meta][slot];
                    o = get3(record::o, slot);
                    d = get3(QUALITY && shadow ? record::shadow_d : record::d, slot);
                    time = FEATURES ? __uint_as_float(rec[record::time][slot]) : 0.0f;
                    from = static_cast<int>(rec[record::from][slot]);
                    skip = QUALITY && shadow ? static_cast<int>(rec[record::skip][slot]) : -1;
                    inward = (meta & (QUALITY && shadow ? pool_shadow_inward : pool_inward)) != 0u;
                    // (a batch's kernel with the features may render a scene without them too: rounded as its own does)
                    const bool features = FEATURES && (!BATCH || has_features(S));
                    inverse_a = 1.0f / (features ? length_squared<rounds::walk_features>(d) : length_squared(d));
                    ray = wide_ray_of(o, d);
                }
                const bool has_query = slot >= 0;
                const auto pop = [&]() -> int {
                    while (sp > 0)
                    {
                        const int2 e = stack[--sp];
                        if ((QUALITY && shadow) || __int_as_float(e.y) < hit.t)
                        {
                            return e.x;
                        }
                    }
                    return traversal_done;
                };
                const int total = __popc(__ballot_sync(full_warp, has_query)) + walk_count + waiting() +
                                  (dry ? 0 : free_count);
                const int enough = min(refill, (total * 5 + 7) / 8);
                while (true)
                {
                    while (true)
                    {
                        const bool descending = has_query && link >= 0;
                        if (!__any_sync(full_warp, descending))
                        {
                            break;
                        }
                        if (descending)
                        {
                            link = wide_step(tree, link, ray, hit.t, stack, sp, pop);
                            if (link < 0 && link != traversal_done && leaf == 0)
                            {
                                leaf = link;
                                link = pop();
                            }
                        }
                        if (!__any_sync(full_warp, has_query && link >= 0 && leaf == 0))
                        {
                            break;
                        }
                    }
                    while (true)
                    {
                        const bool testing = has_query && leaf < 0;
                        if (!__any_sync(full_warp, testing))
                        {
                            break;
                        }
                        if (testing)
                        {
                            if (test_leaf<false, false, FEATURES>(S, leaf, o, d, time, inverse_a, from, inward, skip, hit,
                                                                  nullptr, QUALITY && shadow))
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
                    const int walking =
                        __popc(__ballot_sync(full_warp, has_query && !(link == traversal_done && leaf == 0)));
                    if (walking < enough)
                    {
                        break;
                    }
                }
            }
            __syncwarp();
            continue;
        }
        if (next == phase::start)
        {
            // New samples, a warp's worth of consecutive numbers at a time: a tile's pixels, their camera rays made
            // side by side
            const int wanted = min(min(32, free_count), R.claim);
            unsigned long long base = 0;
            if (lane == 0u)
            {
                base = atomicAdd(BATCH ? W.work_counter : P.work_counter, static_cast<unsigned long long>(wanted));
            }
            base = __shfl_sync(full_warp, base, 0);
            dry = base + static_cast<unsigned long long>(wanted) >= limit;
            const unsigned long long s = base + lane;
            bool started = static_cast<int>(lane) < wanted && s < limit;
            int job = 0;
            const batch_job* J = nullptr;
            if (BATCH && started)
            {
                job = find_job<job_samples>(W.jobs, W.job_first, W.job_end, static_cast<int64_t>(s));
                J = W.jobs + job;
            }
            const camera_params& cam = BATCH && started ? J->cam : P.cam;
            const int64_t index = static_cast<int64_t>(s) - (BATCH && started ? J->sample_begin : 0);
            sample_place at{0, 0, 0};
            if (started)
            {
                at = place_of(index, cam, BATCH ? J->pass_begin : P.pass_begin, BATCH ? J->first_pixel : 0);
                started = at.x < cam.width && at.y < cam.height; // a lane of a tile over the image's edge: no sample
            }
            const unsigned lanes = __ballot_sync(full_warp, started);
            const int p = started ? free_list[free_count - 1 - __popc(lanes & lanes_below)] : 0;
            __syncwarp();
            free_count -= __popc(lanes);
            if (started)
            {
                sampler rng;
                rng.job = BATCH ? J->job : P.job;
                const int round_pass = sample_rng(at, cam, BATCH ? J->seed : P.seed, rng);
                int s_i, s_j;
                stratum_of(cam, round_pass, s_i, s_j);
                camera_ray(cam, at.x, at.y, s_i, s_j, rng.draw(0, 0), o, d);
                put3(record::o, p, o);
                put3(record::d, p, d);
                put3(record::throughput, p, make_float3(1.0f, 1.0f, 1.0f));
                rec[record::pixel][p] = rng.pixel;
                rec[record::pass][p] = rng.pass;
                rec[record::key][p] = rng.key.y;
                rec[record::sample][p] = static_cast<uint32_t>(index);
                rec[record::meta][p] = pool_specular | pool_ext;
                rec[record::from][p] = 0xffffffffu;
                if constexpr (FEATURES)
                {
                    const scene_view& S = BATCH ? J->scene : P.scene;
                    rec[record::time][p] = __float_as_uint(S.has_motion ? rng.draw(0, block_time).x : 0.0f);
                }
                if constexpr (BATCH)
                {
                    rec[record::job][p] = static_cast<uint32_t>(job);
                }
                if constexpr (QUALITY)
                {
                    put3(record::radiance, p, make_float3(0.0f, 0.0f, 0.0f));
                    rec[record::pdf][p] = 0u;
                }
            }
            walk_count = push(walk_list, walk_count, started, p);
            if constexpr (BATCH)
            {
                const unsigned peers = __match_any_sync(full_warp, started ? job : -1);
                if (started && (peers & lanes_below) == 0u)
                {
                    atomicAdd(J->counters, static_cast<unsigned long long>(__popc(peers)));
                }
            }
            else
            {
                rays += static_cast<uint32_t>(__popc(lanes));
            }
            __syncwarp();
            continue;
        }
        // The shading of the answered paths, as the wavefront's shade kernel does it
        const int which = fullest();
        const int taken = min(32, shade_count[which]);
        const bool mine = static_cast<int>(lane) < taken;
        const int p = mine ? shade_list[which * pool_paths + shade_count[which] - taken + static_cast<int>(lane)] : 0;
#pragma unroll
        for (int c = 0; c < shade_classes; ++c)
        {
            shade_count[c] -= c == which ? taken : 0;
        }
        bool goes_on = false;
        bool lit = false;
        int job = 0;
        const batch_job* J = nullptr;
        if (mine)
        {
            job = BATCH ? static_cast<int>(rec[record::job][p]) : 0;
            J = BATCH ? W.jobs + job : nullptr;
            const scene_view& S = BATCH ? J->scene : P.scene;
            const camera_params& cam = BATCH ? J->cam : P.cam;
            const uint32_t meta = rec[record::meta][p];
            path_state ps;
            ps.o = get3(record::o, p);
            ps.d = get3(record::d, p);
            ps.throughput = get3(record::throughput, p);
            ps.radiance = QUALITY ? get3(record::radiance, p) : make_float3(0.0f, 0.0f, 0.0f);
            ps.bsdf_pdf = QUALITY ? __uint_as_float(rec[record::pdf][p]) : 0.0f;
            ps.specular = (meta & pool_specular) != 0u;
            ps.inward = (meta & pool_inward) != 0u;
            ps.depth = static_cast<int>(meta >> 6);
            ps.rays_left = cam.max_depth - ps.depth;
            ps.from = static_cast<int>(rec[record::from][p]);
            ps.time = FEATURES ? __uint_as_float(rec[record::time][p]) : 0.0f;
            sampler rng;
            rng.pixel = rec[record::pixel][p];
            rng.pass = rec[record::pass][p];
            rng.key = make_uint2(static_cast<uint32_t>(BATCH ? J->seed : P.seed), rec[record::key][p]);
            rng.job = BATCH ? J->job : P.job;
            float3 sample = make_float3(0.0f, 0.0f, 0.0f);
            bool finished = false;
            shadow_query sq;
            sq.lit = false;
            if constexpr (QUALITY && FEATURES)
            {
                if (meta & pool_shadow)
                {
                    if ((meta & pool_blocked) == 0u)
                    {
                        const float through = S.medium_count > 0
                                                  ? transmittance(S, ps.o, get3(record::shadow_d, p), ps.time,
                                                                  __uint_as_float(rec[record::shadow_t][p]))
                                                  : 1.0f;
                        ps.radiance = ps.radiance + through * get3(record::light, p);
                    }
                    if ((meta & pool_ext) == 0u)
                    {
                        sample = ps.radiance;
                        finished = true;
                    }
                }
            }
            if (!finished)
            {
                const uint32_t answer = rec[record::hit][p];
                hit_info h;
                h.id = static_cast<int>(answer) < 0 ? -1 : static_cast<int>(answer >> 1);
                h.t = __uint_as_float(rec[record::hit_t][p]);
                h.front = (answer & 1u) != 0u;
                ++ps.depth;
                if (FEATURES && S.medium_count > 0)
                {
                    media_event(S, ps.o, ps.d, ps.time, rng, ps.depth, h);
                }
                step_result res;
                if (QUALITY && (!BATCH || J->quality != 0))
                {
                    res = shade_quality<false, search_tree, FEATURES, true>(S, cam, rng, ps, h, sample, shadow_rays,
                                                                            nullptr, &sq);
                }
                else
                {
                    res = shade_books<FEATURES>(S, cam, rng, ps, h, sample);
                }
                goes_on = res == step_result::go_on;
                lit = QUALITY && sq.lit;
                finished = !goes_on && !lit;
                if (!finished)
                {
                    put3(record::o, p, QUALITY && !goes_on ? sq.o : ps.o);
                    put3(record::d, p, ps.d);
                    put3(record::throughput, p, ps.throughput);
                    rec[record::from][p] = static_cast<uint32_t>(QUALITY && !goes_on ? sq.from : ps.from);
                    rec[record::meta][p] = (static_cast<uint32_t>(ps.depth) << 6) | (ps.inward ? pool_inward : 0u) |
                                           (ps.specular ? pool_specular : 0u) | (goes_on ? pool_ext : 0u) |
                                           (lit ? pool_shadow : 0u) | (lit && sq.inward ? pool_shadow_inward : 0u);
                    if constexpr (QUALITY)
                    {
                        put3(record::radiance, p, ps.radiance);
                        rec[record::pdf][p] = __float_as_uint(ps.bsdf_pdf);
                        if (lit)
                        {
                            put3(record::shadow_d, p, sq.d);
                            rec[record::shadow_t][p] = __float_as_uint(sq.t_max);
                            put3(record::light, p, sq.contribution);
                            rec[record::skip][p] = static_cast<uint32_t>(sq.skip);
                        }
                    }
                }
            }
            if (finished)
            {
                stream_store(R.samples + (BATCH ? J->sample_begin : 0) + rec[record::sample][p],
                             make_float4(sample.x, sample.y, sample.z, 0.0f));
            }
        }
        const bool queued = goes_on || lit;
        walk_count = push(walk_list, walk_count, queued, p);
        free_count = push(free_list, free_count, mine && !queued, p);
        if constexpr (BATCH)
        {
            const unsigned on = __ballot_sync(full_warp, goes_on);
            const unsigned lights = __ballot_sync(full_warp, lit);
            const unsigned peers = __match_any_sync(full_warp, queued ? job : -1);
            if (queued && (peers & lanes_below) == 0u)
            {
                const unsigned e = __popc(peers & on), sh = __popc(peers & lights);
                if (e)
                {
                    atomicAdd(J->counters, static_cast<unsigned long long>(e));
                }
                if (sh)
                {
                    atomicAdd(J->counters + 1, static_cast<unsigned long long>(sh));
                }
            }
        }
        else
        {
            rays += static_cast<uint32_t>(__popc(__ballot_sync(full_warp, goes_on)));
        }
        __syncwarp();
    }
    if constexpr (!BATCH)
    {
        if (lane == 0u && rays != 0u)
        {
            atomicAdd(P.counters, static_cast<unsigned long long>(rays));
        }
        if constexpr (QUALITY)
        {
            const unsigned total = __reduce_add_sync(full_warp, shadow_rays);
            if (lane == 0u && total != 0u)
            {
                atomicAdd(P.counters + 1, static_cast<unsigned long long>(total));
            }
        }
    }
}

// The kernel's shared memory
template <bool QUALITY, bool FEATURES, bool FLAT, bool BATCH, bool MESH = false>
constexpr int pool_shared_bytes()
{
    constexpr pool_shape shape = pool_shape_of<QUALITY, FEATURES, FLAT, BATCH, MESH>();
    return render_block / 32 * shape.paths *
           (static_cast<int>(sizeof(uint32_t)) * pool_record<QUALITY, FEATURES, BATCH>::words + 2 + shape.classes);
}

template <bool QUALITY, bool FEATURES, bool FLAT, bool BATCH, bool MESH = false>
pool_program pool_program_of()
{
    return {pool_kernel<QUALITY, FEATURES, FLAT, BATCH, MESH>, pool_shared_bytes<QUALITY, FEATURES, FLAT, BATCH, MESH>()};
}
