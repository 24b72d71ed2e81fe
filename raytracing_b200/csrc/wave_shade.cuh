// The wavefront's slots and its shade kernel. Included after path.cuh by each source that compiles the kernel.

constexpr uint32_t wave_exhausted = 1u; // no work item left for the slot
constexpr uint32_t wave_ext = 2u;       // the path's next ray is queued (its hit comes back in ext_result)
constexpr uint32_t wave_shadow = 4u;    // a shadow ray is queued (blocked or not comes back in shadow_result)
constexpr uint32_t wave_finish = 8u;    // the sample ended at the shadow ray's vertex: it completes once the ray is in

// A slot in HBM, structure of arrays: five float4 rows of the path and its sample, three of its pending shadow ray,
// each row slot_count long, so that a warp's loads and stores of a row are 512 contiguous bytes. Rows: the ray's
// origin and time; its direction and the last BSDF density; the throughput and the radiance's red; the radiance's
// green and blue, the primitive the ray leaves and the rays left; the depth, the flags, the sample's number and the
// job. The sample's pass, pixel and random-number key are not stored: they follow from its number (sample_rng).
constexpr int wave_rows = 5;
constexpr int wave_shadow_rows = 3;
constexpr int wave_flags_row = 4; // depth, flags, sample, job: a slot whose row is zero has no sample
// A query's flags (its meta's second word): 1 the ray starts inside the surface it leaves, 2 a shadow ray, 4 a new
// sample's camera ray still to be made (a primary query); the job above them (<< 3)
constexpr int wave_query_primary = 4;
constexpr uint32_t wave_specular = 1u << 8;
constexpr uint32_t wave_inward = 1u << 9;
constexpr uint32_t wave_reserved = 1u << 10; // a stream run's slot holds a claim beyond what is published (its number
                                             // in the flags row's last two words) and waits for it

// ---- resident blocks -------------------------------------------------------------------------------------------
// The persistent render kernel's (kernels.cu) resident blocks per multiprocessor, which caps its registers, and which the
// shade kernel takes too unless its source chooses its own: the books' integrator at 64 (8
// blocks of 128 threads measured fastest against 5 and 6 blocks, for the latency they hide), the NEE/MIS integrator,
// whose GGX and environment code spills heavily at 64, at 80 (6 blocks); with the flat search (no tree stack) both
// at 72 (7 blocks), measured fastest against 5, 6 and 8 on the Cornell boxes
#ifndef RTB_MIN_BLOCKS
#define RTB_MIN_BLOCKS 8
#endif
#ifndef RTB_MIN_BLOCKS_QUALITY
#define RTB_MIN_BLOCKS_QUALITY 6
#endif
#ifndef RTB_MIN_BLOCKS_FLAT
#define RTB_MIN_BLOCKS_FLAT 7
#endif
#ifndef RTB_MIN_BLOCKS_QUALITY_FLAT
#define RTB_MIN_BLOCKS_QUALITY_FLAT 7
#endif
// The kernels of scenes with the second book's features (textures, motion, smoke): 96 registers (5 blocks), measured
// fastest against 72 and 80 on the final, smoke, perlin and light scenes (their textures and free flights spill)
#ifndef RTB_MIN_BLOCKS_FEATURES
#define RTB_MIN_BLOCKS_FEATURES 5 // 0: as the kernel without the features
#endif

template <bool QUALITY, bool FLAT, bool FEATURES>
constexpr int render_min_blocks()
{
    if (FEATURES && RTB_MIN_BLOCKS_FEATURES > 0)
    {
        return RTB_MIN_BLOCKS_FEATURES;
    }
    return QUALITY ? (FLAT ? RTB_MIN_BLOCKS_QUALITY_FLAT : RTB_MIN_BLOCKS_QUALITY)
                   : (FLAT ? RTB_MIN_BLOCKS_FLAT : RTB_MIN_BLOCKS);
}

// The shade kernel's resident blocks per multiprocessor: 0 takes the persistent kernel's for the integrator; a source may
// choose its own
#ifndef RTB_WAVE_SHADE_MIN_BLOCKS
#define RTB_WAVE_SHADE_MIN_BLOCKS 0
#endif
template <bool QUALITY, bool FEATURES>
constexpr int wave_shade_min_blocks()
{
    return RTB_WAVE_SHADE_MIN_BLOCKS > 0 ? RTB_WAVE_SHADE_MIN_BLOCKS : render_min_blocks<QUALITY, false, FEATURES>();
}


// A slot's step: the last walk's answers, the shading, the sample's end, a new sample, the next rays queued.
// BATCH: the slots render the samples of a group of batch jobs (W), each slot its job's scene, camera and integrator
// (with QUALITY each job's own, picked at run time; without, a group of books' jobs only, compiled without the NEE/MIS
// code); otherwise the launch's one view (P). A batch kernel keeps the NEE/MIS kernels' register budget either way:
// at the books' tighter one its per-job loads spill.
// Every load of the slot's rows and answer is issued at the start, before any of them is needed, so the step waits
// for one round trip to memory, not one for the flags and another for what they say to read.
template <bool QUALITY, bool FEATURES, bool BATCH>
__global__ void __launch_bounds__(render_block, wave_shade_min_blocks<QUALITY || BATCH, FEATURES>())
    wave_shade_kernel(const __grid_constant__ launch_params P, const __grid_constant__ wave_buffers B,
                      const __grid_constant__ wave_batch W)
{
    const int n = B.slot_count;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    float4* rows = static_cast<float4*>(B.slots);
    float4* shadow_rows = rows + static_cast<int64_t>(wave_rows) * n;
    const int own = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    // The slot's rows and its answer: all loads issued together while samples are left to claim (nearly every slot
    // has work); once every sample is claimed (the drain) the flags first, and the rest only for a slot with work
    float4 r0, r1, r2, r3;
    int4 r5, answer; // r5: the flags row
    // Compact slots, in a session's launch of a scene without the second book's features (nothing moves, so no time;
    // no job; the rays left are max_depth - depth): the depth and the six flags in one word of the flags row, which
    // also holds the sample's number, the primitive left and one more value. The books' paths carry no NEE radiance
    // or density: three rows, (origin, throughput x), (direction, throughput y), flags row (..., throughput z). The
    // NEE/MIS paths: four, (origin, NEE density), (direction, radiance r), (throughput, radiance g), flags row (...,
    // radiance b). A camera ray the trace kernel writes into rows 0 and 1 leaves their last words 0: no density, no
    // radiance. Row 3 (and for the books row 2) is neither read nor written.
    constexpr bool compact_slots = !BATCH && !FEATURES;
    constexpr bool books_slots = compact_slots && !QUALITY;
    int compact_from = -1;
    float compact_last = 0.0f; // the flags row's last word: throughput z (books) or radiance b (NEE/MIS)
    const auto load_flags = [&] {
        r5 = stream_load(reinterpret_cast<const int4*>(rows) + wave_flags_row * n + own);
        if constexpr (compact_slots)
        {
            // into the five-row form's (depth, flags, sample, job)
            const auto w = static_cast<uint32_t>(r5.x);
            compact_from = r5.z;
            compact_last = __int_as_float(r5.w);
            const uint32_t f = ((w & 1u) ? wave_ext : 0u) | ((w & 2u) ? wave_exhausted : 0u) |
                               ((w & 4u) ? wave_inward : 0u) | ((w & 8u) ? wave_specular : 0u) |
                               ((w & 16u) ? wave_shadow : 0u) | ((w & 32u) ? wave_finish : 0u);
            r5 = make_int4(static_cast<int>(w >> 6), static_cast<int>(f), r5.y, 0);
        }
    };
    const auto load_rest = [&] {
        r0 = stream_load(rows + own);
        r1 = stream_load(rows + n + own);
        if constexpr (!books_slots)
        {
            r2 = stream_load(rows + 2 * n + own);
        }
        if constexpr (!compact_slots)
        {
            r3 = stream_load(rows + 3 * n + own);
        }
        answer = stream_load(B.ext_result + own);
    };
    if (!B.draining)
    {
        load_rest();
        load_flags();
    }
    else
    {
        load_flags();
        if ((static_cast<uint32_t>(r5.y) & wave_exhausted) == 0u)
        {
            load_rest();
        }
        else
        {
            r0 = r1 = r2 = r3 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            answer = make_int4(0, 0, 0, 0);
        }
    }
    const int i = own; // the slot this thread shades
    uint32_t flags = static_cast<uint32_t>(r5.y);
    uint32_t shadow_rays = 0; // counted where the walks are (the trace kernel), or as queued (BATCH)
    // Samples may be claimed below `limit`: the launch's count, or what a stream run's host has published
    const bool stream_run = BATCH && W.published != nullptr;
    const unsigned long long limit =
        stream_run ? __ldcg(W.published) : static_cast<unsigned long long>(B.sample_count);
    const int2 window =
        stream_run ? __ldcg(reinterpret_cast<const int2*>(W.window)) : make_int2(W.job_first, W.job_end);
    // a warp whose slots have all run out of work has nothing left to do in this launch
    if (!__all_sync(full_warp, (flags & wave_exhausted) != 0u))
    {
        const bool live = (flags & wave_exhausted) == 0u;
        // the slot's job: its scene, camera and numbers (a session's launch: the launch's own)
        int job = BATCH && (flags & wave_reserved) == 0u ? r5.w : 0;
        const batch_job* J = BATCH ? W.jobs + job : nullptr;
        const auto scene = [&]() -> const scene_view& {
            if constexpr (BATCH)
            {
                return J->scene;
            }
            else
            {
                return P.scene;
            }
        };
        const auto camera = [&]() -> const camera_params& {
            if constexpr (BATCH)
            {
                return J->cam;
            }
            else
            {
                return P.cam;
            }
        };
        const auto quality = [&]() -> bool {
            if constexpr (BATCH)
            {
                return QUALITY && J->quality != 0; // a group of books' jobs only: no NEE/MIS code
            }
            else
            {
                return QUALITY;
            }
        };
        path_state ps;
        sampler rng;
        shadow_query sq;
        int64_t sample_index = 0, pass = 0;
        int px = 0, py = 0; // the pixel of a sample claimed in this step (a slot's camera ray needs no more)
        bool need = false;
        bool start = false;
        bool ready = false;             // a stream run's reservation the host has since published
        unsigned long long reserved = 0;
        int finished_job = -1;          // a stream run's segment whose sample this slot finished
        bool primary = false; // a new sample whose camera ray the trace kernel makes (wave_camera_query)
        int round_pass = 0;   // its pass within its round of strata
        rng.job = BATCH ? J->job : P.job;
        if (live)
        {
            ps.o = make_float3(r0.x, r0.y, r0.z);
            ps.time = r0.w;
            ps.d = make_float3(r1.x, r1.y, r1.z);
            ps.depth = r5.x;
            if constexpr (books_slots)
            {
                ps.time = 0.0f;
                ps.throughput = make_float3(r0.w, r1.w, compact_last);
                ps.bsdf_pdf = 0.0f;
                ps.radiance = make_float3(0.0f, 0.0f, 0.0f);
                ps.from = compact_from;
                ps.rays_left = camera().max_depth - ps.depth;
            }
            else if constexpr (compact_slots)
            {
                ps.time = 0.0f;
                ps.bsdf_pdf = r0.w;
                ps.throughput = make_float3(r2.x, r2.y, r2.z);
                ps.radiance = make_float3(r1.w, r2.w, compact_last);
                ps.from = compact_from;
                ps.rays_left = camera().max_depth - ps.depth;
            }
            else
            {
                ps.throughput = make_float3(r2.x, r2.y, r2.z);
                ps.bsdf_pdf = r1.w;
                ps.radiance = make_float3(r2.w, r3.x, r3.y);
                ps.from = __float_as_int(r3.z);
                ps.rays_left = __float_as_int(r3.w);
            }
            ps.specular = (flags & wave_specular) != 0u;
            ps.inward = (flags & wave_inward) != 0u;
            sample_index = static_cast<int64_t>(static_cast<uint32_t>(r5.z));
            if (flags & (wave_ext | wave_shadow | wave_finish))
            {
                // the sample's stream, from its number
                const int64_t local = sample_index + (BATCH ? J->local_begin : 0);
                const sample_place at = place_of(local, camera(), BATCH ? J->pass_begin : P.pass_begin);
                sample_rng(at, camera(), BATCH ? J->seed : P.seed, rng);
            }
            bool finished = false;
            float3 sample = make_float3(0.0f, 0.0f, 0.0f);
            if (flags & wave_shadow)
            {
                if (stream_load(B.shadow_result + i) == 0)
                {
                    const float4 q0 = stream_load(shadow_rows + i);
                    const float4 q1 = stream_load(shadow_rows + n + i);
                    const int4 q2 = stream_load(reinterpret_cast<const int4*>(shadow_rows) + 2 * n + i);
                    const float3 contribution = make_float3(q1.w, __int_as_float(q2.x), __int_as_float(q2.y));
                    // through smoke, the light arrives with the chance of crossing it (its expected value)
                    const float through =
                        FEATURES && scene().medium_count > 0
                            ? transmittance(scene(), make_float3(q0.x, q0.y, q0.z), make_float3(q1.x, q1.y, q1.z),
                                            ps.time, q0.w)
                            : 1.0f;
                    ps.radiance = ps.radiance + through * contribution;
                }
                flags &= ~wave_shadow;
            }
            if (flags & wave_finish)
            {
                sample = ps.radiance;
                finished = true;
                flags &= ~wave_finish;
            }
            else if (flags & wave_ext)
            {
                const int4 r = answer;
                hit_info h;
                h.id = r.x;
                h.t = __int_as_float(r.y);
                h.front = r.z != 0;
                ++ps.depth;
                if (FEATURES && scene().medium_count > 0)
                {
                    media_event(scene(), ps.o, ps.d, ps.time, rng, ps.depth, h);
                }
                step_result res;
                if (quality())
                {
                    sq.lit = false; // a vertex that ends the path before its light sample queues no shadow ray
                    res = shade_quality<false, search_tree, FEATURES, true>(scene(), camera(), rng, ps, h, sample,
                                                                            shadow_rays, nullptr, &sq);
                    if (sq.lit)
                    {
                        flags |= wave_shadow;
                    }
                }
                else
                {
                    res = shade_books<FEATURES>(scene(), camera(), rng, ps, h, sample);
                }
                if (res == step_result::done)
                {
                    flags &= ~wave_ext;
                    if (flags & wave_shadow)
                    {
                        flags |= wave_finish; // the sample's value waits for its last shadow ray
                    }
                    else
                    {
                        finished = true;
                    }
                }
            }
            else if (BATCH && (flags & wave_reserved))
            {
                // a stream run's claim made before the host published it: taken below once it has
                const unsigned long long held =
                    static_cast<unsigned long long>(static_cast<uint32_t>(r5.z)) |
                    (static_cast<unsigned long long>(static_cast<uint32_t>(r5.w)) << 32);
                if (held < limit)
                {
                    reserved = held;
                    ready = true;
                }
                else
                {
                    sample_index = static_cast<uint32_t>(held);
                    job = static_cast<int>(held >> 32);
                }
            }
            else
            {
                need = true; // a slot without a sample
            }
            if (finished)
            {
                // the sample's value, added into its chunk's partial in pass order by the reduction
                const float4 value = make_float4(sample.x, sample.y, sample.z, 0.0f);
                if (stream_run)
                {
                    stream_store(J->values + sample_index, value);
                    finished_job = job; // counted below, one atomic per segment per warp
                }
                else
                {
                    stream_store(B.samples + (BATCH ? J->sample_begin : 0) + sample_index, value);
                }
                need = true;
            }
        }
        if (stream_run)
        {
            // the warp's finished samples counted per segment: the host reduces a segment once all are in
            const unsigned peers = __match_any_sync(full_warp, finished_job);
            if (finished_job >= 0 && (peers & lanes_below) == 0u)
            {
                atomicAdd(W.jobs[finished_job].done, static_cast<unsigned long long>(__popc(peers)));
            }
        }
        // A stream run's segment (logical number) holding sample s: `hint` first (a warp's claims are consecutive
        // numbers, nearly always in its leader's segment), else a binary search over the ring of segment starts
        const auto find_segment = [&](int64_t s, int hint) -> int {
            const int mask = W.job_mask;
            if (hint >= window.x && hint < window.y && W.starts[hint & mask] <= s &&
                (hint + 1 >= window.y || s < W.starts[(hint + 1) & mask]))
            {
                return hint;
            }
            int lo = window.x, hi = window.y - 1;
            while (lo < hi)
            {
                const int mid = (lo + hi + 1) >> 1;
                if (W.starts[mid & mask] <= s)
                {
                    lo = mid;
                }
                else
                {
                    hi = mid - 1;
                }
            }
            return lo;
        };
        // Sample s taken by this slot: its job, its pixel and pass (false for a lane of a tile over the image's edge,
        // which claims again; in a stream run it counts as done, having no value to wait for)
        const auto take = [&](unsigned long long s, int hint) -> bool {
            int k = 0;
            if constexpr (BATCH)
            {
                k = stream_run ? (find_segment(static_cast<int64_t>(s), hint) & W.job_mask)
                               : find_job<job_samples>(W.jobs, window.x, window.y, static_cast<int64_t>(s));
            }
            const batch_job* K = BATCH ? W.jobs + k : nullptr;
            const camera_params& c = BATCH ? K->cam : P.cam;
            const int64_t index = static_cast<int64_t>(s) - (BATCH ? K->sample_begin : 0);
            if (stream_run && index < 0)
            {
                // below the window the host gave: a sample no entry holds; reported, never written
                atomicOr(B.control + 3, 1u);
                return false;
            }
            const sample_place at = place_of(index + (BATCH ? K->local_begin : 0), c, BATCH ? K->pass_begin : P.pass_begin);
            if (!(at.x < c.width && at.y < c.height))
            {
                if (stream_run)
                {
                    atomicAdd(K->done, 1ull);
                }
                return false;
            }
            px = at.x;
            py = at.y;
            job = k;
            J = K;
            sample_index = index;
            pass = at.pass;
            rng.job = BATCH ? K->job : P.job;
            start = true;
            return true;
        };
        if (ready)
        {
            flags &= ~wave_reserved;
            need = !take(reserved, -1);
        }
        // Samples for the slots that need one, a pass of the image after another (of each job after another): one
        // atomic per warp. In a stream run a claim beyond what is published waits in the slot (wave_reserved).
        while (true)
        {
            const unsigned needing = __ballot_sync(full_warp, need);
            if (needing == 0u)
            {
                break;
            }
            const int leader = __ffs(static_cast<int>(needing)) - 1;
            unsigned long long base = 0;
            if (static_cast<int>(lane) == leader)
            {
                base = atomicAdd(BATCH ? W.work_counter : P.work_counter,
                                 static_cast<unsigned long long>(__popc(needing)));
            }
            base = __shfl_sync(full_warp, base, leader);
            int hint = -1;
            if (stream_run)
            {
                if (static_cast<int>(lane) == leader && base < limit)
                {
                    hint = find_segment(static_cast<int64_t>(base), -1);
                }
                hint = __shfl_sync(full_warp, hint, leader);
            }
            if (need)
            {
                const unsigned long long s = base + static_cast<unsigned long long>(__popc(needing & lanes_below));
                if (s >= limit)
                {
                    if (stream_run)
                    {
                        flags |= wave_reserved;
                        sample_index = static_cast<uint32_t>(s);
                        job = static_cast<int>(s >> 32);
                    }
                    else
                    {
                        flags |= wave_exhausted;
                    }
                    need = false;
                }
                else
                {
                    need = !take(s, hint);
                }
            }
        }
        if (start)
        {
            // A new sample, as the persistent kernel starts one
            const camera_params& cam = camera();
            round_pass = sample_rng({pass, px, py}, cam, BATCH ? J->seed : P.seed, rng);
            // Under a tree walk and the heavier shading (NEE/MIS, the second book's features) the trace kernel makes
            // the camera ray, a warp's 32 at once, instead of this warp for its few new samples: the mesh +3.6%, the
            // second book's final scene +3.7%. The books' plain sphere scenes (-2%) and the flat searches (-3% to
            // -7%: their trace kernel's tail grows by it) make their own here.
            primary = (quality() || FEATURES) && scene().flat == 0;
            if (!primary)
            {
                const float4 u = rng.draw(0, 0);
                int s_i, s_j;
                stratum_of(cam, round_pass, s_i, s_j);
                camera_ray(cam, px, py, s_i, s_j, u, ps.o, ps.d);
                ps.time = FEATURES && scene().has_motion ? rng.draw(0, block_time).x : 0.0f;
            }
            ps.throughput = make_float3(1.0f, 1.0f, 1.0f);
            ps.radiance = make_float3(0.0f, 0.0f, 0.0f);
            ps.bsdf_pdf = 0.0f;
            ps.specular = true;
            ps.rays_left = cam.max_depth;
            ps.depth = 0;
            ps.from = -1;
            ps.inward = false;
            flags |= wave_ext;
        }
        // The slot's queries: one atomic per warp for its next rays and its shadow rays from the bottom of the queue,
        // one for its new samples' camera rays (primary queries) from the top down
        const bool ext = (flags & wave_ext) != 0u && !primary;
        const bool shadow = QUALITY && (flags & wave_shadow) != 0u;
        const unsigned ext_lanes = __ballot_sync(full_warp, ext);
        const unsigned shadow_lanes = __ballot_sync(full_warp, shadow);
        const unsigned primary_lanes = __ballot_sync(full_warp, primary);
        const int queued = __popc(ext_lanes) + __popc(shadow_lanes);
        if constexpr (BATCH)
        {
            // each job's segments and shadow rays, counted as queued: one atomic per job of the warp
            const bool any = ext || shadow || primary;
            const unsigned peers = __match_any_sync(full_warp, any ? job : -1);
            if (any && static_cast<int>(lane) == __ffs(static_cast<int>(peers)) - 1)
            {
                const unsigned e = __popc(peers & (ext_lanes | primary_lanes)), sh = __popc(peers & shadow_lanes);
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
        if (queued > 0)
        {
            unsigned base = 0;
            if (lane == 0u)
            {
                base = atomicAdd(B.control, static_cast<unsigned>(queued));
            }
            base = __shfl_sync(full_warp, base, 0);
            if (ext)
            {
                const unsigned q = base + static_cast<unsigned>(__popc(ext_lanes & lanes_below));
                stream_store(B.query_o + q, make_float4(ps.o.x, ps.o.y, ps.o.z, ps.time));
                stream_store(B.query_d + q, make_float4(ps.d.x, ps.d.y, ps.d.z, infinity_f));
                stream_store(B.query_meta + q, make_int4(ps.from, (ps.inward ? 1 : 0) | (job << 3), -1, i));
            }
            if (shadow)
            {
                const unsigned q = base + static_cast<unsigned>(__popc(ext_lanes)) +
                                   static_cast<unsigned>(__popc(shadow_lanes & lanes_below));
                stream_store(B.query_o + q, make_float4(sq.o.x, sq.o.y, sq.o.z, ps.time));
                stream_store(B.query_d + q, make_float4(sq.d.x, sq.d.y, sq.d.z, sq.t_max));
                stream_store(B.query_meta + q, make_int4(sq.from, (sq.inward ? 1 : 0) | 2 | (job << 3), sq.skip, i));
                // what the next step needs of it: the light it brings and, through smoke, its segment
                stream_store(shadow_rows + i, make_float4(sq.o.x, sq.o.y, sq.o.z, sq.t_max));
                stream_store(shadow_rows + n + i, make_float4(sq.d.x, sq.d.y, sq.d.z, sq.contribution.x));
                stream_store(reinterpret_cast<int4*>(shadow_rows) + 2 * n + i,
                             make_int4(__float_as_int(sq.contribution.y), __float_as_int(sq.contribution.z), 0, 0));
            }
        }
        if (primary_lanes != 0u)
        {
            const int leader = __ffs(static_cast<int>(primary_lanes)) - 1;
            unsigned base = 0;
            if (static_cast<int>(lane) == leader)
            {
                base = atomicAdd(B.control + 2, static_cast<unsigned>(__popc(primary_lanes)));
            }
            base = __shfl_sync(full_warp, base, leader);
            if (primary)
            {
                // the pixel, the pass in its round and the RNG's key: what the camera ray is made of
                const unsigned q = 2u * static_cast<unsigned>(n) - 1u -
                                   (base + static_cast<unsigned>(__popc(primary_lanes & lanes_below)));
                stream_store(B.query_o + q, make_float4(__int_as_float(px), __int_as_float(py),
                                                        __int_as_float(round_pass), 0.0f));
                stream_store(B.query_d + q, make_float4(__uint_as_float(rng.key.x), __uint_as_float(rng.key.y), 0.0f,
                                                        infinity_f));
                stream_store(B.query_meta + q, make_int4(-1, wave_query_primary | (job << 3), -1, i));
            }
        }
        if (live)
        {
            flags = (flags & ~(wave_specular | wave_inward)) | (ps.specular ? wave_specular : 0u) |
                    (ps.inward ? wave_inward : 0u);
            // the compact forms' flags word: depth << 6 and the six flags
            const auto compact_word = [&](int depth) {
                return static_cast<int>((static_cast<uint32_t>(depth) << 6) | ((flags & wave_ext) ? 1u : 0u) |
                                        ((flags & wave_exhausted) ? 2u : 0u) | ((flags & wave_inward) ? 4u : 0u) |
                                        ((flags & wave_specular) ? 8u : 0u) | ((flags & wave_shadow) ? 16u : 0u) |
                                        ((flags & wave_finish) ? 32u : 0u));
            };
            if (flags & wave_exhausted)
            {
                stream_store(reinterpret_cast<int4*>(rows) + wave_flags_row * n + i,
                             compact_slots ? make_int4(compact_word(0), 0, 0, 0)
                                           : make_int4(0, static_cast<int>(flags), 0, 0));
            }
            else if constexpr (books_slots)
            {
                stream_store(rows + i, make_float4(ps.o.x, ps.o.y, ps.o.z, ps.throughput.x));
                stream_store(rows + n + i, make_float4(ps.d.x, ps.d.y, ps.d.z, ps.throughput.y));
                stream_store(reinterpret_cast<int4*>(rows) + wave_flags_row * n + i,
                             make_int4(compact_word(ps.depth), static_cast<int>(static_cast<uint32_t>(sample_index)),
                                       ps.from, __float_as_int(ps.throughput.z)));
            }
            else if constexpr (compact_slots)
            {
                stream_store(rows + i, make_float4(ps.o.x, ps.o.y, ps.o.z, ps.bsdf_pdf));
                stream_store(rows + n + i, make_float4(ps.d.x, ps.d.y, ps.d.z, ps.radiance.x));
                stream_store(rows + 2 * n + i,
                             make_float4(ps.throughput.x, ps.throughput.y, ps.throughput.z, ps.radiance.y));
                stream_store(reinterpret_cast<int4*>(rows) + wave_flags_row * n + i,
                             make_int4(compact_word(ps.depth), static_cast<int>(static_cast<uint32_t>(sample_index)),
                                       ps.from, __float_as_int(ps.radiance.z)));
            }
            else
            {
                stream_store(rows + i, make_float4(ps.o.x, ps.o.y, ps.o.z, ps.time));
                stream_store(rows + n + i, make_float4(ps.d.x, ps.d.y, ps.d.z, ps.bsdf_pdf));
                stream_store(rows + 2 * n + i,
                             make_float4(ps.throughput.x, ps.throughput.y, ps.throughput.z, ps.radiance.x));
                stream_store(rows + 3 * n + i, make_float4(ps.radiance.y, ps.radiance.z, __int_as_float(ps.from),
                                                           __int_as_float(ps.rays_left)));
                stream_store(reinterpret_cast<int4*>(rows) + wave_flags_row * n + i,
                             make_int4(ps.depth, static_cast<int>(flags), static_cast<int>(static_cast<uint32_t>(
                                                                              sample_index)),
                                       job));
            }
        }
    }
}
