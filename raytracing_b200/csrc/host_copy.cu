// Copies between the caller's pageable memory and the device. A pageable copy goes through the driver's own staging on
// one thread, 3 to 4 GB/s into memory the caller has just allocated, most of it page faults: a 1920x1080 image (50 MB)
// took 15 ms of a 100 ms render, and a query of one ray 78 us of allocations, copies and synchronisations. Here the
// kernels read and write blocks of page-locked memory over PCIe, and the calling thread and up to seven helpers move
// the blocks to and from the caller's memory, each with two blocks in flight.
#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "host.h"

namespace rtb
{
namespace
{
constexpr size_t block_bytes = size_t{1} << 20; // a page-locked block: 1 MiB
constexpr int most_helpers = 7;

// Threads that help one caller at a time; another caller meanwhile does its copies alone. They live to the process's end.
class helpers
{
public:
    // run(worker, workers) on `workers` threads at most, the caller's among them; the first exception is rethrown
    void run(int workers, const std::function<void(int, int)>& job)
    {
        std::unique_lock<std::mutex> turn(turn_, std::try_to_lock);
        workers = turn.owns_lock() ? std::min(workers, start(workers - 1) + 1) : 1;
        if (workers <= 1)
        {
            job(0, 1);
            return;
        }
        {
            const std::lock_guard<std::mutex> lock(mutex_);
            job_ = &job;
            workers_ = workers;
            left_ = workers - 1;
            error_ = nullptr;
            ++round_;
        }
        wake_.notify_all();
        std::exception_ptr own;
        try
        {
            job(0, workers);
        }
        catch (...)
        {
            own = std::current_exception();
        }
        std::unique_lock<std::mutex> lock(mutex_);
        done_.wait(lock, [&] { return left_ == 0; });
        if (own || error_)
        {
            std::rethrow_exception(own ? own : error_);
        }
    }

private:
    std::mutex turn_; // held by the caller being helped
    std::mutex mutex_;
    std::condition_variable wake_, done_;
    const std::function<void(int, int)>* job_ = nullptr;
    int workers_ = 0;
    int left_ = 0;
    uint64_t round_ = 0;
    std::exception_ptr error_;
    int started_ = 0;

    // Up to `wanted` helpers running; how many there are
    int start(int wanted)
    {
        const int most = std::min<int>(most_helpers, static_cast<int>(std::thread::hardware_concurrency()) - 1);
        while (started_ < std::min(wanted, most))
        {
            try
            {
                uint64_t seen = 0;
                {
                    const std::lock_guard<std::mutex> lock(mutex_);
                    seen = round_;
                }
                std::thread([this, id = started_ + 1, seen] { serve(id, seen); }).detach();
            }
            catch (const std::system_error&)
            {
                break; // no thread to be had: the ones there are help
            }
            ++started_;
        }
        return started_;
    }

    void serve(int id, uint64_t seen)
    {
        std::unique_lock<std::mutex> lock(mutex_);
        while (true)
        {
            wake_.wait(lock, [&] { return round_ != seen; });
            seen = round_;
            if (id >= workers_)
            {
                continue;
            }
            const auto* job = job_;
            const int workers = workers_;
            lock.unlock();
            std::exception_ptr e;
            try
            {
                (*job)(id, workers);
            }
            catch (...)
            {
                e = std::current_exception();
            }
            lock.lock();
            if (e && !error_)
            {
                error_ = e;
            }
            if (--left_ == 0)
            {
                done_.notify_one();
            }
        }
    }
};

helpers& the_helpers()
{
    static auto* h = new helpers; // to the process's end, as its threads
    return *h;
}

// A page-locked block and the event after the kernel that uses it
struct staging
{
    staging()
    {
        block = acquire_pinned(block_bytes);
        if (const cudaError_t e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming); e != cudaSuccess)
        {
            release_pinned(block, block_bytes);
            check(e, "creating a CUDA event");
        }
    }
    ~staging()
    {
        if (in_use)
        {
            cudaEventSynchronize(done); // an error's unwinding: the kernel must be through with the block
        }
        cudaEventDestroy(done);
        release_pinned(block, block_bytes);
    }
    staging(const staging&) = delete;
    staging& operator=(const staging&) = delete;
    void* block = nullptr;
    cudaEvent_t done = nullptr;
    bool in_use = false;
};

// Blocks [0, blocks) over the threads: launch(block, memory) queues the kernel of a block on `stream_of()`, take(block,
// memory) moves its results out once it has run. Two blocks of a thread are in flight at a time.
template <class Launch, class Take>
void pipeline(int64_t blocks, cudaStream_t stream, bool own_stream, const Launch& launch, const Take& take)
{
    int device = 0;
    check(cudaGetDevice(&device), "querying the device");
    const auto work = [&](int worker, int workers) {
        if (worker > 0)
        {
            check(cudaSetDevice(device), "selecting the device");
        }
        const cudaStream_t s = own_stream ? cudaStreamPerThread : stream;
        staging stage[2];
        const auto queue = [&](int64_t block, staging& g) {
            g.in_use = true;
            launch(block, g.block, s);
            check(cudaEventRecord(g.done, s), "recording a CUDA event");
        };
        int k = 0;
        if (worker < blocks)
        {
            queue(worker, stage[0]);
        }
        for (int64_t block = worker; block < blocks; block += workers, k ^= 1)
        {
            if (block + workers < blocks)
            {
                queue(block + workers, stage[k ^ 1]);
            }
            check(cudaEventSynchronize(stage[k].done), "copying from the GPU");
            stage[k].in_use = false;
            take(block, stage[k].block);
        }
    };
    the_helpers().run(static_cast<int>(std::min<int64_t>(blocks, most_helpers + 1)), work);
}

// out[i] = sums[i] * scale, into page-locked memory: as many 16-byte stores in flight as PCIe takes
__global__ void scale_kernel(const double* sums, double* out, int64_t count, double scale)
{
    const int64_t pairs = count / 2;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < pairs;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const double2 v = reinterpret_cast<const double2*>(sums)[i];
        reinterpret_cast<double2*>(out)[i] = make_double2(__dmul_rn(v.x, scale), __dmul_rn(v.y, scale));
    }
    if ((count & 1) != 0 && blockIdx.x == 0 && threadIdx.x == 0)
    {
        out[count - 1] = __dmul_rn(sums[count - 1], scale);
    }
}
} // namespace

void fetch_image(const double* sums, int64_t count, double scale, double* out, cudaStream_t stream)
{
    constexpr int64_t per_block = static_cast<int64_t>(block_bytes / sizeof(double));
    pipeline(
        (count + per_block - 1) / per_block, stream, false,
        [&](int64_t block, void* memory, cudaStream_t s) {
            const int64_t n = std::min(per_block, count - block * per_block);
            scale_kernel<<<static_cast<unsigned>((n + 511) / 512), 256, 0, s>>>(
                sums + block * per_block, static_cast<double*>(memory), n, scale);
            check(cudaGetLastError(), "scaling the image");
        },
        [&](int64_t block, const void* memory) {
            const int64_t n = std::min(per_block, count - block * per_block);
            std::memcpy(out + block * per_block, memory, static_cast<size_t>(n) * sizeof(double));
        });
}

void trace_rays(const scene_view& scene, const int32_t* prim_source, const float* origins, const float* directions,
                int64_t count, int32_t* ids, float* ts)
{
    // a block: the origins and directions of its rays, then their ids and distances
    constexpr int64_t per_block = 16384;
    static_assert(per_block * 8 * sizeof(float) <= block_bytes);
    const auto rays_of = [&](int64_t block) { return std::min(per_block, count - block * per_block); };
    // Answers over the rays' own memory: a block's would overwrite the rays of one not yet read
    std::vector<float> rays;
    const auto over = [&](const void* out, const float* in) {
        const auto o = reinterpret_cast<uintptr_t>(out), i = reinterpret_cast<uintptr_t>(in);
        const auto n = static_cast<uintptr_t>(count);
        return o < i + n * 3 * sizeof(float) && i < o + n * sizeof(float);
    };
    if (over(ids, origins) || over(ids, directions) || over(ts, origins) || over(ts, directions))
    {
        const size_t n = static_cast<size_t>(count) * 3;
        rays.resize(2 * n);
        std::copy_n(origins, n, rays.data());
        std::copy_n(directions, n, rays.data() + n);
        origins = rays.data();
        directions = rays.data() + n;
    }
    pipeline(
        (count + per_block - 1) / per_block, nullptr, true,
        [&](int64_t block, void* memory, cudaStream_t s) {
            const int64_t n = rays_of(block);
            auto* o = static_cast<float*>(memory);
            std::memcpy(o, origins + 3 * block * per_block, static_cast<size_t>(n) * 3 * sizeof(float));
            std::memcpy(o + 3 * per_block, directions + 3 * block * per_block, static_cast<size_t>(n) * 3 * sizeof(float));
            check(launch_closest_hits(scene, o, o + 3 * per_block, n, prim_source,
                                      reinterpret_cast<int32_t*>(o + 6 * per_block), o + 7 * per_block, s),
                  "launching the closest-hit queries");
        },
        [&](int64_t block, const void* memory) {
            const size_t n = static_cast<size_t>(rays_of(block));
            const auto* o = static_cast<const float*>(memory);
            std::memcpy(ids + block * per_block, o + 6 * per_block, n * sizeof(int32_t));
            std::memcpy(ts + block * per_block, o + 7 * per_block, n * sizeof(float));
        });
}

void table_upload::commit(device_array<unsigned char>& memory)
{
    size_t total = 0;
    for (item& t : items_)
    {
        t.offset = total;
        total += (t.bytes + 255) / 256 * 256;
    }
    if (total > 0)
    {
        memory.allocate(total);
        const cudaStream_t s = allocation_stream();
        if (total <= block_bytes)
        {
            staging g;
            for (const item& t : items_)
            {
                std::memcpy(static_cast<unsigned char*>(g.block) + t.offset, t.data, t.bytes);
            }
            check(cudaMemcpyAsync(memory.data(), g.block, total, cudaMemcpyHostToDevice, s), "copying to the device");
            check(cudaStreamSynchronize(s), "copying to the device");
        }
        else
        {
            for (const item& t : items_)
            {
                check(cudaMemcpy(memory.data() + t.offset, t.data, t.bytes, cudaMemcpyHostToDevice),
                      "copying to the device");
            }
        }
    }
    for (const item& t : items_)
    {
        t.attach(memory.data() + t.offset);
    }
    items_.clear();
}
} // namespace rtb
