// Bulk copies between pageable host memory and the device.
//
// A cudaMemcpy from or to pageable memory goes through the driver's staging
// buffer on one CPU thread: 11 GB/s here, against 52 GB/s for pinned memory
// (138 MB host to device: 12.5 and 2.7 ms).  Here several threads do the same
// staging, each with two pinned slots, so that CPU copies of one slot overlap
// the DMA of others, and first touches of a fresh destination's pages are spread
// over the threads too.  With 16 host threads: prt_build_mesh of a 138 MB soup
// 13.5 -> 6 ms, prt_read_built_mesh of 30 MB into fresh arrays 6.5 -> 3.9 ms.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "prt_internal.h"

namespace prt_b200 {

namespace {

constexpr int kWorkers = 8;
constexpr int kMaxDevices = 64;
constexpr size_t kStageSlot = 512 << 10;
// smaller copies are not worth starting threads for, and the first one has to
// pay for the slots
constexpr size_t kStageMin = 4 << 20;
constexpr size_t kStageFirst = 32 << 20;

struct HostStage
{
    std::mutex lock;
    int users = 0;                         // contexts on the device
    char* pinned = nullptr;
    unsigned long long ctxId = 0;          // CUDA context of the slots and events
    cudaEvent_t done[2 * kWorkers] = {};   // per slot: its last copy

    bool reserve();
    void release();
    void forget();
    template <class Work>
    cudaError_t run(size_t bytes, const Work& work);
};

HostStage g_stage[kMaxDevices];

// The current device's slots, locked, or nullptr to copy without them.
HostStage* acquire(size_t bytes, std::unique_lock<std::mutex>& held)
{
    int device = -1;
    if (bytes < kStageMin || cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return nullptr;
    HostStage& s = g_stage[device];
    std::unique_lock<std::mutex> l(s.lock, std::try_to_lock);
    if (!l.owns_lock() || s.users == 0) return nullptr;
    unsigned long long id = 0;
    if (current_context_id(&id) != cudaSuccess) return nullptr;
    if (s.pinned && s.ctxId != id) s.forget();   // made in a context that a device reset has ended
    s.ctxId = id;
    if (!s.pinned && (bytes < kStageFirst || !s.reserve())) return nullptr;
    held = std::move(l);
    return &s;
}

bool pageable(const void* p)
{
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess)
    {
        cudaGetLastError();
        return true;
    }
    return attr.type == cudaMemoryTypeUnregistered;
}

bool HostStage::reserve()
{
    if (pinned) return true;
    if (host_pinned_alloc(&pinned, kStageSlot * 2 * kWorkers) != cudaSuccess)
    {
        cudaGetLastError();
        pinned = nullptr;
        return false;
    }
    for (int i = 0; i < 2 * kWorkers; ++i)
        if (cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming) != cudaSuccess)
        {
            cudaGetLastError();
            release();
            return false;
        }
    return true;
}

void HostStage::release()
{
    for (int i = 0; i < 2 * kWorkers; ++i)
    {
        if (done[i])
        {
            cudaEventSynchronize(done[i]);   // the slot's last copy
            cudaEventDestroy(done[i]);
        }
        done[i] = nullptr;
    }
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
}

void HostStage::forget()
{
    for (cudaEvent_t& e : done) e = nullptr;
    pinned = nullptr;
}

// Chunks are claimed from a shared counter, so the calling thread alone
// finishes the copy if no other thread can be started.
template <class Work>
cudaError_t HostStage::run(size_t bytes, const Work& work)
{
    const size_t chunks = (bytes + kStageSlot - 1) / kStageSlot;
    std::atomic<size_t> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    auto worker = [&](int w) {
        cudaError_t r = cudaSetDevice(device);
        if (r == cudaSuccess) r = work(w, next, chunks);
        if (r != cudaSuccess) failed = (int)r;
    };
    const int want = (int)std::min<size_t>({(size_t)kWorkers, std::max(1u, std::thread::hardware_concurrency()), chunks});
    std::vector<std::thread> threads;
    try
    {
        threads.reserve(kWorkers);
        for (int w = 1; w < want; ++w) threads.emplace_back(worker, w);
    }
    catch (const std::system_error&)
    {
    }
    catch (const std::bad_alloc&)
    {
    }
    worker(0);
    for (std::thread& t : threads) t.join();
    return (cudaError_t)failed.load();
}

} // namespace

void stage_retain(int device)
{
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> l(g_stage[device].lock);
    ++g_stage[device].users;
}

void stage_release(int device)
{
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> l(g_stage[device].lock);
    HostStage& s = g_stage[device];
    if (--s.users != 0) return;
    unsigned long long id = 0;
    if (current_context_id(&id) == cudaSuccess && id == s.ctxId) s.release();
    else s.forget();
}

cudaError_t stage_upload(void* dst, const void* src, size_t bytes, cudaStream_t stream)
{
    std::unique_lock<std::mutex> held;
    HostStage* s = pageable(src) ? acquire(bytes, held) : nullptr;
    if (!s) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, stream);
    char* const pinned = s->pinned;
    cudaEvent_t* const done = s->done;
    return s->run(bytes, [&](int w, std::atomic<size_t>& next, size_t chunks) -> cudaError_t {
        for (int k = 0;; k ^= 1)
        {
            const size_t c = next.fetch_add(1);
            if (c >= chunks) return cudaSuccess;
            const size_t at = c * kStageSlot, n = std::min(kStageSlot, bytes - at);
            const int slot = 2 * w + k;
            char* buf = pinned + kStageSlot * slot;
            cudaError_t e = cudaEventSynchronize(done[slot]);   // its previous copy
            if (e != cudaSuccess) return e;
            std::memcpy(buf, static_cast<const char*>(src) + at, n);
            e = cudaMemcpyAsync(static_cast<char*>(dst) + at, buf, n, cudaMemcpyHostToDevice, stream);
            if (e == cudaSuccess) e = cudaEventRecord(done[slot], stream);
            if (e != cudaSuccess) return e;
        }
    });
}

cudaError_t stage_download(void* dst, const void* src, size_t bytes, cudaStream_t stream)
{
    std::unique_lock<std::mutex> held;
    HostStage* s = pageable(dst) ? acquire(bytes, held) : nullptr;
    if (!s)
    {
        cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, stream);
        return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
    }
    char* const pinned = s->pinned;
    cudaEvent_t* const done = s->done;
    return s->run(bytes, [&](int w, std::atomic<size_t>& next, size_t chunks) -> cudaError_t {
        size_t at[2] = {0, 0}, n[2] = {0, 0};   // chunk in each slot, n 0: none
        auto take = [&](int k) -> cudaError_t {
            if (!n[k]) return cudaSuccess;
            const cudaError_t e = cudaEventSynchronize(done[2 * w + k]);
            if (e == cudaSuccess) std::memcpy(static_cast<char*>(dst) + at[k], pinned + kStageSlot * (2 * w + k), n[k]);
            n[k] = 0;
            return e;
        };
        cudaError_t e = cudaSuccess;
        for (int k = 0; e == cudaSuccess; k ^= 1)
        {
            const size_t c = next.fetch_add(1);
            if (c >= chunks) break;
            // slot k is free: its chunk was taken before slot k ^ 1 was filled,
            // and an earlier call's copy out of it has been waited for
            e = cudaEventSynchronize(done[2 * w + k]);
            at[k] = c * kStageSlot;
            n[k] = std::min(kStageSlot, bytes - at[k]);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(pinned + kStageSlot * (2 * w + k), static_cast<const char*>(src) + at[k], n[k],
                                    cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaEventRecord(done[2 * w + k], stream);
            if (e != cudaSuccess)
            {
                n[k] = 0;
                break;
            }
            e = take(k ^ 1);
        }
        for (int k = 0; k < 2; ++k)
        {
            const cudaError_t r = take(k);
            if (e == cudaSuccess) e = r;
        }
        return e;
    });
}

} // namespace prt_b200
