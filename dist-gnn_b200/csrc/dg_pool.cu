// Device memory of plans: blocks that outlive the plan that used them.
//
// cudaMalloc and cudaFree cost tens of microseconds at best and, on a device whose memory is mostly mapped, now and then
// milliseconds; building a plan took 45 of the former and 54 of the latter, most of the 8 to 30 ms that plan construction
// and one product of a 300 k-row block cost.  Freed blocks are kept per device, at most kKeepBytes of them, and handed out
// again to requests of a similar size; twice as many while a plan is being built, whose temporaries come back in the middle of
// a caller's call, where a cudaFree would wait for the device: dg_plan_destroy brings the pool back to its size.  A block that does
// not fit any more pushes out those that have lain idle longest: what earlier, larger plans left behind must not keep the blocks of
// those in use now from staying (plan and product of a 55,160-node matrix after others had filled the pool: 930 -> 180 us).  A
// block may come back only when the device is done with it: callers synchronise first (dg_plan_destroy the device, as cudaFree did;
// plan construction its stream).
//
// The program around the library usually has a caching allocator of its own, which may hold the whole device without using it.
// So an allocation that the driver refuses is tried three times: as it is, after the pool has given its idle blocks back, and
// after the program has been asked to (dg_on_low_memory).  dg_pool_trim gives the pool's idle blocks back on request.
#include <atomic>
#include <map>
#include <mutex>
#include <new>
#include <unordered_map>
#include "dg_internal.h"

namespace {

constexpr size_t kKeepBytes = (size_t)512 << 20;
constexpr int kMaxDevices = 64;

struct Idle { void* ptr; uint64_t since; };
struct Pool {
    std::mutex mu;
    uint64_t clock = 0;                                           // counts the blocks that were given back
    std::multimap<size_t, Idle> unused[kMaxDevices];
    size_t unused_bytes[kMaxDevices] = {};
    std::unordered_map<void*, size_t> size[kMaxDevices];
};
Pool& pool() { static Pool* p = new Pool(); return *p; }      // never destroyed: the driver may be gone first

std::atomic<void (*)(void)> g_give_back{nullptr};                 // the program's own cache

// Sizes in steps of an eighth of their power of two, so that blocks of nearly equal plans fit one another.
size_t rounded(size_t bytes)
{
    size_t step = 512;
    while (step * 16 < bytes) step *= 2;
    return (bytes + step - 1) / step * step;
}

void release_unused(Pool& p, int dev)                             // caller holds the mutex and has dev current
{
    for (auto& b : p.unused[dev]) {
        cudaFree(b.second.ptr);
        p.size[dev].erase(b.second.ptr);
    }
    p.unused[dev].clear();
    p.unused_bytes[dev] = 0;
}

int trim(int dev)
{
    if (dev < 0 || dev >= kMaxDevices) return DG_ERR_STATE;
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    release_unused(p, dev);
    return DG_OK;
}

}  // namespace

// cudaMalloc that makes room where there is none.  No lock is held while the program gives its memory back, and a refusal leaves
// nothing behind for the next cudaGetLastError() to report.
int dg_device_alloc(void** out, size_t bytes)
{
    int dev = -1;
    DG_CUDA(cudaGetDevice(&dev));
    cudaError_t e = cudaMalloc(out, bytes);
    for (int attempt = 0; attempt < 2 && e == cudaErrorMemoryAllocation; ++attempt) {
        cudaGetLastError();
        if (attempt == 0) {
            trim(dev);
        } else {
            void (*give_back)(void) = g_give_back.load();
            if (!give_back) break;
            give_back();
        }
        e = cudaMalloc(out, bytes);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *out = nullptr;
    }
    return (int)e;
}

int dg_exception() noexcept
{
    try {
        throw;
    } catch (const std::bad_alloc&) {
        return (int)cudaErrorMemoryAllocation;
    } catch (...) {
        return DG_ERR_STATE;
    }
}

// One word per device, zero until a tensor-core kernel gives up on a bounded wait.
int* dg_status_word()
{
    static std::mutex mu;
    static int* word[kMaxDevices] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (word[dev]) return word[dev];
    }
    int* w = nullptr;                                             // no lock while the program may be asked for memory
    if (dg_device_alloc((void**)&w, sizeof(int)) != DG_OK) return nullptr;
    if (cudaMemset(w, 0, sizeof(int)) != cudaSuccess || cudaStreamSynchronize(nullptr) != cudaSuccess) {
        cudaFree(w);
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (word[dev]) cudaFree(w);                                   // another thread was faster
    else word[dev] = w;
    return word[dev];
}

extern "C" int dg_on_low_memory(void (*give_back)(void))
{
    g_give_back.store(give_back);
    return DG_OK;
}

int dg_pool_alloc(void** out, size_t bytes)
{
    int dev = -1;
    DG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return DG_ERR_STATE;
    const size_t want = rounded(bytes ? bytes : 1);
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        auto it = p.unused[dev].lower_bound(want);
        if (it != p.unused[dev].end() && it->first <= want + want / 4) {
            *out = it->second.ptr;
            p.unused_bytes[dev] -= it->first;
            p.unused[dev].erase(it);
            return DG_OK;
        }
    }
    const int rc = dg_device_alloc(out, want);
    if (rc) return rc;
    try {
        std::lock_guard<std::mutex> lock(p.mu);
        p.size[dev][*out] = want;
    } catch (...) {
        cudaFree(*out);
        throw;
    }
    return DG_OK;
}

void dg_pool_free(void* ptr, bool building) noexcept
{
    const size_t keep = building ? 2 * kKeepBytes : kKeepBytes;
    int dev = -1;
    if (!ptr || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    auto it = p.size[dev].find(ptr);
    if (it == p.size[dev].end()) return;
    if (it->second > kKeepBytes) {
        p.size[dev].erase(it);
        cudaFree(ptr);
        return;
    }
    auto& unused = p.unused[dev];
    while (p.unused_bytes[dev] + it->second > keep) {
        auto oldest = unused.begin();
        for (auto u = unused.begin(); u != unused.end(); ++u)
            if (u->second.since < oldest->second.since) oldest = u;
        cudaFree(oldest->second.ptr);
        p.unused_bytes[dev] -= oldest->first;
        p.size[dev].erase(oldest->second.ptr);
        unused.erase(oldest);
    }
    try {
        unused.emplace(it->second, Idle{ptr, p.clock++});
        p.unused_bytes[dev] += it->second;
    } catch (...) {                                               // no room on the host to remember it
        p.size[dev].erase(it);
        cudaFree(ptr);
    }
}

extern "C" int dg_pool_trim(void)
try {
    int dev = -1;
    DG_CUDA(cudaGetDevice(&dev));
    return trim(dev);
} catch (...) {
    return dg_exception();
}
