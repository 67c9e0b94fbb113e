// Time marks: pooled CUDA events behind small integer ids, for the keyed timers of the training loop.
//
// A timed region costs two marks.  Taking one is a pool lookup and a cudaEventRecord (about 1 us through ctypes); an event
// object of the framework above, created, recorded and destroyed per region end, was about 10 us, 0.2 ms of a 1.2 ms
// training step on a 10,000-node graph.  Ids are (device << 24) | slot; a slot goes back to its device's pool on release.
#include <mutex>
#include <vector>
#include "dg_internal.h"

namespace {

constexpr int kMaxDevices = 64, kSlotBits = 24;

struct MarkPool {
    std::mutex mu;
    std::vector<cudaEvent_t> events[kMaxDevices];
    std::vector<int> unused[kMaxDevices];
};
MarkPool& pool() { static MarkPool* p = new MarkPool(); return *p; }      // never destroyed: the driver may be gone first

cudaEvent_t event_of(int id)
{
    const int dev = id >> kSlotBits, slot = id & ((1 << kSlotBits) - 1);
    MarkPool& p = pool();
    if (id < 0 || dev >= kMaxDevices || slot >= (int)p.events[dev].size()) return nullptr;
    return p.events[dev][slot];
}

}  // namespace

extern "C" int dg_mark_record(void* stream)
try {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DG_ERR_STATE;
    MarkPool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    int slot;
    if (!p.unused[dev].empty()) {
        slot = p.unused[dev].back();
        p.unused[dev].pop_back();
    } else {
        cudaEvent_t e;
        if (p.events[dev].size() >= (size_t)1 << kSlotBits || cudaEventCreate(&e) != cudaSuccess) return DG_ERR_STATE;
        slot = (int)p.events[dev].size();
        p.events[dev].push_back(e);
    }
    if (cudaEventRecord(p.events[dev][slot], (cudaStream_t)stream) != cudaSuccess) {
        p.unused[dev].push_back(slot);
        return DG_ERR_STATE;
    }
    return (dev << kSlotBits) | slot;
} catch (...) {
    return dg_exception();
}

extern "C" int dg_mark_elapsed(int begin, int end, float* host_ms)
try {
    if (!host_ms) return DG_ERR_NULL;
    MarkPool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    cudaEvent_t a = event_of(begin), b = event_of(end);
    if (!a || !b) return DG_ERR_STATE;
    DG_CUDA(cudaEventElapsedTime(host_ms, a, b));
    return DG_OK;
} catch (...) {
    return dg_exception();
}

extern "C" int dg_mark_release(int id)
try {
    MarkPool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    if (!event_of(id)) return DG_ERR_STATE;
    p.unused[id >> kSlotBits].push_back(id & ((1 << kSlotBits) - 1));
    return DG_OK;
} catch (...) {
    return dg_exception();
}
