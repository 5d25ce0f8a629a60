#include "workspace.h"

#include <algorithm>
#include <mutex>

namespace dugks {
namespace {

// Every pool of the process and the bytes they keep (never destroyed: handles
// may outlive static objects).
struct Registry {
    std::mutex m;
    std::vector<WorkPool*> pools;
    size_t kept = 0;
};
Registry& registry() {
    static Registry* r = new Registry();
    return *r;
}

}  // namespace

WorkPool::WorkPool() {
    Registry& r = registry();
    std::lock_guard<std::mutex> l(r.m);
    r.pools.push_back(this);
}

WorkPool::~WorkPool() {
    Registry& r = registry();
    std::lock_guard<std::mutex> l(r.m);
    r.pools.erase(std::remove(r.pools.begin(), r.pools.end(), this), r.pools.end());
    r.kept -= counted_;
    drop();
}

size_t WorkPool::drop() {
    size_t n = 0;
    for (const Chunk& c : chunks_) {
        cudaFree(c.p);  // waits for the device
        n += c.n;
    }
    chunks_.clear();
    counted_ = 0;
    return n;
}

void WorkPool::settle() {
    Registry& r = registry();
    std::lock_guard<std::mutex> l(r.m);
    r.kept -= counted_;
    counted_ = 0;
    size_t n = 0;
    for (const Chunk& c : chunks_) {
        if (r.kept + c.n <= kKeep) {
            r.kept += c.n;
            counted_ += c.n;
            chunks_[n++] = c;
        } else {
            cudaFree(c.p);
        }
    }
    chunks_.resize(n);
}

size_t WorkPool::kept() const {
    std::lock_guard<std::mutex> l(registry().m);
    return counted_;
}

size_t WorkPool::kept_by_others() const {
    Registry& r = registry();
    std::lock_guard<std::mutex> l(r.m);
    size_t n = 0;
    for (const WorkPool* p : r.pools)
        if (p != this && !p->taken_) n += p->counted_;
    return n;
}

bool WorkPool::give_back_idle() {
    Registry& r = registry();
    std::lock_guard<std::mutex> l(r.m);
    size_t n = 0;
    for (WorkPool* p : r.pools) {
        if (!p->try_take()) continue;  // a call works on it
        r.kept -= p->counted_;
        n += p->drop();
        p->give();
    }
    return n > 0;
}

cudaError_t device_malloc(void** p, size_t n) {
    cudaError_t e = cudaMalloc(p, n);
    if (e != cudaErrorMemoryAllocation) return e;
    if (!WorkPool::give_back_idle()) return e;
    cudaGetLastError();
    return cudaMalloc(p, n);
}

}  // namespace dugks
