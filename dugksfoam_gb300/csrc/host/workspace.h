// Device memory that the objective calls of a handle keep between them, and
// the allocation every other part of the library uses, which takes kept memory
// back before it gives up.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <vector>

namespace dugks {

// Chunks of one handle.  A call takes the pool (try_take), carves the chunks
// and gives it back; a call that finds it taken by another thread's works on
// memory of its own.  All pools of the process together keep at most kKeep
// bytes: a few calls' worth of small buffers, whose allocation and release cost
// 4 of the 32 ms of a 48^2 x 28^2 adjoint (1.1 GB in some 60 buffers).
class WorkPool {
public:
    struct Chunk {
        char* p;
        size_t n;
    };
    static constexpr size_t kKeep = 4ull << 30;
    WorkPool();
    ~WorkPool();  // frees the chunks
    WorkPool(const WorkPool&) = delete;
    WorkPool& operator=(const WorkPool&) = delete;
    bool try_take() { return !taken_.exchange(true, std::memory_order_acquire); }
    void give() { taken_.store(false, std::memory_order_release); }
    // for the call that took the pool
    std::vector<Chunk>& chunks() { return chunks_; }
    void settle();  // after a call: frees what is beyond kKeep
    size_t kept() const;  // bytes it keeps between calls
    // Bytes that idle pools other than this one keep: free for whoever asks.
    size_t kept_by_others() const;

private:
    friend cudaError_t device_malloc(void**, size_t);
    static bool give_back_idle();  // frees the chunks of every pool that no call has taken
    size_t drop();                 // frees this pool's chunks; their bytes
    std::atomic<bool> taken_{false};
    std::vector<Chunk> chunks_;
    size_t counted_ = 0;  // of the chunks, what the process's total holds
};

// cudaMalloc on the current device; refused for want of memory, once more after
// the memory that idle pools keep has been given back.
cudaError_t device_malloc(void** p, size_t n);

}  // namespace dugks
