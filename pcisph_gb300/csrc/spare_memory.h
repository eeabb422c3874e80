// spare_memory.h -- device memory that its owner can do without (the rebuilt neighbour lists of a scene): any allocation of
// the library that finds no room has it given up first, whichever context holds it.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

namespace pcisph {
namespace host {

class SpareBlock {
   public:
    explicit SpareBlock() {
        std::lock_guard<std::mutex> l(registry().m);
        registry().all.push_back(this);
    }
    ~SpareBlock() {
        {
            std::lock_guard<std::mutex> l(registry().m);
            auto& a = registry().all;
            a.erase(std::find(a.begin(), a.end(), this));
        }
        release();
    }
    SpareBlock(const SpareBlock&) = delete;
    SpareBlock& operator=(const SpareBlock&) = delete;

    // The owner holds this while it looks at the block and submits work that uses it. It allocates nothing meanwhile.
    std::mutex use;

    void* p() const { return p_; }
    size_t bytes() const { return p_ ? cap_ : 0; }
    // bytes on the current device, if an eighth of the device stays free; the owner has no work in flight. Any error means no.
    bool acquire(size_t bytes) {
        std::lock_guard<std::mutex> l(use);
        if (p_ && cap_ >= bytes) return true;
        drop();
        size_t room = 0, total = 0;
        void* q = nullptr;
        if (cudaMemGetInfo(&room, &total) != cudaSuccess || room < bytes + total / 8 || cudaMalloc(&q, bytes) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        p_ = q;
        cap_ = bytes;
        kept_ = false;
        cudaGetDevice(&device_);
        return true;
    }
    void release() {
        std::lock_guard<std::mutex> l(use);
        drop();
    }
    // Some graph of a caller's holds the address from now on: the block stays.
    void keep() { kept_ = true; }

    // Give up every block of the current device; true if there was one. Waits for the owners' submissions and their work.
    static bool give_back() {
        int device = -1;
        if (cudaGetDevice(&device) != cudaSuccess) return false;
        bool any = false;
        std::lock_guard<std::mutex> l(registry().m);
        for (SpareBlock* b : registry().all) {
            std::lock_guard<std::mutex> u(b->use);
            if (!b->p_ || b->device_ != device || b->kept_) continue;
            if (cudaDeviceSynchronize() != cudaSuccess) return any;
            b->drop();
            any = true;
        }
        return any;
    }

   private:
    struct Registry {
        std::mutex m;
        std::vector<SpareBlock*> all;
    };
    static Registry& registry() {
        static Registry* r = new Registry;  // outlives every context, whatever the order of destruction at exit
        return *r;
    }
    void drop() {
        if (p_) cudaFree(p_);
        p_ = nullptr;
        cap_ = 0;
    }
    void* p_ = nullptr;
    size_t cap_ = 0;
    int device_ = -1;
    bool kept_ = false;
};

// cudaMalloc; without room, once more after the spare memory of the device was given up.
inline cudaError_t device_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && SpareBlock::give_back()) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

}  // namespace host
}  // namespace pcisph
