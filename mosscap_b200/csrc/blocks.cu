// Device memory blocks kept from one adjoint to the next (blocks.h).
#include "blocks.h"

#include <list>
#include <mutex>

namespace mc {
namespace {

struct Block {
    void* p;
    size_t bytes;
    int device;
};

// leaked on purpose: blocks may be freed by destructors that run after this file's
std::list<Block>& kept() {
    static std::list<Block>* l = new std::list<Block>();
    return *l;
}
size_t g_bytes = 0;
std::mutex g_mutex;

} // namespace

cudaError_t block_alloc(void** p, size_t bytes) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        return e;
    }
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        for (auto it = kept().begin(); it != kept().end(); ++it) {
            if (it->bytes == bytes && it->device == device) {
                *p = it->p;
                g_bytes -= bytes;
                kept().erase(it);
                return cudaSuccess;
            }
        }
    }
    return device_alloc(p, bytes);
}

void block_free(void* p, size_t bytes, int device) {
    if (!p) {
        return;
    }
    if (bytes > kKeptBytes) {
        cudaFree(p);
        return;
    }
    std::lock_guard<std::mutex> lock(g_mutex);
    while (g_bytes + bytes > kKeptBytes) {
        cudaFree(kept().front().p);
        g_bytes -= kept().front().bytes;
        kept().pop_front();
    }
    kept().push_back({p, bytes, device});
    g_bytes += bytes;
}

void blocks_release() {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (const Block& b : kept()) {
        cudaFree(b.p);
    }
    kept().clear();
    g_bytes = 0;
}

cudaError_t device_alloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        blocks_release();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

} // namespace mc
