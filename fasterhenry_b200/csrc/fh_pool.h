// Device workspace of a system's sweeps, kept between calls: one buffer per
// role (slot), grown when a sweep needs more.  Repeated sweeps then allocate
// nothing, and no cudaFree (which synchronizes the device) runs inside a
// sweep after the first.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <utility>
#include <vector>

namespace fhb {

// The memory cache (fh_mem.cu).
cudaError_t cache_alloc(void **p, size_t bytes, cudaStream_t s);
void cache_free(void *p, cudaStream_t s);

struct DevPool {
    std::vector<std::pair<void *, size_t>> slot;
    cudaStream_t stream = nullptr;  // the owner's stream: allocations and frees are ordered on it
    // Frequencies per batch whose buffers are all in the slots, by precision:
    // such a batch needs no look at the free memory.
    size_t batch[3] = {0, 0, 0};
    ~DevPool() { release(); }
    void release() {
        for (auto &b : slot)
            if (b.first) cache_free(b.first, stream);
        slot.clear();
        forget();
    }
    void forget() { std::fill(batch, batch + 3, (size_t)0); }
    size_t held() const {
        size_t t = 0;
        for (const auto &b : slot) t += b.second;
        return t;
    }
    // A slot that grows is freed first: where its new size cannot be had, the
    // batches that it held cannot be had without a look at the memory, either.
    cudaError_t get(int id, size_t bytes, void **out) {
        if ((int)slot.size() <= id) slot.resize((size_t)id + 1, {nullptr, 0});
        auto &b = slot[(size_t)id];
        if (b.second < bytes) {
            if (b.first) cache_free(b.first, stream);
            b = {nullptr, 0};
            const cudaError_t e = cache_alloc(&b.first, std::max<size_t>(bytes, 1), stream);
            if (e != cudaSuccess) {
                b.first = nullptr;
                forget();
                return e;
            }
            b.second = bytes;
        }
        *out = b.first;
        return cudaSuccess;
    }
};

}  // namespace fhb
