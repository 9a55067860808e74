// Buffers that only grow, on memory that Mem allocates and frees.
#pragma once

#include <algorithm>
#include <cstddef>

namespace art {

// It grows by at least half its size (in 2 MiB steps), so a stream of solves of
// slowly growing size -- batches of a decode pipeline -- reallocates rarely:
// cudaFree waits for the whole device, which would serialise contexts working
// side by side, and a new address forces the iteration graph to be captured
// again.
//
// Mem::alloc(void **, size_t) returns an error (0: none) and Mem::free(void *)
// gives the memory back.
template <class Mem>
struct GrowBuf {
    void *p = nullptr;
    size_t n = 0;
    // Set by every allocation, for an owner that has to initialise new memory and
    // clears it then. The address does not tell: the old memory is freed before
    // the new is allocated, and the allocator may hand out the same place.
    bool fresh = false;
    // Room for `bytes`, or Mem's error and no memory.
    auto ensure(size_t bytes) -> decltype(Mem::alloc(&p, bytes))
    {
        if (bytes <= n) return {};
        if (n) bytes = std::max(bytes, n + n / 2);
        bytes = (bytes + (2u << 20) - 1) / (2u << 20) * (2u << 20);
        release();
        const auto e = Mem::alloc(&p, bytes);
        if (e) {
            p = nullptr;
            return e;
        }
        n = bytes;
        fresh = true;
        return {};
    }
    void release()
    {
        if (p) Mem::free(p);
        p = nullptr;
        n = 0;
    }
};

}  // namespace art
