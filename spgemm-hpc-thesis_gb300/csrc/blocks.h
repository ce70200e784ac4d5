// Device memory of the engine's calls, kept between them.
//
// A call allocates a dozen arrays, the largest of 8 bytes per scalar product, and
// frees all but its result.  Through the driver's stream-ordered pool alone that
// takes 25 us a call, and 3-6 ms at 7 GB: while the previous result lives, the
// pool finds no contiguous piece of the right size between the small blocks that
// come and go, and maps memory anew.  So every handle keeps the blocks it frees
// (BlockCache) and serves its next calls from them, by size.
//
// Bounds: the handles of a device keep at most 1/16 of its memory between them; a
// handle's oldest blocks go back to the pool first.  When an allocation fails, every
// handle's kept blocks go back and it is tried again.  A handle's blocks are reused
// on its own stream only, in stream order, so no event is needed; a block that
// another handle frees goes to the pool, on that handle's stream.  All of it is
// under one lock.
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace spg {

class BlockCache {
public:
    BlockCache(int device, cudaStream_t stream);
    ~BlockCache();  // the kept blocks go back to the pool
    BlockCache(const BlockCache&) = delete;
    BlockCache& operator=(const BlockCache&) = delete;

    // At least `bytes` of device memory for work on the cache's stream.
    cudaError_t alloc(void** p, size_t bytes);
    // Frees a block of this or another cache (or any memory of the stream-ordered
    // pool) after the work queued on the cache's stream.
    void free(void* p);
    // While the stream is captured into a graph, its kept blocks stay (giving them
    // back would become part of the graph).
    void set_capturing(bool on);

private:
    friend void give_back_all();
    struct Kept {
        void* p;
        size_t bytes;
    };
    void give_back_locked(size_t most);  // until at most `most` bytes are kept

    const uint64_t id_;
    const int device_;
    const cudaStream_t stream_;
    bool capturing_ = false;
    size_t limit_ = 0, kept_bytes_ = 0;
    std::vector<Kept> kept_;  // oldest first
};

// Frees a block synchronously, without a handle.
void block_release(void* p);

// cudaMalloc, tried again without the kept blocks and the pool's unused memory.
cudaError_t device_malloc(void** p, size_t bytes);

}  // namespace spg
