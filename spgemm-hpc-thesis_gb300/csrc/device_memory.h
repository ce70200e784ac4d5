// Device memory of a handle's calls.
//
// A call allocates a dozen temporary arrays, the largest of 8 bytes per scalar
// product, and its result.  The two come from different stream-ordered pools:
// results, which outlive the call, from the device's default pool, temporaries from
// one that the handles of a device share for nothing else.  In one pool a call of
// 600 M products spent 3-6 ms mapping memory anew whenever the previous result was
// still alive, because the pieces between results fitted no array; apart, an
// allocation of a repeated call takes 1-5 us, at 8 M to 600 M products.  Both pools
// keep what is freed into them, and the driver takes unused memory of either for any
// other allocation of the process that would fail (a cudaMalloc that needs 20 of 40
// unused GB: 64 ms).
//
// A handle keeps the temporaries of up to kKeptBlock bytes itself, at most kKeptBytes
// of them (they go back with the handle, or when an allocation fails): a pair of
// calls to the pool takes 2-3 us, and a small product has a dozen temporaries.  A
// 1,000-row square takes 178 us a call so, 187 with the line at 4 MiB, 174 with every
// block kept, results too: that put up to 1/16 of the device out of the reach of
// other allocations.  A handle with a budget keeps blocks only while they and those
// in use stay within it, and takes them in the sizes asked for.
//
// Used by the handle's calls only, one at a time: no lock.
#pragma once

#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

namespace spg {

// A temporary array, or with bytes == 0 memory that belongs to a result.
struct Block {
    void* p = nullptr;
    size_t bytes = 0;
};

class DeviceMemory {
public:
    static constexpr size_t kKeptBlock = size_t{32} << 20;
    static constexpr size_t kKeptBytes = size_t{128} << 20;
    static constexpr size_t kKeptCount = 256;

    DeviceMemory(int device, cudaStream_t stream, size_t budget);
    ~DeviceMemory();
    DeviceMemory(const DeviceMemory&) = delete;
    DeviceMemory& operator=(const DeviceMemory&) = delete;

    // At least `bytes` for work on the handle's stream; where the block may become
    // memory of a result, at most an eighth more, and no more above kKeptBlock.
    cudaError_t temporary(Block* b, size_t bytes, bool may_leave) noexcept;
    // Exactly `bytes` for a result that the caller keeps.
    cudaError_t result(Block* b, size_t bytes) noexcept;
    // Frees a block after the work queued on the handle's stream; memory of results
    // (of any handle) has bytes == 0.
    void free(Block b) noexcept;
    // The block becomes memory of a result.
    Block let_go(Block b) noexcept;
    // The kept blocks go back to the pool, for an allocation that failed.
    void give_back() noexcept;

private:
    const cudaStream_t stream_;
    const size_t budget_;
    const cudaMemPool_t pool_;  // of temporaries; nullptr: the default pool
    size_t live_ = 0, kept_bytes_ = 0;
    std::vector<Block> kept_;  // oldest first
};

}  // namespace spg
