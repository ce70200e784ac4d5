// DeviceMemory: pools and kept blocks of a handle's calls (device_memory.h).
#include "device_memory.h"

#include <algorithm>
#include <cstdint>
#include <mutex>

namespace spg {
namespace {

// The device's pool of temporaries, made on first use; its unused memory stays until
// the driver needs it, as the default pool's does (spg_create).
cudaMemPool_t temporaries_pool(int device) {
    struct Pools {
        std::mutex lock;
        std::vector<cudaMemPool_t> of_device;
    };
    static Pools* pools = new Pools;  // outlives handles destroyed at exit
    std::lock_guard<std::mutex> g(pools->lock);
    if (pools->of_device.size() <= static_cast<size_t>(device)) pools->of_device.resize(device + 1, nullptr);
    cudaMemPool_t& pool = pools->of_device[device];
    if (!pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            pool = nullptr;
        } else {
            uint64_t threshold = UINT64_MAX;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold);
        }
    }
    return pool;
}

// Small blocks come in steps of an eighth where there is no budget, so that calls of
// about the same size share them; the pools' own granularity is 512 bytes.
size_t block_size(size_t bytes, bool exact) {
    size_t step = 512;
    if (!exact && bytes <= DeviceMemory::kKeptBlock)
        for (size_t p = 4096; p * 2 <= bytes; p *= 2) step = p / 4;
    return std::max(step, (bytes + step - 1) / step * step);
}

}  // namespace

DeviceMemory::DeviceMemory(int device, cudaStream_t stream, size_t budget)
    : stream_(stream), budget_(budget), pool_(temporaries_pool(device)) {
    kept_.reserve(kKeptCount + 1);
}

DeviceMemory::~DeviceMemory() { give_back(); }

cudaError_t DeviceMemory::temporary(Block* b, size_t bytes, bool may_leave) noexcept {
    const size_t want = block_size(bytes, budget_ != 0);
    const size_t most = budget_ || may_leave ? want : want + want / 4;
    if (budget_ && live_ + kept_bytes_ + want > budget_) give_back();
    size_t best = kept_.size();  // the smallest kept block that is not much too large
    for (size_t i = 0; i < kept_.size(); ++i)
        if (kept_[i].bytes >= want && kept_[i].bytes <= most &&
            (best == kept_.size() || kept_[i].bytes < kept_[best].bytes))
            best = i;
    if (best < kept_.size()) {
        *b = kept_[best];
        kept_.erase(kept_.begin() + static_cast<std::ptrdiff_t>(best));
        kept_bytes_ -= b->bytes;
        live_ += b->bytes;
        return cudaSuccess;
    }
    const auto alloc = [&] {
        return pool_ ? cudaMallocFromPoolAsync(&b->p, want, pool_, stream_) : cudaMallocAsync(&b->p, want, stream_);
    };
    cudaError_t e = alloc();
    if (e == cudaErrorMemoryAllocation && !kept_.empty()) {
        cudaGetLastError();
        give_back();
        cudaStreamSynchronize(stream_);
        e = alloc();
    }
    if (e != cudaSuccess) return e;
    b->bytes = want;
    live_ += want;
    return cudaSuccess;
}

cudaError_t DeviceMemory::result(Block* b, size_t bytes) noexcept {
    b->bytes = 0;
    const size_t want = std::max<size_t>(bytes, 16);
    cudaError_t e = cudaMallocAsync(&b->p, want, stream_);
    if (e == cudaErrorMemoryAllocation && !kept_.empty()) {
        cudaGetLastError();
        give_back();
        cudaStreamSynchronize(stream_);
        e = cudaMallocAsync(&b->p, want, stream_);
    }
    return e;
}

Block DeviceMemory::let_go(Block b) noexcept {
    live_ -= b.bytes;
    b.bytes = 0;
    return b;
}

void DeviceMemory::free(Block b) noexcept {
    if (!b.p) return;
    live_ -= b.bytes;
    if (b.bytes == 0 || b.bytes > kKeptBlock || (budget_ && live_ + kept_bytes_ + b.bytes > budget_)) {
        cudaFreeAsync(b.p, stream_);
        return;
    }
    kept_.push_back(b);  // (room was reserved)
    kept_bytes_ += b.bytes;
    size_t n = 0;
    for (; kept_bytes_ > kKeptBytes || kept_.size() - n > kKeptCount; ++n) {
        cudaFreeAsync(kept_[n].p, stream_);
        kept_bytes_ -= kept_[n].bytes;
    }
    kept_.erase(kept_.begin(), kept_.begin() + static_cast<std::ptrdiff_t>(n));
}

void DeviceMemory::give_back() noexcept {
    for (const Block& b : kept_) cudaFreeAsync(b.p, stream_);
    kept_.clear();
    kept_bytes_ = 0;
}

}  // namespace spg
