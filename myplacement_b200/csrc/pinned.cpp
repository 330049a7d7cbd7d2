// The pinned blocks kept between engines (pinned.hpp).
#include "pinned.hpp"

#include <cuda_runtime.h>

#include <iterator>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace mpgp {
namespace {

// The kept blocks by size.  Never destroyed: at process exit the driver may be gone
// before a static destructor would run, and it releases the memory itself.
struct Kept {
    std::mutex mutex;
    std::multimap<std::size_t, unsigned char*> blocks;
    std::size_t bytes = 0;
};

Kept& kept() {
    static Kept* instance = new Kept;
    return *instance;
}

// Sizes are powers of two from 4 KB up, so a block serves every request of its class.
std::size_t classOf(std::size_t bytes) {
    std::size_t size = 4096;
    while (size < bytes) size *= 2;
    return size;
}

}  // namespace

PinnedBlock::PinnedBlock(std::size_t bytes, const char* what) {
    const std::size_t size = classOf(bytes);
    Kept& k = kept();
    {
        const std::lock_guard<std::mutex> lock(k.mutex);
        const auto found = k.blocks.find(size);
        if (found != k.blocks.end()) {
            data_ = found->second;
            size_ = size;
            k.blocks.erase(found);
            k.bytes -= size;
            return;
        }
    }
    void* p = nullptr;
    checkCuda(cudaHostAlloc(&p, size, cudaHostAllocMapped | cudaHostAllocPortable), what);
    data_ = static_cast<unsigned char*>(p);
    size_ = size;
}

PinnedBlock& PinnedBlock::operator=(PinnedBlock&& other) noexcept {
    if (this != &other) {
        release();
        data_ = std::exchange(other.data_, nullptr);
        size_ = other.size_;
    }
    return *this;
}

void PinnedBlock::release() noexcept {
    if (data_ == nullptr) return;
    unsigned char* p = std::exchange(data_, nullptr);
    Kept& k = kept();
    {
        const std::lock_guard<std::mutex> lock(k.mutex);
        if (k.bytes + size_ <= kPinnedKept) {
            try {
                k.blocks.emplace(size_, p);
                k.bytes += size_;
                return;
            } catch (...) {  // no memory for the entry: free the block below
            }
        }
    }
    cudaFreeHost(p);
}

}  // namespace mpgp
