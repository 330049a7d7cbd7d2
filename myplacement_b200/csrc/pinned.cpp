// The pinned blocks kept between engines (pinned.hpp).
#include "pinned.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <iterator>
#include <list>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace mpgp {
namespace {

// The kept blocks, the one given back last in front.  Never destroyed: at process exit the driver
// may be gone before a static destructor would run, and it releases the memory itself.
struct Kept {
    struct Block {
        std::size_t size;
        unsigned char* data;
    };
    std::mutex mutex;
    std::list<Block> blocks;
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
        const auto found = std::find_if(k.blocks.begin(), k.blocks.end(), [&](const Kept::Block& b) { return b.size == size; });
        if (found != k.blocks.end()) {
            data_ = found->data;
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
    std::list<Kept::Block> freed;
    {
        const std::lock_guard<std::mutex> lock(k.mutex);
        try {
            k.blocks.push_front({size_, p});
            k.bytes += size_;
            p = nullptr;
        } catch (...) {  // no memory for the entry: free the block below
        }
        // The blocks that nobody has asked for the longest make room.
        while (k.bytes > kPinnedKept) {
            k.bytes -= k.blocks.back().size;
            freed.splice(freed.end(), k.blocks, std::prev(k.blocks.end()));
        }
    }
    for (const Kept::Block& b : freed) cudaFreeHost(b.data);
    if (p != nullptr) cudaFreeHost(p);
}

}  // namespace mpgp
