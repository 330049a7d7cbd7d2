// Pinned, mapped host memory kept between engines.
//
// The driver backs small pinned allocations with a chunk that it pins when the first
// one is made and releases with the last one: a process that places one design after
// another paid for that chunk (3 ms, and 0.7 ms to release it) in every session, for a
// record of a few hundred bytes.  Blocks given back here stay pinned for the next
// engine, up to kPinnedKept bytes in all; beyond that those that nobody has asked for the
// longest are freed.  (The backends' 8 MB ring has to find room: with 16 MB, and the block that
// came back freed instead, it was pinned anew with every first backend once others had left their
// slots here.  Making a backend of 45,000 cells then took 11 ms and takes 3.3, from four threads
// at once 28 and 5.2; 6.3 and 7.5 with allocations per backend.)
//
// Measured on one B200 box, whole placements with 16 iterations: 7.1 ms with allocations
// per session and 3.8 ms with kept blocks for 5,000 cells, 28.9 and 25.6 ms for 210,000;
// a batch of 24 designs of about 3,000 cells 46 and 36 ms.
#pragma once

#include <cstddef>

namespace mpgp {

constexpr std::size_t kPinnedKept = std::size_t{32} << 20;

// One block of at least `bytes` pinned bytes (portable: usable from every device, and
// addressable by kernels), its contents undefined.  Movable; given back when destroyed.
// The owner must have finished every copy and kernel that uses the block by then.
class PinnedBlock {
public:
    PinnedBlock() = default;
    explicit PinnedBlock(std::size_t bytes, const char* what);
    ~PinnedBlock() { release(); }
    PinnedBlock(PinnedBlock&& other) noexcept : data_(other.data_), size_(other.size_) { other.data_ = nullptr; }
    PinnedBlock& operator=(PinnedBlock&& other) noexcept;
    PinnedBlock(const PinnedBlock&) = delete;
    PinnedBlock& operator=(const PinnedBlock&) = delete;
    [[nodiscard]] unsigned char* data() const { return data_; }
    [[nodiscard]] std::size_t size() const { return data_ != nullptr ? size_ : 0; }

private:
    void release() noexcept;
    unsigned char* data_ = nullptr;
    std::size_t size_ = 0;
};

}  // namespace mpgp
