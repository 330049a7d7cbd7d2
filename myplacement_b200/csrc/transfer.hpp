// Copies between a caller's pageable arrays and the device for the drop-in backend.
//
// A pageable cudaMemcpy is staged by the driver on the calling thread: one evaluation of
// 260,000 particles spent 210 us uploading 4 MB and 590 us downloading 8 MB beside 120 us on
// the device, and checked the positions in a pass of its own (280 us).  Here the data go
// through a ring of pinned slots: a few helper threads copy (and check) slot by slot while the
// copy engine moves the slots before, and the downloads are on the stream before the
// evaluation has ended.
//
// Measured on a B200 with 16 host CPUs, whole evaluations through the Python mirror, before
// and after: 5,000 cells 163 and 113 us, 37,411 cells 457 and 235, 210,000 cells 1,748 and 589
// (273 instead of 789 without a gradient), 1.3 million cells 9.9 and 4.0 ms.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <functional>
#include <memory>
#include <vector>

#include "pinned.hpp"

namespace mpgp {

// What the process's large transfers share: a ring of pinned slots (8 MB: pinning that much
// takes 20 ms, so not one a backend) and helper threads.  Made with the first HostTransfer of
// large arrays and given up with the last; used by one call at a time.  The helpers spin for
// kSpin after a job (transfer.cpp) before they sleep: on a virtual machine waking them takes
// longer than the copies they help with, and a controller's next evaluation follows soon.
class TransferHub {
public:
    TransferHub();
    ~TransferHub();
    TransferHub(const TransferHub&) = delete;
    TransferHub& operator=(const TransferHub&) = delete;
    static std::shared_ptr<TransferHub> shared();

    // The right to use the ring and the helpers; fails while another thread has it.
    bool acquire();
    void release();
    [[nodiscard]] unsigned char* ring() const { return ring_.data(); }
    // Opens a job: helpers that are free, now or while it is open, call body() once.  body must
    // not throw.  close() waits for the helpers inside it; one that has not begun will not.
    void open(const std::function<void()>& body);
    void close() noexcept;

private:
    struct State;
    PinnedBlock ring_;
    std::unique_ptr<State> state_;
};

// One stream's transfers, used by one host thread at a time, within a Call.
class HostTransfer {
public:
    // `bytes`: the size of the arrays that will be moved.
    HostTransfer(cudaStream_t stream, std::size_t bytes);
    ~HostTransfer();
    HostTransfer(const HostTransfer&) = delete;
    HostTransfer& operator=(const HostTransfer&) = delete;

    // One call's transfers (null: none).  Large arrays move through the hub, unless another
    // thread's call has it; then the driver copies them.  Small arrays move through two slots of
    // this object's own.  At the end a download not finished is given up and copies that nothing
    // has waited for (settled) are waited for.
    //
    // Calls of several threads at once, by the driver's copies before there was a hub / beside it
    // / with two 64 KB slots beside it, ms a round of calls: 210,000 cells 2 threads 1.78 / 0.95 /
    // 1.09, 8 threads 4.4 / 3.08 / 4.15; 45,000 cells 4 threads 0.82 / 0.49 / 0.66, without a
    // gradient 0.27 / 0.18 / 0.31; 1.3 million cells 2 threads 8.8 / 5.3 / 6.2.
    class Call {
    public:
        explicit Call(HostTransfer* transfer);
        ~Call();
        Call(const Call&) = delete;
        Call& operator=(const Call&) = delete;

    private:
        HostTransfer* transfer_;
    };

    // Large arrays: checked while they are copied, by the helpers too (or before, by the caller).
    [[nodiscard]] bool large() const { return hub_ != nullptr; }
    // Whether all values are finite, in one pass on the calling thread.
    static bool allFinite(const double* values, std::size_t count);
    // Copies `count` doubles to the device on the stream.  With `check`, returns whether all
    // are finite.  The source has been read when this returns.
    bool upload(const double* source, double* destination, std::size_t count, bool check);

    struct Piece {
        const void* device = nullptr;
        void* host = nullptr;
        std::size_t bytes = 0;
    };
    // Puts the first slots' copies behind the work already on the stream and wakes the
    // helpers; nothing is written to the host arrays before finishDownload, which copies
    // everything out.
    void startDownload(const std::vector<Piece>& pieces);
    void finishDownload();
    // The caller has waited for everything on the stream.
    void settled() { in_flight_ = false; }

private:
    struct Chunk {
        const unsigned char* device;
        unsigned char* host;
        std::size_t bytes;
    };
    struct Download;
    [[nodiscard]] unsigned char* slot(std::size_t k) const { return ring_ + (k % slots_) * slot_bytes_; }
    bool move(const unsigned char* source, unsigned char* destination, std::size_t bytes, bool check);
    void issue(std::size_t k);
    [[nodiscard]] bool arrived(std::size_t k);
    bool copyOne(Download& download);
    void cancelDownload() noexcept;

    cudaStream_t stream_;
    std::shared_ptr<TransferHub> hub_;  // of large arrays
    PinnedBlock own_;
    std::size_t own_slot_bytes_ = 0;
    // The call's ring: the hub's or this object's own, or none.
    bool helped_ = false;
    bool direct_ = false;  // the driver's own copies
    std::vector<Piece> pieces_;  // then, of the download in progress
    unsigned char* ring_ = nullptr;
    std::size_t slots_ = 0, slot_bytes_ = 0;
    std::vector<cudaEvent_t> events_;
    std::vector<Chunk> chunks_;  // of the download in progress
    std::unique_ptr<Download> download_;
    std::size_t issued_ = 0;
    std::size_t moved_ = 0;   // chunks of the call's last move
    bool in_flight_ = false;  // copies that nothing has waited for may still use the slots
};

}  // namespace mpgp
