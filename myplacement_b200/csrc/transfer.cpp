// The drop-in backend's host transfers (transfer.hpp).
#include "transfer.hpp"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

#include "common.cuh"

namespace mpgp {
namespace {

// The hub's slots: 8 x 256 KB in their place made an evaluation of 260,000 particles take 782
// us instead of 592, one of 1.35 million 5.6 ms instead of 3.7.
constexpr std::size_t kHubSlots = 16;
constexpr std::size_t kHubSlotBytes = std::size_t{512} << 10;
constexpr std::size_t kSmallestSlot = std::size_t{32} << 10;
constexpr std::size_t kOwnSlots = 2;
// Arrays from this size on move through the hub: below, the hand-over to the helpers costs more
// than they save.  Evaluations with a gradient (three arrays) and without (one), this object's
// slots against the hub, us: 80 KB 98 / 105 and 57 / 63, 235 KB 121 / 128 and 65 / 70, 390 KB 158 /
// 152 and 75 / 80, 510 KB 201 / 178 and 83 / 92, 780 KB 271 / 214 and 113 / 105, 1.25 MB 384 / 265
// and 157 / 122.
constexpr std::size_t kLargeBytes = std::size_t{512} << 10;
constexpr int kHelpers = 6;
constexpr std::chrono::microseconds kSpin{300};  // a helper's wait for the next job before it sleeps

inline void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

}  // namespace

// v * 0 is 0 for a finite v and NaN otherwise.  Eight sums, so that the loop is a vector loop.
bool HostTransfer::allFinite(const double* v, std::size_t count) {
    double sum[8] = {};
    std::size_t i = 0;
    for (; i + 8 <= count; i += 8) {
        for (std::size_t j = 0; j < 8; ++j) sum[j] += v[i + j] * 0.0;
    }
    for (; i < count; ++i) sum[0] += v[i] * 0.0;
    double total = 0.0;
    for (double s : sum) total += s;
    return total == 0.0;
}

struct TransferHub::State {
    // The gate: helpers inside the job (low 16 bits), whether it is open, and its number.
    static constexpr uint64_t kOpen = uint64_t{1} << 16;
    static constexpr uint64_t kJob = uint64_t{1} << 17;
    std::atomic<uint64_t> gate{0};
    std::atomic<int> sleeping{0};
    std::atomic<bool> stopping{false};
    std::mutex mutex;                  // of the sleepers
    std::condition_variable wake;
    std::mutex owner;                  // held by the thread whose call uses the hub
    const std::function<void()>* body = nullptr;
    std::vector<std::thread> threads;

    void work() {
        uint64_t seen = 0;  // the job last run or missed
        const auto news = [&] { return gate.load(std::memory_order_acquire) / kJob != seen || stopping.load(); };
        while (!stopping.load()) {
            const auto until = std::chrono::steady_clock::now() + kSpin;
            for (int polls = 1; !news(); ++polls) {
                if ((polls & 63) == 0 && std::chrono::steady_clock::now() >= until) {
                    std::unique_lock<std::mutex> lock(mutex);
                    sleeping.fetch_add(1);
                    wake.wait(lock, news);
                    sleeping.fetch_sub(1);
                    break;
                }
                pause();
            }
            uint64_t now = gate.load(std::memory_order_acquire);
            seen = now / kJob;
            while ((now & kOpen) != 0 && now / kJob == seen) {
                if (gate.compare_exchange_weak(now, now + 1, std::memory_order_acq_rel)) {
                    (*body)();
                    gate.fetch_sub(1, std::memory_order_release);
                    break;
                }
            }
        }
    }
};

TransferHub::TransferHub()
    : ring_(kHubSlots * kHubSlotBytes, "pinned transfer ring"), state_(std::make_unique<State>()) {
    const int helpers = std::min(kHelpers, static_cast<int>(std::thread::hardware_concurrency()) / 2);
    try {
        for (int i = 0; i < helpers; ++i) state_->threads.emplace_back([s = state_.get()] { s->work(); });
    } catch (...) {  // the caller works with those that started
    }
}

TransferHub::~TransferHub() {
    {
        const std::lock_guard<std::mutex> lock(state_->mutex);
        state_->stopping.store(true);
    }
    state_->wake.notify_all();
    for (std::thread& t : state_->threads) t.join();
}

std::shared_ptr<TransferHub> TransferHub::shared() {
    static std::mutex mutex;
    static std::weak_ptr<TransferHub> hub;
    const std::lock_guard<std::mutex> lock(mutex);
    std::shared_ptr<TransferHub> held = hub.lock();
    if (held == nullptr) {
        held = std::make_shared<TransferHub>();
        hub = held;
    }
    return held;
}

bool TransferHub::acquire() { return state_->owner.try_lock(); }

void TransferHub::release() { state_->owner.unlock(); }

void TransferHub::open(const std::function<void()>& body) {
    State& s = *state_;
    s.body = &body;
    bool asleep;
    {
        // Under the sleepers' lock: a helper about to sleep sees the job or is seen asleep.
        const std::lock_guard<std::mutex> lock(s.mutex);
        s.gate.fetch_add(State::kJob + State::kOpen, std::memory_order_acq_rel);
        asleep = s.sleeping.load() > 0;
    }
    if (asleep) s.wake.notify_all();
}

void TransferHub::close() noexcept {
    State& s = *state_;
    s.gate.fetch_and(~State::kOpen, std::memory_order_acq_rel);
    while ((s.gate.load(std::memory_order_acquire) & (State::kOpen - 1)) != 0) pause();
}

HostTransfer::HostTransfer(cudaStream_t stream, std::size_t bytes) : stream_(stream) {
    if (bytes >= kLargeBytes) {
        hub_ = TransferHub::shared();
    } else {  // a small array takes one slot
        own_slot_bytes_ = std::max(kSmallestSlot, (bytes + 4095) / 4096 * 4096);
        own_ = PinnedBlock(kOwnSlots * own_slot_bytes_, "pinned transfer slots");
    }
    events_.resize(hub_ != nullptr ? kHubSlots : kOwnSlots);
    for (cudaEvent_t& e : events_) checkCuda(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "Create event");
}

HostTransfer::~HostTransfer() {
    for (cudaEvent_t e : events_) {
        if (e != nullptr) cudaEventDestroy(e);
    }
}

HostTransfer::Call::Call(HostTransfer* transfer) : transfer_(transfer) {
    if (transfer_ == nullptr) return;
    HostTransfer& t = *transfer_;
    t.helped_ = t.hub_ != nullptr && t.hub_->acquire();
    t.direct_ = t.hub_ != nullptr && !t.helped_;
    t.moved_ = 0;
    t.ring_ = t.helped_ ? t.hub_->ring() : t.own_.data();
    t.slots_ = t.helped_ ? kHubSlots : kOwnSlots;
    t.slot_bytes_ = t.helped_ ? kHubSlotBytes : t.own_slot_bytes_;
}

HostTransfer::Call::~Call() {
    if (transfer_ == nullptr) return;
    HostTransfer& t = *transfer_;
    t.cancelDownload();
    if (t.in_flight_) cudaStreamSynchronize(t.stream_);
    t.in_flight_ = false;
    if (t.helped_) t.hub_->release();
}

// The helpers' part of a download in progress.
struct HostTransfer::Download {
    explicit Download(std::size_t chunks) : copied(chunks) {}
    std::atomic<bool> stop{false};
    std::atomic<std::size_t> next{0}, ready{0};
    std::vector<std::atomic<char>> copied;
    std::function<void()> help;
};

bool HostTransfer::upload(const double* source, double* destination, std::size_t count, bool check) {
    if (direct_) {
        if (check && !allFinite(source, count)) return false;
        checkCuda(cudaMemcpyAsync(destination, source, count * sizeof(double), cudaMemcpyHostToDevice, stream_),
                  "Upload to the device");
        return true;
    }
    return move(reinterpret_cast<const unsigned char*>(source), reinterpret_cast<unsigned char*>(destination),
                count * sizeof(double), check);
}

bool HostTransfer::move(const unsigned char* source, unsigned char* destination, std::size_t bytes, bool check) {
    // Slots that an earlier move of this call still uses: its last copies, from the last slots' events.
    if (in_flight_) {
        for (std::size_t k = 0; k < std::min(slots_, moved_); ++k) {
            checkCuda(cudaEventSynchronize(events_[k]), "Wait for earlier transfers");
        }
    }
    in_flight_ = true;
    const std::size_t chunks = (bytes + slot_bytes_ - 1) / slot_bytes_;
    moved_ = chunks;
    const auto size = [&](std::size_t k) { return std::min(slot_bytes_, bytes - k * slot_bytes_); };
    std::atomic<bool> finite{true};
    // Chunks below `allowed` may use their slot and are claimed in order.
    std::atomic<std::size_t> next{0}, allowed{std::min(chunks, slots_)};
    std::atomic<bool> stop{false};
    std::vector<std::atomic<char>> filled(chunks);
    // Claims and fills one chunk, if one may be filled.
    const auto fillOne = [&]() {
        std::size_t k = next.load(std::memory_order_relaxed);
        do {
            if (k >= allowed.load(std::memory_order_acquire)) return false;
        } while (!next.compare_exchange_weak(k, k + 1, std::memory_order_relaxed));
        const unsigned char* from = source + k * slot_bytes_;
        std::memcpy(slot(k), from, size(k));
        if (check && !allFinite(reinterpret_cast<const double*>(from), size(k) / sizeof(double))) {
            finite.store(false, std::memory_order_relaxed);
        }
        filled[k].store(1, std::memory_order_release);
        return true;
    };
    const std::function<void()> help = [&] {
        while (next.load(std::memory_order_relaxed) < chunks && !stop.load(std::memory_order_acquire)) {
            if (!fillOne()) pause();
        }
    };
    struct Job {
        TransferHub* hub;
        std::atomic<bool>& stop;
        ~Job() {
            stop.store(true, std::memory_order_release);
            if (hub != nullptr) hub->close();
        }
    } job{helped_ ? hub_.get() : nullptr, stop};
    if (helped_) hub_->open(help);
    std::size_t sent = 0, done = 0;  // chunks given to the copy engine, and out of their slots
    while (sent < chunks) {
        if (filled[sent].load(std::memory_order_acquire) != 0) {
            checkCuda(cudaMemcpyAsync(destination + sent * slot_bytes_, slot(sent), size(sent), cudaMemcpyHostToDevice,
                                      stream_),
                      "Upload to the device");
            checkCuda(cudaEventRecord(events_[sent % slots_], stream_), "Record an upload");
            ++sent;
        } else if (!fillOne()) {
            // Every allowed chunk is claimed: slots that have been sent make room for more.
            if (done < sent && arrived(done)) {
                ++done;
                allowed.store(std::min(chunks, done + slots_), std::memory_order_release);
            } else {
                pause();
            }
        }
    }
    return finite.load();
}

void HostTransfer::issue(std::size_t k) {
    const Chunk& c = chunks_[k];
    checkCuda(cudaMemcpyAsync(slot(k), c.device, c.bytes, cudaMemcpyDeviceToHost,
                              stream_),
              "Download from the device");
    checkCuda(cudaEventRecord(events_[k % slots_], stream_), "Record a download");
    issued_ = k + 1;
}

bool HostTransfer::arrived(std::size_t k) {
    const cudaError_t status = cudaEventQuery(events_[k % slots_]);
    if (status == cudaSuccess) return true;
    if (status != cudaErrorNotReady) checkCuda(status, "Download from the device");
    return false;
}

void HostTransfer::startDownload(const std::vector<Piece>& pieces) {
    if (direct_) {
        pieces_ = pieces;
        return;
    }
    chunks_.clear();
    issued_ = 0;
    in_flight_ = true;
    for (const Piece& p : pieces) {
        for (std::size_t at = 0; at < p.bytes; at += slot_bytes_) {
            chunks_.push_back({static_cast<const unsigned char*>(p.device) + at, static_cast<unsigned char*>(p.host) + at,
                               std::min(slot_bytes_, p.bytes - at)});
        }
    }
    // The uploads before it on the stream have left the slots when these copies run.
    for (std::size_t k = 0; k < std::min(chunks_.size(), slots_); ++k) issue(k);
    download_ = std::make_unique<Download>(chunks_.size());
    Download* d = download_.get();
    d->help = [this, d] {
        while (d->next.load(std::memory_order_relaxed) < chunks_.size() && !d->stop.load(std::memory_order_acquire)) {
            if (!copyOne(*d)) pause();
        }
    };
    if (helped_) hub_->open(d->help);
}

// Claims one chunk that has arrived in its slot and copies it to its host array.
bool HostTransfer::copyOne(Download& d) {
    std::size_t k = d.next.load(std::memory_order_relaxed);
    do {
        if (k >= d.ready.load(std::memory_order_acquire)) return false;
    } while (!d.next.compare_exchange_weak(k, k + 1, std::memory_order_relaxed));
    std::memcpy(chunks_[k].host, slot(k), chunks_[k].bytes);
    d.copied[k].store(1, std::memory_order_release);
    return true;
}

void HostTransfer::cancelDownload() noexcept {
    if (download_ == nullptr) return;
    download_->stop.store(true, std::memory_order_release);
    if (helped_) hub_->close();
    download_.reset();
}

void HostTransfer::finishDownload() {
    if (direct_) {
        for (const Piece& p : pieces_) {
            checkCuda(cudaMemcpyAsync(p.host, p.device, p.bytes, cudaMemcpyDeviceToHost, stream_), "Download from the device");
        }
        checkCuda(cudaStreamSynchronize(stream_), "Download from the device");
        return;
    }
    Download& d = *download_;
    const std::size_t chunks = chunks_.size();
    std::size_t done = 0, out = 0;  // chunks that have arrived, and (in order) been copied
    while (out < chunks) {
        if (done < issued_ && arrived(done)) {
            ++done;
            d.ready.store(done, std::memory_order_release);
        } else if (!copyOne(d)) {
            pause();
        }
        while (out < chunks && d.copied[out].load(std::memory_order_acquire) != 0) {
            if (out + slots_ < chunks) issue(out + slots_);
            ++out;
        }
    }
    cancelDownload();  // nothing is left to copy
}

}  // namespace mpgp
