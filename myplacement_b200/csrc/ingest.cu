// Device-side design ingest: the wirelength pass's net layout and the particle
// pin lists, built on the GPU from the flat pin CSR (buildHostLayout,
// CudaPlacementBackend.cu:784-839, produces the same CSR on the host).
//
//   1. netCountsKernel: every net's degree bucket (2, <= 4, <= 8, <= 16, <= 32,
//      larger; nets with fewer than two pins are dropped) and static pins, and per
//      block of nets and bucket the sums of both and of the degrees;
//   2. layoutScanKernel: one block scans those sums bucket by bucket; the host
//      reads the totals and allocates the layout's arrays;
//   3. placeNetsKernel: ranks within the blocks complete each net's place, pin
//      offset and first static number.  Nets keep their order within a bucket, so
//      the layout equals the host layout net for net;
//   4. copyPinsKernel: eight lanes per net copy its pins (particle, FP32 offset;
//      static pins keep their absolute FP64 position, numbered in layout order)
//      and count the particles' pins;
//   5. a scan of the counts, pinListsKernel and slotsKernel give every movable pin
//      its gradient slot: a particle's pins own a contiguous range, in ascending
//      layout order, which the gather reads in a fixed order.  A particle with more
//      than kListMax pins sends the pins through a stable radix sort instead.
// Every step is deterministic (integer sums, counts and ranks; the lists' order of
// arrival is replaced by ranks).
//
// The launches and the host's waits bound small designs: as two radix sorts and four scans
// with three read-backs the layout was 30 launches.  With 9, a 5,000-cell session of two
// iterations takes 1.50 ms instead of 1.65, and in a batch, whose sessions share the
// driver and one stream, 24 sessions of 3,000 cells 26.7 ms instead of 31 and 13 of 1,500
// cells 12.1 instead of 15; 210,000 cells are the same (6.5 ms).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "ingest.cuh"
#include "pinned.hpp"

namespace mpgp {
namespace {

constexpr int kExcluded = 6;  // the bucket key of nets with fewer than two pins

__device__ __forceinline__ int bucketOf(long long degree) {
    if (degree < 2) return kExcluded;
    return degree <= 2 ? 0 : degree <= 4 ? 1 : degree <= 8 ? 2 : degree <= 16 ? 3 : degree <= 32 ? 4 : 5;
}

// Pins of a flat CSR (Problem): the particle (negative: static) and its offset or position.
struct FlatPins {
    const int* pin_particle;
    const double* pin_x;
    const double* pin_y;
    __device__ __forceinline__ int pin(long long k, double& x, double& y) const {
        x = pin_x[k];
        y = pin_y[k];
        return pin_particle[k];
    }
};

constexpr int kBuckets = 7;   // with the excluded one
constexpr int kSums = 3;      // nets, pins, static pins
constexpr int kNetBlock = 256;
constexpr int kPinLanes = 8;  // lanes per net where its pins are read
constexpr int kListMax = 256;

// What the host reads between the passes.
struct LayoutTotals {
    int bucket_first[kBuckets + 1];  // [kExcluded] = kept nets, [kBuckets] = nets
    int kept_pins;
    int static_pins;
    int error;
    int long_list;  // a particle has more than kListMax pins
};

// sums[(bucket * kSums + q) * blocks + block] over the block's nets; static_count per net.
template <class Source>
__global__ void __launch_bounds__(kNetBlock) netCountsKernel(Source source, const long long* net_pin_start, int nets,
                                                             int* static_count, int* sums, int blocks) {
    __shared__ int total[kBuckets * kSums];
    if (threadIdx.x < kBuckets * kSums) total[threadIdx.x] = 0;
    __syncthreads();
    const int first = blockIdx.x * kNetBlock;
    const int lane = threadIdx.x & (kPinLanes - 1);
    for (int round = 0; round < kPinLanes; ++round) {
        const int n = first + round * (kNetBlock / kPinLanes) + static_cast<int>(threadIdx.x) / kPinLanes;
        const long long begin = n < nets ? net_pin_start[n] : 0;
        const long long end = n < nets ? net_pin_start[n + 1] : 0;
        const bool kept = end - begin >= 2;
        int fixed = 0;
        for (long long p = begin + lane; p < end && kept; p += kPinLanes) {
            double x, y;
            fixed += source.pin(p, x, y) < 0 ? 1 : 0;
        }
#pragma unroll
        for (int offset = kPinLanes / 2; offset > 0; offset >>= 1) fixed += __shfl_xor_sync(0xffffffffu, fixed, offset);
        if (lane == 0 && n < nets) {
            const int bucket = bucketOf(end - begin);
            static_count[n] = fixed;
            atomicAdd(&total[bucket * kSums], 1);
            if (kept) atomicAdd(&total[bucket * kSums + 1], static_cast<int>(end - begin));
            if (fixed > 0) atomicAdd(&total[bucket * kSums + 2], fixed);
        }
    }
    __syncthreads();
    if (threadIdx.x < kBuckets * kSums) sums[static_cast<size_t>(threadIdx.x) * blocks + blockIdx.x] = total[threadIdx.x];
}

// Replaces the sums of each quantity by their exclusive prefixes in (bucket, block) order and
// writes the totals.  One block: 6,000 entries a quantity for 220,000 nets.
__global__ void __launch_bounds__(1024) layoutScanKernel(int* sums, int blocks, int nets, LayoutTotals* totals) {
    __shared__ int warp_sum[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    for (int q = 0; q < kSums; ++q) {
        if (threadIdx.x == 0) carry = 0;
        __syncthreads();
        const int count = kBuckets * blocks;
        for (int base = 0; base < count; base += 1024) {
            const int k = base + static_cast<int>(threadIdx.x);
            const int bucket = k / blocks;
            const size_t at = static_cast<size_t>(bucket * kSums + q) * blocks + (k - bucket * blocks);
            const int mine = k < count ? sums[at] : 0;
            int end = mine;
#pragma unroll
            for (int step = 1; step < 32; step <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, end, step);
                if (lane >= step) end += other;
            }
            if (lane == 31) warp_sum[warp] = end;
            __syncthreads();
            if (warp == 0) {
                int sum = warp_sum[lane];
#pragma unroll
                for (int step = 1; step < 32; step <<= 1) {
                    const int other = __shfl_up_sync(0xffffffffu, sum, step);
                    if (lane >= step) sum += other;
                }
                warp_sum[lane] = sum;
            }
            __syncthreads();
            const int prefix = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + end - mine;
            if (k < count) {
                sums[at] = prefix;
                if (q == 0 && k - bucket * blocks == 0) totals->bucket_first[bucket] = prefix;
            }
            __syncthreads();
            if (threadIdx.x == 0) carry += warp_sum[31];
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            if (q == 0) totals->bucket_first[kBuckets] = nets;
            if (q == 1) totals->kept_pins = carry;
            if (q == 2) totals->static_pins = carry;
            if (q == 0) totals->error = totals->long_list = 0;
        }
        __syncthreads();
    }
}

// Each kept net's place (in bucket and net order), pin offset and first static number, and its
// weights; net_start[kept] = pins.
__global__ void __launch_bounds__(kNetBlock) placeNetsKernel(const long long* net_pin_start, const double* weight, int nets,
                                                             const int* static_count, const int* firsts, int blocks,
                                                             const LayoutTotals* totals, int* order, int* net_start,
                                                             int* static_first, float* out_weight,
                                                             double* out_weight64) {
    constexpr int kWarps = kNetBlock / 32;
    __shared__ int warp_total[kWarps][kBuckets * kSums];
    const int n = blockIdx.x * kNetBlock + static_cast<int>(threadIdx.x);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const long long degree = n < nets ? net_pin_start[n + 1] - net_pin_start[n] : 0;
    const int bucket = n < nets ? bucketOf(degree) : -1;
    const int value[kSums] = {1, degree >= 2 ? static_cast<int>(degree) : 0, n < nets ? static_count[n] : 0};
    int before[kSums] = {};
#pragma unroll
    for (int b = 0; b < kBuckets; ++b) {
#pragma unroll
        for (int q = 0; q < kSums; ++q) {
            const int mine = bucket == b ? value[q] : 0;
            int end = mine;
#pragma unroll
            for (int step = 1; step < 32; step <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, end, step);
                if (lane >= step) end += other;
            }
            if (bucket == b) before[q] = end - mine;
            if (lane == 31) warp_total[warp][b * kSums + q] = end;
        }
    }
    __syncthreads();
    if (n == 0) net_start[totals->bucket_first[kExcluded]] = totals->kept_pins;
    if (bucket < 0 || bucket == kExcluded) return;
    for (int w = 0; w < warp; ++w) {
#pragma unroll
        for (int q = 0; q < kSums; ++q) before[q] += warp_total[w][bucket * kSums + q];
    }
#pragma unroll
    for (int q = 0; q < kSums; ++q) before[q] += firsts[static_cast<size_t>(bucket * kSums + q) * blocks + blockIdx.x];
    const int k = before[0];
    order[k] = n;
    net_start[k] = before[1];
    static_first[k] = before[2];
    const double w = weight[n];
    out_weight[k] = static_cast<float>(w);
    out_weight64[k] = w;
}

// Eight lanes per kept net.
template <class Source>
__global__ void __launch_bounds__(kThreads) copyPinsKernel(Source source, const long long* net_pin_start, const int* order,
                                                           const int* net_start, const int* static_first, int kept,
                                                           int movable, int* out_particle, float2* out_offset,
                                                           double2* static_pins, int* counts, LayoutTotals* totals) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) / kPinLanes;
    const int lane = threadIdx.x & (kPinLanes - 1);
    const int group = (threadIdx.x & 31) & ~(kPinLanes - 1);  // the net's first lane in the warp
    const int dst = k < kept ? net_start[k] : 0;
    const int degree = k < kept ? net_start[k + 1] - dst : 0;
    const long long src = k < kept ? net_pin_start[order[k]] : 0;
    int number = k < kept ? static_first[k] : 0;
    for (int j0 = 0; __any_sync(0xffffffffu, j0 < degree ? 1 : 0) != 0; j0 += kPinLanes) {
        const int j = j0 + lane;
        const bool mine = j < degree;
        double x = 0.0, y = 0.0;
        const int particle = mine ? source.pin(src + j, x, y) : 0;
        const unsigned fixed = __ballot_sync(0xffffffffu, mine && particle < 0 ? 1 : 0) >> group & ((1u << kPinLanes) - 1u);
        if (mine) {
            if (particle >= 0) {
                if (particle >= movable) {
                    totals->error = 1;
                } else {
                    atomicAdd(counts + particle, 1);
                }
                out_particle[dst + j] = particle;
                out_offset[dst + j] = make_float2(static_cast<float>(x), static_cast<float>(y));
            } else {
                const int s = number + __popc(fixed & ((1u << lane) - 1u));
                out_particle[dst + j] = -s - 1;
                out_offset[dst + j] = make_float2(0.0f, 0.0f);
                static_pins[s] = make_double2(x, y);
            }
        }
        number += __popc(fixed);
    }
}

// The particles' pins in order of arrival; static pins have no slot.
__global__ void __launch_bounds__(kThreads) pinListsKernel(int pins, const int* pin_particle, int movable,
                                                           const int* particle_pin_start, int* filled, int* list,
                                                           int* slot) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pins) return;
    const int particle = pin_particle[i];
    if (particle < 0 || particle >= movable) {
        slot[i] = -1;
        return;
    }
    list[particle_pin_start[particle] + atomicAdd(filled + particle, 1)] = i;
}

// A pin's slot is its particle's first plus its rank among the particle's pins.  A thread ranks
// short lists (four pins are common), its warp longer ones.  Neighbours are on different warps:
// macros, whose lists are the long ones, stand next to one another.  Ranks are n^2 comparisons:
// with a warp for 32 neighbours and lists of up to 1,024 pins (kListMax), a backend of 20,000 cells
// with 32 modules of 1,000 pins each took 9.0 ms (3.2 with a sort of all pins) and takes 1.4, with
// 400 modules of 250 pins 2.6 and 2.0.
__global__ void __launch_bounds__(kThreads) slotsKernel(int movable, const int* particle_pin_start, const int* list,
                                                        int* slot, LayoutTotals* totals) {
    constexpr int kShort = 32;
    const int lane = threadIdx.x & 31;
    const int warp = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int p = lane * static_cast<int>((gridDim.x * blockDim.x) >> 5) + warp;
    const int first = p < movable ? particle_pin_start[p] : 0;
    const int count = p < movable ? particle_pin_start[p + 1] - first : 0;
    if (count <= kShort) {
        for (int a = 0; a < count; ++a) {
            const int pin = list[first + a];
            int rank = 0;
            for (int b = 0; b < count; ++b) rank += list[first + b] < pin ? 1 : 0;
            slot[pin] = first + rank;
        }
    }
    for (unsigned longer = __ballot_sync(0xffffffffu, count > kShort ? 1 : 0); longer != 0u; longer &= longer - 1u) {
        const int from = __ffs(static_cast<int>(longer)) - 1;
        const int start = __shfl_sync(0xffffffffu, first, from);
        const int n = __shfl_sync(0xffffffffu, count, from);
        if (n > kListMax) {
            if (lane == 0) totals->long_list = 1;
            continue;
        }
        for (int a = lane; a < n; a += 32) {
            const int pin = list[start + a];
            int rank = 0;
            for (int b = 0; b < n; ++b) rank += list[start + b] < pin ? 1 : 0;
            slot[pin] = start + rank;
        }
    }
}

// The general path's keys: the particle, or `movable` (static pins, sorted last).
__global__ void __launch_bounds__(kThreads) pinKeysKernel(int pins, const int* pin_particle, int movable, int* keys,
                                                          int* index) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pins) return;
    keys[i] = pin_particle[i] < 0 ? movable : pin_particle[i];
    index[i] = i;
}

__global__ void __launch_bounds__(kThreads) sortedSlotsKernel(int pins, const int* sorted_keys, const int* sorted_pins,
                                                              int movable, int* slot) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pins) return;
    // The movable pins take slots 0 .. (movable pins - 1), in particle order.
    slot[sorted_pins[i]] = sorted_keys[i] < movable ? i : -1;
}

int blocksFor(long long count) { return std::max(1, ceilDiv(std::max(1LL, count), kThreads)); }

int bitsFor(int value) {
    int bits = 1;
    while (bits < 31 && (1LL << bits) <= value) ++bits;
    return bits;
}

template <typename T>
void uploadVector(T* device, const std::vector<T>& host, cudaStream_t stream) {
    if (!host.empty()) {
        checkCuda(cudaMemcpyAsync(device, host.data(), host.size() * sizeof(T), cudaMemcpyHostToDevice, stream),
                  "ingest upload");
    }
}

}  // namespace

namespace {

template <class Source>
NetLayout layOutNets(const Source& source, const long long* net_pin_start, const double* weight, int nets, int movable,
                     const DeviceAllocator& lasting, Scratch& scratch, cudaStream_t stream) {
    NetLayout out;
    // The layout's lasting arrays, checked against the budget beside the scratch.
    const auto allocate = [&](std::size_t bytes, const char* what) {
        scratch.check(bytes);
        return lasting(bytes, what);
    };

    // 1-2: the sums and their prefixes.
    const int blocks = std::max(1, ceilDiv(std::max(1, nets), kNetBlock));
    int* static_count = scratch.array<int>(static_cast<std::size_t>(nets));
    int* sums = scratch.array<int>(static_cast<std::size_t>(kBuckets * kSums) * blocks);
    LayoutTotals* totals = scratch.array<LayoutTotals>(1);
    netCountsKernel<<<blocks, kNetBlock, 0, stream>>>(source, net_pin_start, nets, static_count, sums, blocks);
    layoutScanKernel<<<1, 1024, 0, stream>>>(sums, blocks, nets, totals);
    checkCuda(cudaGetLastError(), "Launch the net ordering");
    const PinnedBlock readback(sizeof(LayoutTotals), "net layout totals");
    LayoutTotals* const host = reinterpret_cast<LayoutTotals*>(readback.data());
    const auto readTotals = [&] {
        checkCuda(cudaMemcpyAsync(host, totals, sizeof(LayoutTotals), cudaMemcpyDeviceToHost, stream), "ingest");
        checkCuda(cudaStreamSynchronize(stream), "net layout");
    };
    readTotals();
    for (int b = 0; b <= kExcluded; ++b) out.bucket_first[b] = host->bucket_first[b];
    out.kept_nets = host->bucket_first[kExcluded];
    out.kept_pins = host->kept_pins;
    out.static_count = host->static_pins;

    // 3-4: the nets in their places, their pins, weights and static positions.
    const std::size_t kept = std::max<std::size_t>(1, static_cast<std::size_t>(out.kept_nets));
    const std::size_t pins = static_cast<std::size_t>(std::max(1, out.kept_pins));
    out.net_start = static_cast<int*>(allocate((static_cast<std::size_t>(nets) + 1) * sizeof(int), "net offsets"));
    out.pin_particle = static_cast<int*>(allocate(pins * sizeof(int), "pin particles"));
    out.pin_offset = static_cast<float2*>(allocate(pins * sizeof(float2), "pin offsets"));
    out.net_weight = static_cast<float*>(allocate(kept * sizeof(float), "net weights"));
    out.net_weight64 = static_cast<double*>(allocate(kept * sizeof(double), "net weights"));
    out.static_pins = static_cast<double2*>(
        allocate(std::max<std::size_t>(1, static_cast<std::size_t>(out.static_count)) * sizeof(double2), "static pins"));
    out.particle_pin_start =
        static_cast<int*>(allocate((static_cast<std::size_t>(movable) + 1) * sizeof(int), "particle pin offsets"));
    out.pin_slot = static_cast<int*>(allocate(pins * sizeof(int), "pin gradient slots"));
    int* order = scratch.array<int>(kept);
    int* static_first = scratch.array<int>(kept);
    int* list = scratch.array<int>(pins);
    // The pin counts (one past the particles stays zero) and, behind them, the lists' fill counts.
    const std::size_t particles = static_cast<std::size_t>(movable) + 1;
    int* counts = scratch.array<int>(2 * particles);
    checkCuda(cudaMemsetAsync(counts, 0, 2 * particles * sizeof(int), stream), "ingest");
    placeNetsKernel<<<blocks, kNetBlock, 0, stream>>>(net_pin_start, weight, nets, static_count, sums, blocks, totals, order,
                                                      out.net_start, static_first, out.net_weight, out.net_weight64);
    if (out.kept_nets > 0) {
        copyPinsKernel<<<blocksFor(static_cast<long long>(kPinLanes) * out.kept_nets), kThreads, 0, stream>>>(
            source, net_pin_start, order, out.net_start, static_first, out.kept_nets, movable, out.pin_particle,
            out.pin_offset, out.static_pins, counts, totals);
    }
    checkCuda(cudaGetLastError(), "Launch the pin copy");

    // 5: gradient slots.
    {
        std::size_t bytes = 0;
        checkCuda(cub::DeviceScan::ExclusiveSum(nullptr, bytes, counts, out.particle_pin_start, movable + 1, stream),
                  "scan size");
        void* temp = scratch.array<unsigned char>(bytes);
        checkCuda(cub::DeviceScan::ExclusiveSum(temp, bytes, counts, out.particle_pin_start, movable + 1, stream),
                  "particle scan");
    }
    if (out.kept_pins > 0) {
        pinListsKernel<<<blocksFor(out.kept_pins), kThreads, 0, stream>>>(
            out.kept_pins, out.pin_particle, movable, out.particle_pin_start, counts + particles, list, out.pin_slot);
        slotsKernel<<<blocksFor(movable), kThreads, 0, stream>>>(movable, out.particle_pin_start, list, out.pin_slot, totals);
        checkCuda(cudaGetLastError(), "Launch the slot assignment");
    }
    readTotals();
    require(host->error == 0, "A pin refers to a non-movable particle.");
    if (host->long_list != 0) {
        int* keys = scratch.array<int>(pins);
        int* index = scratch.array<int>(pins);
        int* sorted_keys = scratch.array<int>(pins);
        pinKeysKernel<<<blocksFor(out.kept_pins), kThreads, 0, stream>>>(out.kept_pins, out.pin_particle, movable, keys, index);
        std::size_t bytes = 0;
        const int bits = bitsFor(movable);
        checkCuda(cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys, sorted_keys, index, list, out.kept_pins, 0, bits,
                                                  stream),
                  "pin sort size");
        void* temp = scratch.array<unsigned char>(bytes);
        checkCuda(cub::DeviceRadixSort::SortPairs(temp, bytes, keys, sorted_keys, index, list, out.kept_pins, 0, bits,
                                                  stream),
                  "pin sort");
        sortedSlotsKernel<<<blocksFor(out.kept_pins), kThreads, 0, stream>>>(out.kept_pins, sorted_keys, list, movable,
                                                                             out.pin_slot);
        checkCuda(cudaGetLastError(), "Launch the slot assignment");
        checkCuda(cudaStreamSynchronize(stream), "net layout");
    }
    return out;
}

}  // namespace

NetLayout buildNetLayoutOnDevice(const Problem& p, int movable, const DeviceAllocator& lasting,
                                 const BudgetHeadroom& headroom, cudaStream_t stream) {
    const int nets = static_cast<int>(p.net_weight.size());
    const int pins_in = static_cast<int>(p.pin_particle.size());
    Scratch scratch(stream, headroom);
    // The flat CSR on the device.
    long long* net_pin_start = scratch.array<long long>(static_cast<std::size_t>(nets) + 1);
    int* pin_particle = scratch.array<int>(static_cast<std::size_t>(pins_in));
    double* pin_x = scratch.array<double>(static_cast<std::size_t>(pins_in));
    double* pin_y = scratch.array<double>(static_cast<std::size_t>(pins_in));
    double* weight = scratch.array<double>(static_cast<std::size_t>(nets));
    static_assert(sizeof(long long) == sizeof(int64_t), "64-bit offsets");
    checkCuda(cudaMemcpyAsync(net_pin_start, p.net_pin_start.data(), (static_cast<std::size_t>(nets) + 1) * 8,
                              cudaMemcpyHostToDevice, stream),
              "ingest upload");
    uploadVector(pin_particle, p.pin_particle, stream);
    uploadVector(pin_x, p.pin_x, stream);
    uploadVector(pin_y, p.pin_y, stream);
    uploadVector(weight, p.net_weight, stream);
    return layOutNets(FlatPins{pin_particle, pin_x, pin_y}, net_pin_start, weight, nets, movable, lasting, scratch,
                      stream);
}

NetLayout buildNetLayoutOnDevice(const DesignPins& pins, const long long* net_pin_start, const double* weight, int nets,
                                 int movable, const DeviceAllocator& lasting, const BudgetHeadroom& headroom,
                                 cudaStream_t stream) {
    Scratch scratch(stream, headroom);
    return layOutNets(pins, net_pin_start, weight, nets, movable, lasting, scratch, stream);
}

}  // namespace mpgp
