// Device-side design ingest (ingest.cu): the wirelength pass's bucketed net
// layout and the particle pin lists, built on the GPU from a Problem's pin CSR.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <functional>
#include <utility>
#include <vector>

#include "common.cuh"
#include "setup.hpp"

namespace mpgp {

// Device memory for the layout's lasting arrays (the engine's budgeted arena).
using DeviceAllocator = std::function<void*(std::size_t bytes, const char* what)>;
// Bytes the budget still allows (transient scratch counts against it while it lives).
using BudgetHeadroom = std::function<uint64_t()>;

// Stream-ordered scratch from the device's pool, released when it goes out of scope.  While it
// lives it counts against the engine's device-memory budget like the lasting arrays.
class Scratch {
public:
    Scratch(cudaStream_t stream, BudgetHeadroom headroom) : stream_(stream), headroom_(std::move(headroom)) {}
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch() {
        for (void* p : blocks_) cudaFreeAsync(p, stream_);
    }
    // Fails unless `bytes` more fit in the budget beside the scratch held now.
    void check(std::size_t bytes) const {
        if (held_ + bytes > headroom_()) {
            fail(MPGP_ERR_BUDGET, "CUDA allocation budget exceeded while ingesting the design.");
        }
    }
    template <typename T>
    T* array(std::size_t count) {
        const std::size_t bytes = std::max<std::size_t>(1, count) * sizeof(T);
        check(bytes);
        void* p = nullptr;
        int device = 0;
        checkCuda(cudaGetDevice(&device), "Query the current device");
        checkCuda(cudaMallocFromPoolAsync(&p, bytes, devicePool(device), stream_), "ingest scratch");
        blocks_.push_back(p);
        held_ += bytes;
        return static_cast<T*>(p);
    }

    [[nodiscard]] uint64_t held() const { return held_; }

private:
    cudaStream_t stream_;
    BudgetHeadroom headroom_;
    std::vector<void*> blocks_;
    uint64_t held_ = 0;
};

#ifdef __CUDACC__
// Pins of a design: its module's particle and the offset in the module's orientation
// (transformOffset, PlacementDatabase.cpp:55-68), or a fixed module's absolute position
// (buildProblemPins).
struct DesignPins {
    const int* pin_module;
    const double* offset_x;
    const double* offset_y;
    const int* module_particle;
    const int* module_orientation;  // null: all N
    const double* module_x;
    const double* module_y;
    __device__ __forceinline__ int pin(long long k, double& x, double& y) const {
        const int m = pin_module[k];
        const double ox = offset_x[k], oy = offset_y[k];
        switch (module_orientation != nullptr ? module_orientation[m] : 0) {
            case 1: x = -ox; y = -oy; break;
            case 2: x = -oy; y = ox; break;
            case 3: x = oy; y = -ox; break;
            case 4: x = -ox; y = oy; break;
            case 5: x = ox; y = -oy; break;
            case 6: x = oy; y = ox; break;
            case 7: x = -oy; y = -ox; break;
            default: x = ox; y = oy; break;
        }
        const int particle = module_particle[m];
        if (particle < 0) {
            x = module_x[m] + x;
            y = module_y[m] + y;
        }
        return particle;
    }
};
#endif

struct NetLayout {
    int kept_nets = 0;            // nets with two or more pins, in bucket order
    int kept_pins = 0;
    int static_count = 0;
    int bucket_first[7] = {};     // first net of buckets 0..5; [6] = kept_nets
    int* net_start = nullptr;     // kept_nets + 1 pin offsets
    int* pin_particle = nullptr;  // particle, or -(static index) - 1
    float2* pin_offset = nullptr; // FP32 offset from the particle centre
    double2* static_pins = nullptr;
    float* net_weight = nullptr;  // FP32 (wirelength pass)
    double* net_weight64 = nullptr;  // FP64 (RUDY)
    int* particle_pin_start = nullptr;  // movable + 1
    int* pin_slot = nullptr;      // a pin's slot in its particle's range, -1 for static pins
};

NetLayout buildNetLayoutOnDevice(const Problem& problem, int movable, const DeviceAllocator& allocate,
                                 const BudgetHeadroom& headroom, cudaStream_t stream);
#ifdef __CUDACC__
// The same from a design's arrays on the device (offsets and weights in the caller's net order).
NetLayout buildNetLayoutOnDevice(const DesignPins& pins, const long long* net_pin_start, const double* weight, int nets,
                                 int movable, const DeviceAllocator& allocate, const BudgetHeadroom& headroom,
                                 cudaStream_t stream);
#endif

}  // namespace mpgp
