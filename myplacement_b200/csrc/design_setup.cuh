// A session's problem built on the device from the caller's design (design_setup.cu): the module
// map, the pin CSR's source, the static density layers, the fillers' sizes and the particle
// arrays.  Every value is the one setup.cpp forms (the same operations in the same order), so
// a session is the same whichever path set it up.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <functional>

#include "ingest.cuh"
#include "setup.hpp"

namespace mpgp {

// The rule of a session's set-up: the device takes designs of at least this many modules and
// pins whose scratch fits the budget (deviceSetupBytes).  Whole placements of two iterations
// on a B200 with 16 host CPUs, host set-up against device set-up: 25,000 items 1.49 / 1.47
// ms, 51,000 1.80 / 1.62, 101,000 2.54 / 2.02, 226,000 5.9 / 2.87, 1.06 million 20.6 / 6.6.  The
// host's part that is left is the validation, the module lists and sums that must be added in
// order; below the line both are launch and allocation latency.
constexpr int64_t kDeviceSetupItems = int64_t{1} << 15;
// Set-ups on the device at once in a process; a session that finds as many under way is set up
// on the host.  With many, each one's read-backs wait for the others' kernels and copies, and the
// helper threads of all of them for host CPUs (16 of these).  Placements of 16 iterations from
// several threads, without a limit / with 6 / with 4 / all on the host, ms a round of calls: 45,000
// cells 6 threads 14.4 / 14.3 / 14.9 / 16.7, 10 threads 28 / 22 / 22 / 22, 16 threads 55 / 32.7 /
// 33.4 / 34, 24 threads 85-108 / 49 / 50 / 51; 16 threads of 100,000 cells 88-129 / 59 / 58 / 65, of
// 20,000 39-47 / 25 / 25 / 24.5; 8 threads of 210,000 58-64 / 54 / 52 / 63, 4 threads 30 / 29 / 28 / 37.
constexpr int kDeviceSetupsAtOnce = 6;
// In a batch the set-ups of several sessions and the running rounds share one stream, so every
// read-back of a set-up on the device waits for them, while the host's set-ups run on threads of
// their own.  Batches of 16 iterations, host against device: 24 sessions of 12,000 cells (60,000
// items) 38 / 65 ms, 16 of 30,000 (151,000) 43 / 43, 12 of 80,000 (404,000) 76 / 66.
constexpr int64_t kBatchDeviceSetupItems = int64_t{1} << 18;

// Whether the static layers' lists, which the host builds and uploads, cost less than what the
// device saves otherwise.  Whole placements of two iterations, device against host, by (entries
// + 2 x fixed modules) / items: 30,000 cells 0.50: 3.3 / 4.1 ms, 0.71: 3.5 / 4.1, 0.92: 5.0 / 4.9,
// 1.7: 5.2 / 4.6, 6.6: 18 / 5.8; 210,000 cells 0.22: 9.0 / 14.9, 0.44: 17.4 / 17.1, 0.50: 13.8 /
// 17.7, 0.70: 24 / 18, 1.0: 28 / 19.6, 1.9: 55 / 23; 8,000 cells 0.16: 1.64 / 1.62, 1.0: 2.0 / 1.6.
inline bool listsPay(uint64_t entries, uint64_t fixed, int64_t items) {
    return entries + 2 * fixed <= static_cast<uint64_t>(items) / 2;
}
// The static layers' list entries: one per SiteRow or fixed module and bin row that it spans.
uint64_t staticEntryCount(const mpgp_design& design, const DerivedDesign& derived, int bins_x, int bins_y);
// More than the set-up's transient device memory and the net layout's lasting arrays together.
uint64_t deviceSetupBytes(const mpgp_design& design, uint64_t static_entries, int bins_x, int bins_y);

// The design's modules on the device: scratch that lives until the set-up is done.
struct DeviceModules {
    int count = 0;
    double* width = nullptr;
    double* height = nullptr;
    double* x = nullptr;
    double* y = nullptr;
    int* orientation = nullptr;      // null: all N
    int* movable = nullptr;          // particle -> module
    int* particle = nullptr;         // module -> particle, -1 for fixed modules
    int* pins = nullptr;             // pins per module
};
void launchMapModules(const DeviceModules& modules, int movable, cudaStream_t stream);
void launchCountPins(const int* pin_module, int pins, int* count, cudaStream_t stream);

// What the host needs to know of the static layers: their sums in bin order.
struct StaticSums {
    double fixed = 0.0;      // physical areas
    double dark = 0.0;
    double placeable = 0.0;  // sum of bin area - dark
    double charge = 0.0;     // sum of t * (fixed + dark), DensityMap::metrics(false) of the static map
};

// The static layers (staticDensity) formed per bin; static_charge (device, per bin) receives
// t * (fixed + dark).  Waits for the stream.
StaticSums staticLayersOnDevice(const mpgp_design& design, const DerivedDesign& derived, int bins_x, int bins_y,
                                double target_density, double* static_charge, const BudgetHeadroom& headroom,
                                cudaStream_t stream);

// The movable modules' areas inside the core in ascending order (createFillers), in `sorted`
// (device, `movable` doubles); areas of at most kEpsilon come last, as infinities.  Launched,
// not waited for.
void sortAreasOnDevice(const DeviceModules& modules, int movable, const Rect2& core, double* sorted,
                       const BudgetHeadroom& headroom, cudaStream_t stream);

// Hands `count` doubles of a device array to consume(values, count) piece by piece in order,
// through two pinned slots: the next piece comes down while one is consumed.
void readDown(const double* device, std::size_t count, const std::function<void(const double*, std::size_t)>& consume,
              cudaStream_t stream);

// The particle arrays (buildProblemParticles) and initial positions: movable modules, then fillers.
struct ParticleArrays {
    double2* size = nullptr;
    unsigned char* layer = nullptr;
    double* charge = nullptr;
    double* precond = nullptr;
    double2* position = nullptr;
    const double2* filler_position = nullptr;  // device
    double filler_width = 0.0, filler_height = 0.0;
    int movable = 0;
    int count = 0;
    double target_density = 0.0;
    double nominal_row_height = 0.0;
    double average_area = 0.0;  // of the movable modules
};
void launchParticles(const DeviceModules& modules, const ParticleArrays& arrays, cudaStream_t stream);

}  // namespace mpgp
