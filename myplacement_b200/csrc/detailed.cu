// Detailed placement by window reordering, the orderings evaluated on the
// device: the reference's CUDA detailed-placement backend
// (src/placement/cuda/CudaDetailedPlacementBackend.cu:144-709) with the CPU rule
// it keeps for the windows the device does not take (:328-354).
//
// Each pass cuts the rows into segments of abutting standard cells and the
// segments into windows of four consecutive cells, staggered by two cells on
// odd passes.  One warp evaluates one window: lanes 0..23 each place the cells
// in one of the 24 orders (lexicographic, the order std::next_permutation
// visits) and sum the weighted HPWL of the window's nets; lane 24 sums it for
// the placement as it is.  The sum with fused multiply-adds (what the
// reference's kernel compiles to) picks the best order.
//
// The reference then accepts the windows one after another, each by its host
// arithmetic (products and sums rounded separately) against the placement the
// earlier acceptances left.  A second kernel evaluates that rule
// speculatively: every window's before and after values on the assumption
// that each earlier window decided as the previous round said.  The segment ends
// the reference keeps on the host (two or three cells, every order by its
// exhaustive rule) go through a tail kernel the same way, after the four-cell
// windows.  The result is the reference's exactly.
//
// Whole passes run on the device (placeOnDevice): it builds the windows and
// repeats the rounds until one changes no decision.  Where the host has to look,
// it builds the windows (buildWindows), the device runs a few rounds, and the
// host walks the windows in the reference's order: it takes the device's values
// unless a net of the window belongs to an earlier window whose actual decision
// differed from the assumption, and re-evaluates only those windows.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#include <memory>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "design_setup.cuh"
#include "detailed.hpp"
#include "ingest.cuh"
#include "pinned.hpp"
#include "setup.hpp"
#include "workers.hpp"

namespace mpgp {
namespace {

constexpr int kWindow = 4;
constexpr int kOrders = 24;
constexpr int kCurrentLane = kOrders;  // the lane that evaluates the placement as it is
constexpr int kWindowsPerBlock = 8;
constexpr int kSpeculations = 3;  // rounds of speculative re-decision beside the host's walk
constexpr int kOrientationUnknown = 8;
constexpr double kLargest = std::numeric_limits<double>::max();

// Order k (0..n!-1) of n <= 4 cells in lexicographic order (the order
// std::next_permutation visits from 0, 1, ..., n - 1), as 4-bit fields: field
// i is the window cell placed i-th.  The Lehmer digits of k (k / (n-1)!, then
// the remainder's digit for (n-2)!, ...) each pick a field of the cells not yet
// placed (`pool`, packed the same way) and remove it.
__host__ __device__ inline unsigned orderCode(int k, int n = kWindow) {
    unsigned pool = 0x3210u;
    unsigned code = 0u;
    int rest = k;
#pragma unroll
    for (int i = 0; i < kWindow - 1; ++i) {
        if (i >= n - 1) break;
        const int place = n - 1 - i;
        const int factorial = place == 3 ? 6 : place == 2 ? 2 : 1;
        const unsigned d = static_cast<unsigned>(rest / factorial);
        rest %= factorial;
        code |= ((pool >> (4u * d)) & 0xFu) << (4u * static_cast<unsigned>(i));
        pool = (pool & ((1u << (4u * d)) - 1u)) | ((pool >> (4u * (d + 1u))) << (4u * d));
    }
    return code | ((pool & 0xFu) << (4u * static_cast<unsigned>(n - 1)));
}

__host__ __device__ inline int factorialOf(int n) { return n == 4 ? 24 : n == 3 ? 6 : n == 2 ? 2 : 1; }

inline void orderOf(int k, int order[kWindow], int n = kWindow) {
    const unsigned code = orderCode(k, n);
    for (int i = 0; i < n; ++i) order[i] = static_cast<int>((code >> (4u * static_cast<unsigned>(i))) & 0xFu);
}

// alignUp(width, 0, spacing) (DetailedPlacer.cpp:67-70), products and sums
// rounded separately.
__device__ inline double roundedWidthDevice(double width, double spacing) {
    return spacing <= kEpsilon ? width : __dmul_rn(ceil((width - kEpsilon) / spacing), spacing);
}

struct WindowArrays {
    const int4* modules;
    const double* start_x;  // lower-left x of the window's first cell
    const double* bottom;
    const double* spacing;
    const int* net_start;   // windows + 1
    const int* nets;
};

// What a window of a pass is: evaluated as a four-cell window, as a tail (a segment end), or not.
enum WindowKind : uint8_t { kNotEvaluated = 0, kFourCells = 1, kTail = 2 };

// Rounds of re-decision until nothing changes (stamp != null): in round k a window is
// evaluated again if a window that shares a net with it changed its decision in round k - 1
// (every window in round 1), otherwise it decides as before.  A round after one without a
// change does nothing.
struct Rounds {
    int round = 0;
    int* stamp = nullptr;    // per net: the latest round that has to look at its windows again
    int* changed = nullptr;  // per round: decisions that differ from the round's input
};

// Whether the warp's window has nothing new to decide in this round.
__device__ __forceinline__ bool settledWindow(const Rounds& r, const int* nets, int first, int last) {
    if (r.round <= 1) return false;
    bool again = false;
    for (int e = first + static_cast<int>(threadIdx.x & 31); e < last; e += 32) again = again || __ldcg(r.stamp + nets[e]) >= r.round;
    return __any_sync(0xffffffffu, again ? 1 : 0) == 0;
}

// The window changed its decision in this round: its nets' windows are looked at in the next one.
__device__ __forceinline__ void stampWindow(const Rounds& r, const int* nets, int first, int last) {
    for (int e = first + static_cast<int>(threadIdx.x & 31); e < last; e += 32) __stcg(r.stamp + nets[e], r.round + 1);
    if ((threadIdx.x & 31) == 0) atomicAdd(r.changed + r.round, 1);
}

constexpr int kPinChunk = 64;  // pins a warp loads at a time, two per lane

// The pins of up to 32 nets one net after another, so that a warp's lanes load a pin each
// whatever the nets' degrees: lane e holds net e's part.
struct PinRun {
    int offset = 0;  // of the net's first pin in the run
    int degree = 0;
    int shift = 0;   // first pin - offset
    int count = 0;   // nets
    int total = 0;   // pins
};

__device__ __forceinline__ PinRun pinRun(const int* nets, int count, const int* net_pin_start) {
    const int lane = threadIdx.x & 31;
    PinRun run;
    run.count = count;
    int first = 0;
    if (lane < count) {
        const int net = nets[lane];
        first = net_pin_start[net];
        run.degree = net_pin_start[net + 1] - first;
    }
    int end = run.degree;  // inclusive scan
#pragma unroll
    for (int step = 1; step < 32; step <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, end, step);
        if (lane >= step) end += other;
    }
    run.offset = end - run.degree;
    run.shift = first - run.offset;
    run.total = __shfl_sync(0xffffffffu, end, 31);
    return run;
}

// The pin at place at + lane of the run (a whole warp calls it; past the end, some pin of the
// run).  The nets of a window have a pin at least, so each begins at a place of its own.
__device__ __forceinline__ int pinAt(const PinRun& run, int at) {
    const int lane = threadIdx.x & 31;
    const bool net = lane < run.count;
    const int begun = __popc(__ballot_sync(0xffffffffu, net && run.offset < at ? 1 : 0));
    const unsigned begins = __reduce_or_sync(
        0xffffffffu, net && run.offset >= at && run.offset < at + 32 ? 1u << (run.offset - at) : 0u);
    const int e = begun + __popc(begins & (0xffffffffu >> (31 - lane))) - 1;
    return __shfl_sync(0xffffffffu, run.shift, e) + min(at + lane, run.total - 1);
}

// Up to 32 nets of a window, as the lanes that try the window's orders need them: of each net
// the box of its pins on other cells, which no order moves, and its pins on the window's own
// cells.  The chains of loads (pin, cell, centre) bound the kernels; a warp follows 64 of them
// at once and every lane then has only the window's own pins to place.  Of 210,000 cells the
// tails took 344 us with every lane walking every pin, 182 with a net per lane and 124 so; the
// four-cell windows 745, 410 and 430, and 220 (with 50 for the extremes) from the nets'
// extremes below: a window of the design touches 16 nets of 153 pins, 16 of them its own.
constexpr int kOwnPins = 64;  // of a batch of nets (about 14 are common); more take the pin by pin walk
struct WindowNets {
    double2 point[kPinChunk];
    double2 low[32];
    double2 high[32];
    double2 offset[kOwnPins];
    uint8_t cell[kOwnPins];
    uint8_t start[36];  // the nets' ranges of the own pins
};

__device__ __forceinline__ int slotOf(const int (&module)[kWindow], int m) {
    int slot = -1;
#pragma unroll
    for (int i = 0; i < kWindow; ++i) slot = module[i] == m ? i : slot;  // a window's cells are distinct
    return slot;
}

// Gathers `count` <= 32 nets (a whole warp); false, for every lane, with more than kOwnPins own
// pins.  position(p, m): a pin of another cell; offset(p, m): an own pin's offset.
template <typename Position, typename Offset>
__device__ __forceinline__ bool gatherNets(WindowNets& g, const int* nets, int count, const int* net_pin_start,
                                           const int* pin_module, const int (&module)[kWindow],
                                           const Position& position, const Offset& offset) {
    const int lane = threadIdx.x & 31;
    const PinRun run = pinRun(nets, count, net_pin_start);
    double2 low = make_double2(kLargest, kLargest);
    double2 high = make_double2(-kLargest, -kLargest);
    int own = 0;        // of the lane's net
    int own_total = 0;  // so far
    __syncwarp();       // the last batch has been read
    for (int at = 0; at < run.total; at += kPinChunk) {
        int p[2], m[2], slot[2];
        double2 v[2];
        unsigned mine[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) p[u] = pinAt(run, at + 32 * u);
#pragma unroll
        for (int u = 0; u < 2; ++u) m[u] = pin_module[p[u]];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            slot[u] = slotOf(module, m[u]);
            v[u] = slot[u] < 0 ? position(p[u], m[u]) : offset(p[u], m[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            mine[u] = __ballot_sync(0xffffffffu, slot[u] >= 0 && at + 32 * u + lane < run.total ? 1 : 0);
            g.point[32 * u + lane] = v[u];
            const int to = own_total + __popc(mine[u] & ((1u << lane) - 1u));
            if ((mine[u] >> lane & 1u) != 0u && to < kOwnPins) {
                g.offset[to] = v[u];
                g.cell[to] = static_cast<uint8_t>(slot[u]);
            }
            own_total += __popc(mine[u]);
        }
        __syncwarp();
        const int stop = min(run.offset + run.degree, at + kPinChunk);
        for (int k = max(run.offset, at); k < stop; ++k) {
            const int i = k - at;
            if ((mine[i >> 5] >> (i & 31) & 1u) != 0u) {
                ++own;
                continue;
            }
            const double2 c = g.point[i];
            low.x = c.x < low.x ? c.x : low.x;  // std::min / std::max
            high.x = high.x < c.x ? c.x : high.x;
            low.y = c.y < low.y ? c.y : low.y;
            high.y = high.y < c.y ? c.y : high.y;
        }
        __syncwarp();
    }
    if (own_total > kOwnPins) return false;
    int end = own;  // inclusive scan
#pragma unroll
    for (int step = 1; step < 32; step <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, end, step);
        if (lane >= step) end += other;
    }
    g.low[lane] = low;
    g.high[lane] = high;
    g.start[lane + 1] = static_cast<uint8_t>(end);
    if (lane == 0) g.start[0] = 0;
    __syncwarp();
    return true;
}

// The half perimeter of gathered net `e` with the window's cells at (cx, cy).
__device__ __forceinline__ double gatheredSpan(const WindowNets& g, int e, const double (&cx)[kWindow],
                                               const double (&cy)[kWindow]) {
    double2 low = g.low[e];
    double2 high = g.high[e];
    for (int k = g.start[e]; k < g.start[e + 1]; ++k) {
        const double2 o = g.offset[k];
        const int slot = g.cell[k];
        double x = cx[0], y = cy[0];
#pragma unroll
        for (int i = 1; i < kWindow; ++i) {
            x = slot == i ? cx[i] : x;
            y = slot == i ? cy[i] : y;
        }
        x += o.x;
        y += o.y;
        low.x = x < low.x ? x : low.x;
        high.x = high.x < x ? x : high.x;
        low.y = y < low.y ? y : low.y;
        high.y = high.y < y ? y : high.y;
    }
    return (high.x - low.x) + (high.y - low.y);
}

// The same pin by pin.
template <typename Position, typename Offset>
__device__ __forceinline__ double walkedSpan(int net, const int* net_pin_start, const int* pin_module,
                                             const int (&module)[kWindow], const double (&cx)[kWindow],
                                             const double (&cy)[kWindow], const Position& position,
                                             const Offset& offset) {
    double2 low = make_double2(kLargest, kLargest);
    double2 high = make_double2(-kLargest, -kLargest);
    for (int p = net_pin_start[net]; p < net_pin_start[net + 1]; ++p) {
        const int m = pin_module[p];
        double2 at;
        if (slotOf(module, m) >= 0) {
            at = offset(p, m);
#pragma unroll
            for (int i = 0; i < kWindow; ++i) {
                if (module[i] == m) at = make_double2(cx[i] + at.x, cy[i] + at.y);
            }
        } else {
            at = position(p, m);
        }
        low.x = at.x < low.x ? at.x : low.x;
        high.x = high.x < at.x ? at.x : high.x;
        low.y = at.y < low.y ? at.y : low.y;
        high.y = high.y < at.y ? at.y : high.y;
    }
    return (high.x - low.x) + (high.y - low.y);
}

// Calls take(net, half perimeter) on lanes below `active` for the window's nets in order, with
// the lane's cells at (cx, cy); gather(base, count, position, offset) fills `g` with up to 32
// of them.  The whole warp calls it.
template <typename Position, typename Offset, typename Take, typename Gather>
__device__ __forceinline__ void forWindowNets(WindowNets& g, const int* nets, int first, int last, int active,
                                              const int* net_pin_start, const int* pin_module,
                                              const int (&module)[kWindow], const double (&cx)[kWindow],
                                              const double (&cy)[kWindow], const Position& position,
                                              const Offset& offset, const Take& take, const Gather& gather) {
    const int lane = threadIdx.x & 31;
    for (int base = first; base < last; base += 32) {
        const int count = min(32, last - base);
        const bool gathered = gather(base, count, position, offset);
        if (lane >= active) continue;
        for (int e = 0; e < count; ++e) {
            const int net = nets[base + e];
            take(net, gathered ? gatheredSpan(g, e, cx, cy)
                               : walkedSpan(net, net_pin_start, pin_module, module, cx, cy, position, offset));
        }
    }
}

// The least and greatest pin coordinates of a net, each with the window that owns the pin's cell
// (-1: none) and the same over the pins of every other window: the box of the pins on other
// cells than a window's, for any window, without a walk over the net.
struct NetExtremes {
    double2 low, high;            // over all pins
    double2 next_low, next_high;  // over the pins of other owners than those below
    int2 low_owner, high_owner;
};

// What a pass on the device knows of its windows' nets beside WindowArrays: entry e of the nets
// has own pins pin[own[e]] .. pin[own[e + 1] - 1].
struct OwnPins {
    const int* own = nullptr;
    const int* pin = nullptr;
    const NetExtremes* extremes = nullptr;
};

// Fills `g` for `count` <= 32 nets of window w from the nets' extremes (gatherNets otherwise).
__device__ __forceinline__ bool gatherFromExtremes(WindowNets& g, const OwnPins& pins, int w, const int* nets, int base,
                                                   int count, const int* pin_module, const int (&module)[kWindow],
                                                   const double2* pin_offset) {
    const int lane = threadIdx.x & 31;
    const int first = pins.own[base];
    const int total = pins.own[base + count] - first;
    if (total > kOwnPins) return false;
    __syncwarp();  // the last batch has been read
    for (int k = lane; k < total; k += 32) {
        const int p = pins.pin[first + k];
        g.offset[k] = pin_offset[p];
        g.cell[k] = static_cast<uint8_t>(slotOf(module, pin_module[p]));
    }
    if (lane < count) {
        const NetExtremes x = pins.extremes[nets[base + lane]];
        g.low[lane] = make_double2(x.low_owner.x == w ? x.next_low.x : x.low.x,
                                   x.low_owner.y == w ? x.next_low.y : x.low.y);
        g.high[lane] = make_double2(x.high_owner.x == w ? x.next_high.x : x.high.x,
                                    x.high_owner.y == w ? x.next_high.y : x.high.y);
        g.start[lane + 1] = static_cast<uint8_t>(pins.own[base + lane + 1] - first);
    }
    if (lane == 0) g.start[0] = 0;
    __syncwarp();
    return true;
}

// kKnown: the nets' extremes and the windows' own pins are known (a pass on the device).
template <bool kKnown>
__global__ void __launch_bounds__(32 * kWindowsPerBlock)
    windowOrdersKernel(const double2* __restrict__ center, const double2* __restrict__ size,
                       const int* __restrict__ pin_module, const double2* __restrict__ pin_offset,
                       const int* __restrict__ net_pin_start, const double* __restrict__ net_weight,
                       WindowArrays windows, int window_count, const uint8_t* __restrict__ kind, double epsilon,
                       int* __restrict__ best_order, uint8_t* __restrict__ decided,
                       double2* __restrict__ moved_center, OwnPins own_pins) {
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * kWindowsPerBlock + static_cast<int>(threadIdx.x >> 5);
    if (w >= window_count) return;  // whole warps leave together
    if (kind != nullptr && kind[w] != kFourCells) {
        if (lane == 0) {
            best_order[w] = 0;
            decided[w] = 0;
        }
        return;
    }
    const int4 m4 = windows.modules[w];
    const int module[kWindow] = {m4.x, m4.y, m4.z, m4.w};

    // The window's cells where this lane puts them (registers only: the cell of
    // each slot is picked by comparisons, never by a computed index).
    double cx[kWindow];
    double cy[kWindow];
#pragma unroll
    for (int i = 0; i < kWindow; ++i) {
        const double2 c = center[module[i]];
        cx[i] = c.x;
        cy[i] = c.y;
    }
    if (lane < kOrders) {
        const unsigned code = orderCode(lane);
        double cursor = windows.start_x[w];
        const double bottom = windows.bottom[w];
        const double spacing = windows.spacing[w];
#pragma unroll
        for (int i = 0; i < kWindow; ++i) {
            const unsigned local = (code >> (4u * static_cast<unsigned>(i))) & 0xFu;
            int placed = module[0];
#pragma unroll
            for (int j = 1; j < kWindow; ++j) placed = local == static_cast<unsigned>(j) ? module[j] : placed;
            const double2 s = size[placed];
            const double x = __dadd_rn(cursor, __dmul_rn(s.x, 0.5));
            const double y = __dadd_rn(bottom, __dmul_rn(s.y, 0.5));
#pragma unroll
            for (int j = 0; j < kWindow; ++j) {
                if (local == static_cast<unsigned>(j)) {
                    cx[j] = x;
                    cy[j] = y;
                }
            }
            cursor = __dadd_rn(cursor, roundedWidthDevice(s.x, spacing));
        }
    }

    __shared__ WindowNets gathered[kWindowsPerBlock];
    double fused = 0.0;
    double plain = 0.0;
    forWindowNets(
        gathered[threadIdx.x >> 5], windows.nets, windows.net_start[w], windows.net_start[w + 1], kCurrentLane + 1,
        net_pin_start, pin_module, module, cx, cy,
        [&](int p, int m) {
            const double2 c = center[m];
            const double2 o = pin_offset[p];
            return make_double2(c.x + o.x, c.y + o.y);
        },
        [&](int p, int) { return pin_offset[p]; },
        [&](int net, double span) {
            const double weight = net_weight[net];
            fused = fma(weight, span, fused);
            plain = __dadd_rn(plain, __dmul_rn(weight, span));
        },
        [&](int base, int count, const auto& position, const auto& offset) {
            WindowNets& g = gathered[threadIdx.x >> 5];
            if constexpr (kKnown) {
                return gatherFromExtremes(g, own_pins, w, windows.nets, base, count, pin_module, module, pin_offset);
            } else {
                return gatherNets(g, windows.nets + base, count, net_pin_start, pin_module, module, position, offset);
            }
        });
    __syncwarp();

    // The smallest fused value, the lowest order on ties, to every lane.
    double best = lane < kOrders ? fused : kLargest;
    int index = lane;
    for (int offset = 16; offset > 0; offset >>= 1) {
        const double other = __shfl_xor_sync(0xffffffffu, best, offset);
        const int other_index = __shfl_xor_sync(0xffffffffu, index, offset);
        if (other < best || (other == best && other_index < index)) {
            best = other;
            index = other_index;
        }
    }
    const double before = __shfl_sync(0xffffffffu, plain, kCurrentLane);
    const double after = __shfl_sync(0xffffffffu, plain, index);
    if (lane == 0) {
        best_order[w] = index;
        decided[w] = index > 0 && index < kOrders && after < before - epsilon ? 1 : 0;
    }
    if (lane == index) {  // where the best order puts the window's cells (applyOrder's arithmetic)
#pragma unroll
        for (int i = 0; i < kWindow; ++i) moved_center[module[i]] = make_double2(cx[i], cy[i]);
    }
}

// transformOffset (PlacementDatabase.cpp:55-68).
__host__ __device__ inline double2 transformed(double2 o, int orientation) {
    switch (orientation) {
        case 1: return make_double2(-o.x, -o.y);
        case 2: return make_double2(-o.y, o.x);
        case 3: return make_double2(o.y, -o.x);
        case 4: return make_double2(-o.x, o.y);
        case 5: return make_double2(o.x, -o.y);
        case 6: return make_double2(o.y, o.x);
        case 7: return make_double2(-o.y, -o.x);
        default: return o;
    }
}

// The host's before / after values of every window (its best order against
// its current placement) on the assumption that each earlier window decided as
// `decided_in` says, and the decisions they give.  A cell of an earlier window
// assumed accepted sits where that window's best order puts it, with the
// orientation of its row; every other cell is where the pass found it.  One
// warp per window: its lanes load the nets' pins (PinRun), each lane then forms
// the two terms of one net (products rounded separately), and the warp adds them
// in net order, as the host does: 490 us in the first round with a net per lane, 276 so
// (51,000 windows of 210,000 cells).
__global__ void __launch_bounds__(32 * kWindowsPerBlock)
    speculativeValuesKernel(const double2* __restrict__ center, const double2* __restrict__ moved_center,
                            const int* __restrict__ owner, const int8_t* __restrict__ moved_orientation,
                            const double2* __restrict__ raw_offset, const double2* __restrict__ pin_offset,
                            const int* __restrict__ pin_module, const int* __restrict__ net_pin_start,
                            const double* __restrict__ net_weight, WindowArrays windows, int window_count,
                            const int* __restrict__ best_order, double epsilon, const uint8_t* __restrict__ decided_in,
                            uint8_t* __restrict__ decided_out, double* __restrict__ value_before,
                            double* __restrict__ value_after, Rounds rounds) {
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * kWindowsPerBlock + static_cast<int>(threadIdx.x >> 5);
    if (w >= window_count) return;  // whole warps leave together
    if (rounds.round > 1 && rounds.changed[rounds.round - 1] == 0) return;  // in and out agree
    const int best = best_order[w];
    if (best <= 0 || best >= kOrders) {
        if (lane == 0) decided_out[w] = 0;
        return;
    }
    const int first = windows.net_start[w];
    const int last = windows.net_start[w + 1];
    if (rounds.stamp != nullptr && settledWindow(rounds, windows.nets, first, last)) {
        if (lane == 0) decided_out[w] = decided_in[w];
        return;
    }
    __shared__ double4 chunk[kWindowsPerBlock][kPinChunk];
    double4* const points = chunk[threadIdx.x >> 5];
    double before = 0.0;
    double after = 0.0;
    for (int base = first; base < last; base += 32) {
        const int count = min(32, last - base);
        const PinRun run = pinRun(windows.nets + base, count, net_pin_start);
        double min_b = kLargest, max_b = -kLargest, min_by = kLargest, max_by = -kLargest;
        double min_a = kLargest, max_a = -kLargest, min_ay = kLargest, max_ay = -kLargest;
        for (int at = 0; at < run.total; at += kPinChunk) {
            int p[2], m[2], own[2];
            double2 now_c[2], offset[2];
            bool moved[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) p[u] = pinAt(run, at + 32 * u);
#pragma unroll
            for (int u = 0; u < 2; ++u) m[u] = pin_module[p[u]];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                now_c[u] = center[m[u]];
                own[u] = owner[m[u]];
                offset[u] = pin_offset[p[u]];
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) moved[u] = own[u] >= 0 && own[u] < w && decided_in[max(own[u], 0)] != 0;
            __syncwarp();  // the last chunk has been read
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                double2 then_c = now_c[u];  // with this window's best order applied
                if (own[u] == w) {
                    then_c = moved_center[m[u]];  // its orientation changes only once accepted
                } else if (moved[u]) {
                    now_c[u] = moved_center[m[u]];
                    then_c = now_c[u];
                    offset[u] = transformed(raw_offset[p[u]], moved_orientation[m[u]]);
                }
                points[32 * u + lane] =
                    make_double4(now_c[u].x + offset[u].x, now_c[u].y + offset[u].y, then_c.x + offset[u].x,
                                 then_c.y + offset[u].y);
            }
            __syncwarp();
            const int stop = min(run.offset + run.degree, at + kPinChunk);
            for (int k = max(run.offset, at); k < stop; ++k) {
                const double4 v = points[k - at];
                min_b = v.x < min_b ? v.x : min_b;
                max_b = max_b < v.x ? v.x : max_b;
                min_by = v.y < min_by ? v.y : min_by;
                max_by = max_by < v.y ? v.y : max_by;
                min_a = v.z < min_a ? v.z : min_a;
                max_a = max_a < v.z ? v.z : max_a;
                min_ay = v.w < min_ay ? v.w : min_ay;
                max_ay = max_ay < v.w ? v.w : max_ay;
            }
        }
        double term_before = 0.0;
        double term_after = 0.0;
        if (lane < count) {
            const double weight = net_weight[windows.nets[base + lane]];
            term_before = __dmul_rn(weight, (max_b - min_b) + (max_by - min_by));
            term_after = __dmul_rn(weight, (max_a - min_a) + (max_ay - min_ay));
        }
        for (int j = 0; j < count; ++j) {
            before = __dadd_rn(before, __shfl_sync(0xffffffffu, term_before, j));
            after = __dadd_rn(after, __shfl_sync(0xffffffffu, term_after, j));
        }
    }
    const uint8_t decision = after < before - epsilon ? 1 : 0;
    if (rounds.stamp != nullptr) {
        if (decision != decided_in[w]) stampWindow(rounds, windows.nets, first, last);
    } else if (lane == 0) {
        value_before[w] = before;
        value_after[w] = after;
    }
    if (lane == 0) decided_out[w] = decision;
}

// The windows the reference keeps on the host (segment ends of two or three
// cells), those with nets to evaluate, in the reference's order.
struct TailArrays {
    const int4* modules;  // unused slots -1
    const int* count;
    const double* start_x;
    const double* bottom;
    const double* spacing;
    const int* net_start;
    const int* nets;
};

// Where each tail window's assumed order (-1: none) puts its cells.
__global__ void __launch_bounds__(256)
    tailPlacementKernel(TailArrays tail, int tail_count, const double2* __restrict__ size,
                        const int8_t* __restrict__ assumed, double2* __restrict__ moved_center, Rounds rounds) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tail_count || assumed[t] < 0) return;
    if (rounds.round > 1 && rounds.changed[rounds.round - 1] == 0) return;
    const int n = tail.count[t];
    const int4 m4 = tail.modules[t];
    const int module[kWindow] = {m4.x, m4.y, m4.z, m4.w};
    const unsigned code = orderCode(assumed[t], n);
    double cursor = tail.start_x[t];
    for (int i = 0; i < n; ++i) {
        const unsigned local = (code >> (4u * static_cast<unsigned>(i))) & 0xFu;
        int placed = module[0];
#pragma unroll
        for (int j = 1; j < kWindow; ++j) placed = local == static_cast<unsigned>(j) ? module[j] : placed;
        const double2 s = size[placed];
        moved_center[placed] = make_double2(__dadd_rn(cursor, __dmul_rn(s.x, 0.5)),
                                            __dadd_rn(tail.bottom[t], __dmul_rn(s.y, 0.5)));
        cursor = __dadd_rn(cursor, roundedWidthDevice(s.x, tail.spacing[t]));
    }
}

// optimizeCpuWindow (CudaDetailedPlacementBackend.cu:328-354) for every tail
// window on the assumption that each earlier tail window took the order
// `assumed_in` says: every order in lexicographic order, each taken when it
// beats the best so far by more than epsilon, from the placement as it is.
// Writes the order taken, or -1.  A cell of an earlier tail window assumed
// reordered sits where that order puts it, with its row's orientation; every
// other cell is where the four-cell windows left it.  One warp per window:
// lane k < n! evaluates order k, lane n! the placement as it is, and every lane
// then runs the same selection over the lanes' values in order.
__global__ void __launch_bounds__(32 * kWindowsPerBlock)
    tailOrdersKernel(const double2* __restrict__ center, const int8_t* __restrict__ orientation,
                     const double2* __restrict__ moved_center, const int* __restrict__ owner, int tail_base,
                     const int8_t* __restrict__ moved_orientation, const double2* __restrict__ raw_offset,
                     const double2* __restrict__ size, const int* __restrict__ pin_module,
                     const int* __restrict__ net_pin_start, const double* __restrict__ net_weight, TailArrays tail,
                     int tail_count, const uint8_t* __restrict__ kind, double epsilon,
                     const int8_t* __restrict__ assumed_in, int8_t* __restrict__ order_out, Rounds rounds) {
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * kWindowsPerBlock + static_cast<int>(threadIdx.x >> 5);
    if (t >= tail_count) return;  // whole warps leave together
    if (rounds.round > 1 && rounds.changed[rounds.round - 1] == 0) return;  // in and out agree
    if (kind != nullptr && kind[t] != kTail) {
        if (lane == 0) order_out[t] = -1;
        return;
    }
    const int first = tail.net_start[t];
    const int last = tail.net_start[t + 1];
    if (rounds.stamp != nullptr && settledWindow(rounds, tail.nets, first, last)) {
        if (lane == 0) order_out[t] = assumed_in[t];
        return;
    }
    const int n = tail.count[t];
    const int orders = factorialOf(n);
    const int4 m4 = tail.modules[t];
    const int module[kWindow] = {m4.x, m4.y, m4.z, m4.w};
    double cx[kWindow];
    double cy[kWindow];
#pragma unroll
    for (int i = 0; i < kWindow; ++i) {
        const double2 c = module[i] >= 0 ? center[module[i]] : make_double2(0.0, 0.0);
        cx[i] = c.x;
        cy[i] = c.y;
    }
    if (lane < orders) {
        const unsigned code = orderCode(lane, n);
        double cursor = tail.start_x[t];
        for (int i = 0; i < n; ++i) {
            const unsigned local = (code >> (4u * static_cast<unsigned>(i))) & 0xFu;
            int placed = module[0];
#pragma unroll
            for (int j = 1; j < kWindow; ++j) placed = local == static_cast<unsigned>(j) ? module[j] : placed;
            const double2 s = size[placed];
            const double x = __dadd_rn(cursor, __dmul_rn(s.x, 0.5));
            const double y = __dadd_rn(tail.bottom[t], __dmul_rn(s.y, 0.5));
#pragma unroll
            for (int j = 0; j < kWindow; ++j) {
                if (local == static_cast<unsigned>(j)) {
                    cx[j] = x;
                    cy[j] = y;
                }
            }
            cursor = __dadd_rn(cursor, roundedWidthDevice(s.x, tail.spacing[t]));
        }
    }
    // The window's weighted HPWL with its own cells at (cx, cy).
    __shared__ WindowNets gathered[kWindowsPerBlock];
    double mine = 0.0;
    forWindowNets(
        gathered[threadIdx.x >> 5], tail.nets, first, last, orders + 1, net_pin_start, pin_module, module, cx, cy,
        [&](int p, int m) {
            double2 c = center[m];
            int turn = orientation[m];
            const int j = owner[m] - tail_base;
            if (j >= 0 && j < t && assumed_in[j] >= 0) {
                c = moved_center[m];
                turn = moved_orientation[m];
            }
            const double2 o = transformed(raw_offset[p], turn);
            return make_double2(c.x + o.x, c.y + o.y);
        },
        [&](int p, int m) { return transformed(raw_offset[p], orientation[m]); },
        [&](int net, double span) { mine = __dadd_rn(mine, __dmul_rn(net_weight[net], span)); },
        [&](int base, int count, const auto& position, const auto& offset) {
            return gatherNets(gathered[threadIdx.x >> 5], tail.nets + base, count, net_pin_start, pin_module, module,
                              position, offset);
        });
    __syncwarp();
    double best = __shfl_sync(0xffffffffu, mine, orders);
    int taken = -1;
    for (int k = 0; k < orders; ++k) {
        const double v = __shfl_sync(0xffffffffu, mine, k);
        if (v < best - epsilon) {
            best = v;
            taken = k;
        }
    }
    if (rounds.stamp != nullptr && taken != assumed_in[t]) stampWindow(rounds, tail.nets, first, last);
    if (lane == 0) order_out[t] = static_cast<int8_t>(taken);
}

// ---- host ---------------------------------------------------------------------------------

// transformOffset (PlacementDatabase.cpp:55-68).
inline void transform(double x, double y, int orientation, double& ox, double& oy) {
    switch (orientation) {
        case 1: ox = -x; oy = -y; return;
        case 2: ox = -y; oy = x; return;
        case 3: ox = y; oy = -x; return;
        case 4: ox = -x; oy = y; return;
        case 5: ox = x; oy = -y; return;
        case 6: ox = y; oy = x; return;
        case 7: ox = -y; oy = -x; return;
        default: ox = x; oy = y; return;
    }
}

// alignUp(width, 0, spacing) (CudaDetailedPlacementBackend.cu:229-236).
inline double roundedWidth(double width, double spacing) {
    if (spacing <= kEpsilon) return width;
    return 0.0 + std::ceil((width - 0.0 - kEpsilon) / spacing) * spacing;
}

template <typename T>
class DeviceArray {
public:
    DeviceArray() = default;
    DeviceArray(const DeviceArray&) = delete;
    DeviceArray& operator=(const DeviceArray&) = delete;
    ~DeviceArray() {
        if (data_ != nullptr) cudaFree(data_);
    }
    void allocate(std::size_t count, uint64_t& reserved, uint64_t limit, const char* what) {
        const uint64_t bytes = static_cast<uint64_t>(std::max<std::size_t>(count, 1)) * sizeof(T);
        if (bytes > limit - std::min(limit, reserved)) {
            fail(MPGP_ERR_BUDGET, std::string("CUDA detailed-placement budget exceeded while reserving ") + what + ".");
        }
        checkCuda(cudaMalloc(reinterpret_cast<void**>(&data_), bytes), what);
        reserved += bytes;
    }
    void upload(const std::vector<T>& values, cudaStream_t stream) {
        if (!values.empty()) {
            checkCuda(cudaMemcpyAsync(data_, values.data(), values.size() * sizeof(T), cudaMemcpyHostToDevice, stream),
                      "detailed-placement upload");
        }
    }
    void download(std::vector<T>& values, cudaStream_t stream) const {
        if (!values.empty()) {
            checkCuda(cudaMemcpyAsync(values.data(), data_, values.size() * sizeof(T), cudaMemcpyDeviceToHost, stream),
                      "detailed-placement download");
        }
    }
    [[nodiscard]] T* get() const { return data_; }

private:
    T* data_ = nullptr;
};

class Stream {
public:
    Stream() { checkCuda(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate"); }
    ~Stream() { cudaStreamDestroy(stream_); }
    Stream(const Stream&) = delete;
    Stream& operator=(const Stream&) = delete;
    [[nodiscard]] cudaStream_t get() const { return stream_; }

private:
    cudaStream_t stream_ = nullptr;
};

class Event {
public:
    Event() { checkCuda(cudaEventCreateWithFlags(&event_, cudaEventDisableTiming), "cudaEventCreate"); }
    ~Event() { cudaEventDestroy(event_); }
    Event(const Event&) = delete;
    Event& operator=(const Event&) = delete;
    [[nodiscard]] cudaEvent_t get() const { return event_; }

private:
    cudaEvent_t event_ = nullptr;
};

// The placement state the passes change, with the design's fixed data.
struct Placement {
    const mpgp_design& d;
    std::vector<double> cx, cy;
    std::vector<int32_t> orientation;
    std::vector<int32_t> pin_net;
    std::vector<int64_t> module_pin_start;  // module -> its pins, in pin order
    std::vector<int32_t> module_pins;

    explicit Placement(const mpgp_design& design) : d(design) {
        const std::size_t m = static_cast<std::size_t>(d.module_count);
        cx.assign(d.module_x, d.module_x + m);
        cy.assign(d.module_y, d.module_y + m);
        orientation.assign(m, 0);
        if (d.module_orientation != nullptr) orientation.assign(d.module_orientation, d.module_orientation + m);
        pin_net.resize(static_cast<std::size_t>(d.pin_count));
        for (int32_t n = 0; n < d.net_count; ++n) {
            for (int64_t p = d.net_pin_start[n]; p < d.net_pin_start[n + 1]; ++p) pin_net[p] = n;
        }
        module_pin_start.assign(m + 1, 0);
        for (int64_t p = 0; p < d.pin_count; ++p) ++module_pin_start[d.pin_module[p] + 1];
        for (std::size_t k = 0; k < m; ++k) module_pin_start[k + 1] += module_pin_start[k];
        module_pins.resize(static_cast<std::size_t>(d.pin_count));
        std::vector<int64_t> fill(module_pin_start.begin(), module_pin_start.end() - 1);
        for (int64_t p = 0; p < d.pin_count; ++p) module_pins[fill[d.pin_module[p]]++] = static_cast<int32_t>(p);
    }

    [[nodiscard]] double lowerLeftX(int m) const { return cx[m] - d.module_width[m] * 0.5; }
    [[nodiscard]] double lowerLeftY(int m) const { return cy[m] - d.module_height[m] * 0.5; }

    // localHpwl (CudaDetailedPlacementBackend.cu:282-302) with the window's cells
    // at (wx, wy).
    double windowHpwl(const int32_t* modules, int count, const int32_t* nets, int net_count, const double* wx,
                      const double* wy) const {
        double result = 0.0;
        for (int e = 0; e < net_count; ++e) {
            const int32_t net = nets[e];
            double min_x = std::numeric_limits<double>::infinity();
            double max_x = -std::numeric_limits<double>::infinity();
            double min_y = std::numeric_limits<double>::infinity();
            double max_y = -std::numeric_limits<double>::infinity();
            for (int64_t p = d.net_pin_start[net]; p < d.net_pin_start[net + 1]; ++p) {
                const int32_t m = d.pin_module[p];
                double x = cx[m];
                double y = cy[m];
                for (int i = 0; i < count; ++i) {
                    if (modules[i] == m) {
                        x = wx[i];
                        y = wy[i];
                        break;
                    }
                }
                double ox = 0.0;
                double oy = 0.0;
                transform(d.pin_offset_x[p], d.pin_offset_y[p], orientation[m], ox, oy);
                x = x + ox;
                y = y + oy;
                min_x = std::min(min_x, x);
                max_x = std::max(max_x, x);
                min_y = std::min(min_y, y);
                max_y = std::max(max_y, y);
            }
            result += d.net_weight[net] * ((max_x - min_x) + (max_y - min_y));
        }
        return result;
    }

    // centersForOrder (:304-315).
    void centersForOrder(const int32_t* modules, const int* order, int count, double bottom, double spacing,
                         double* wx, double* wy) const {
        double cursor = lowerLeftX(modules[0]);
        for (int i = 0; i < count; ++i) {
            const int local = order[i];
            const int32_t m = modules[local];
            wx[local] = cursor + d.module_width[m] * 0.5;
            wy[local] = bottom + d.module_height[m] * 0.5;
            cursor += roundedWidth(d.module_width[m], spacing);
        }
    }

    // applyOrder (:317-326): setLowerLeft, then the row's orientation when known.
    void applyOrder(const int32_t* modules, const int* order, int count, double bottom, double spacing,
                    int row_orientation) {
        double cursor = lowerLeftX(modules[0]);
        for (int i = 0; i < count; ++i) {
            const int32_t m = modules[order[i]];
            cx[m] = cursor + d.module_width[m] * 0.5;
            cy[m] = bottom + d.module_height[m] * 0.5;
            if (row_orientation != kOrientationUnknown) orientation[m] = row_orientation;
            cursor += roundedWidth(d.module_width[m], spacing);
        }
    }

    // calculateHpwl (Metrics.cpp:128-147): the nets' terms on several threads,
    // summed in net order.
    [[nodiscard]] double hpwl(const Workers& workers) const {
        std::vector<double> term(static_cast<std::size_t>(d.net_count), 0.0);
        workers.blocks(term.size(), 8192, [&](std::size_t b, std::size_t e) {
            for (std::size_t n = b; n < e; ++n) term[n] = netTerm(static_cast<int32_t>(n));
        });
        double result = 0.0;
        for (int32_t n = 0; n < d.net_count; ++n) {
            if (d.net_pin_start[n + 1] - d.net_pin_start[n] >= 2) result += term[n];
        }
        return result;
    }

    // One net's weighted HPWL at the current placement.
    [[nodiscard]] double netTerm(int32_t n) const {
        double min_x = std::numeric_limits<double>::infinity();
        double max_x = -std::numeric_limits<double>::infinity();
        double min_y = std::numeric_limits<double>::infinity();
        double max_y = -std::numeric_limits<double>::infinity();
        for (int64_t p = d.net_pin_start[n]; p < d.net_pin_start[n + 1]; ++p) {
            const int32_t m = d.pin_module[p];
            double ox = 0.0;
            double oy = 0.0;
            transform(d.pin_offset_x[p], d.pin_offset_y[p], orientation[m], ox, oy);
            const double x = cx[m] + ox;
            const double y = cy[m] + oy;
            min_x = std::min(min_x, x);
            max_x = std::max(max_x, x);
            min_y = std::min(min_y, y);
            max_y = std::max(max_y, y);
        }
        return d.net_weight[n] * ((max_x - min_x) + (max_y - min_y));
    }
};

// A window: up to four consecutive cells of a segment and the nets they touch.
struct Windows {
    std::vector<int32_t> row;
    std::vector<int32_t> count;
    std::vector<int32_t> modules;  // kWindow per window (unused slots -1)
    std::vector<int64_t> net_start{0};
    std::vector<int32_t> nets;     // sorted, unique per window
    std::vector<uint8_t> device;   // evaluated on the device (gpu_eligible)

    void clear() {
        row.clear();
        count.clear();
        modules.clear();
        net_start.assign(1, 0);
        nets.clear();
        device.clear();
    }
};

// buildRowSegments (:238-274) and makeWindow (:276-293) for one pass: the
// windows in the reference's order, whichever list they go to.  Rows are
// independent: each sorts its cells (in module order before the sort, as the
// reference collects them, so std::sort leaves ties as the reference's does)
// and cuts its segments and windows on a thread of its own.
void buildWindows(const Placement& s, const std::vector<uint8_t>& standard, int phase, uint64_t maximum_net_degree,
                  const Workers& workers, Windows& out) {
    const mpgp_design& d = s.d;
    out.clear();
    if (d.row_count == 0) return;
    std::vector<std::size_t> sorted_rows(static_cast<std::size_t>(d.row_count));
    std::iota(sorted_rows.begin(), sorted_rows.end(), 0U);
    std::sort(sorted_rows.begin(), sorted_rows.end(),
              [&](std::size_t a, std::size_t b) { return d.row_bottom[a] < d.row_bottom[b]; });
    const auto centre = [&](std::size_t r) { return d.row_bottom[r] + d.row_height[r] * 0.5; };
    const auto nearestRow = [&](double coordinate) {
        const auto it = std::lower_bound(sorted_rows.begin(), sorted_rows.end(), coordinate,
                                         [&](std::size_t r, double value) { return centre(r) < value; });
        if (it == sorted_rows.begin()) return *it;
        if (it == sorted_rows.end()) return sorted_rows.back();
        const std::size_t right = *it;
        const std::size_t left = *(it - 1);
        return std::abs(centre(left) - coordinate) <= std::abs(centre(right) - coordinate) ? left : right;
    };
    constexpr double kSegmentEpsilon = 1e-6;
    const std::size_t modules = static_cast<std::size_t>(d.module_count);
    const std::size_t rows = static_cast<std::size_t>(d.row_count);
    std::vector<int32_t> row_of(modules, -1);
    workers.blocks(modules, 16384, [&](std::size_t b, std::size_t e) {
        for (std::size_t m = b; m < e; ++m) {
            if (standard[m] == 0) continue;
            const std::size_t r = nearestRow(s.cy[m]);
            if (std::abs(s.lowerLeftY(static_cast<int>(m)) - d.row_bottom[r]) <= kSegmentEpsilon) {
                row_of[m] = static_cast<int32_t>(r);
            }
        }
    });
    std::vector<std::size_t> row_start(rows + 1, 0);
    for (const int32_t r : row_of) {
        if (r >= 0) ++row_start[static_cast<std::size_t>(r) + 1];
    }
    for (std::size_t r = 0; r < rows; ++r) row_start[r + 1] += row_start[r];
    std::vector<int32_t> cells(row_start[rows]);
    {
        std::vector<std::size_t> fill(row_start.begin(), row_start.end() - 1);
        for (std::size_t m = 0; m < modules; ++m) {
            if (row_of[m] >= 0) cells[fill[static_cast<std::size_t>(row_of[m])]++] = static_cast<int32_t>(m);
        }
    }

    struct RowWindows {
        std::vector<int32_t> count, modules, nets;
        std::vector<int64_t> net_end;
        std::vector<uint8_t> device;
    };
    std::vector<RowWindows> per_row(rows);
    workers.run(rows, [&](std::size_t r) {
        if (row_start[r + 1] - row_start[r] < 2U) return;
        std::vector<int32_t> row_cells(cells.begin() + static_cast<std::ptrdiff_t>(row_start[r]),
                                       cells.begin() + static_cast<std::ptrdiff_t>(row_start[r + 1]));
        std::sort(row_cells.begin(), row_cells.end(),
                  [&](int32_t a, int32_t b) { return s.lowerLeftX(a) < s.lowerLeftX(b); });
        RowWindows& mine = per_row[r];
        std::vector<int32_t> window_nets;
        const auto emit = [&](std::size_t first, std::size_t size) {
            if (size < 2U) return;
            for (std::size_t start = static_cast<std::size_t>(phase); start + 1U < size; start += kWindow) {
                const std::size_t count = std::min<std::size_t>(kWindow, size - start);
                if (count < 2U) break;
                window_nets.clear();
                for (std::size_t i = 0; i < count; ++i) {
                    const int32_t m = row_cells[first + start + i];
                    for (int64_t k = s.module_pin_start[m]; k < s.module_pin_start[m + 1]; ++k) {
                        window_nets.push_back(s.pin_net[s.module_pins[k]]);
                    }
                }
                std::sort(window_nets.begin(), window_nets.end());
                window_nets.erase(std::unique(window_nets.begin(), window_nets.end()), window_nets.end());
                bool device = count == static_cast<std::size_t>(kWindow) && !window_nets.empty();
                for (const int32_t n : window_nets) {
                    if (static_cast<uint64_t>(d.net_pin_start[n + 1] - d.net_pin_start[n]) > maximum_net_degree) {
                        device = false;
                    }
                }
                mine.count.push_back(static_cast<int32_t>(count));
                for (std::size_t i = 0; i < kWindow; ++i) {
                    mine.modules.push_back(i < count ? row_cells[first + start + i] : -1);
                }
                mine.nets.insert(mine.nets.end(), window_nets.begin(), window_nets.end());
                mine.net_end.push_back(static_cast<int64_t>(mine.nets.size()));
                mine.device.push_back(device ? 1 : 0);
            }
        };
        std::size_t first = 0;
        for (std::size_t i = 1; i < row_cells.size(); ++i) {
            const int32_t previous = row_cells[i - 1];
            const double expected =
                s.lowerLeftX(previous) + roundedWidth(d.module_width[previous], d.row_site_spacing[r]);
            if (std::abs(s.lowerLeftX(row_cells[i]) - expected) > kSegmentEpsilon) {
                emit(first, i - first);
                first = i;
            }
        }
        emit(first, row_cells.size() - first);
    });
    for (std::size_t r = 0; r < rows; ++r) {
        const RowWindows& mine = per_row[r];
        const int64_t base = static_cast<int64_t>(out.nets.size());
        out.row.insert(out.row.end(), mine.count.size(), static_cast<int32_t>(r));
        out.count.insert(out.count.end(), mine.count.begin(), mine.count.end());
        out.modules.insert(out.modules.end(), mine.modules.begin(), mine.modules.end());
        out.nets.insert(out.nets.end(), mine.nets.begin(), mine.nets.end());
        for (const int64_t end : mine.net_end) out.net_start.push_back(base + end);
        out.device.insert(out.device.end(), mine.device.begin(), mine.device.end());
    }
}

// ---- the whole pass on the device ------------------------------------------------------------
//
// From the host's lists above, a pass over 210,000 cells spent 23 ms around 2.4 ms of kernels:
// rows, segments, windows and their nets (7 ms), the lists of each kind and the owners (4.5),
// uploads (3.3), the walk over the decisions (4) and the tails (1.6); and a call 30 ms more for
// the pin lists (10), 30 allocations (5) and the uploads of the design (6).  Here the design goes
// up once and the passes are kernels: the cells are sorted by row and x, cut into segments and
// windows by scans, and the windows' nets come from one stable sort of the pins by window.  The
// decisions are re-evaluated until a round changes none: the k-th window's decision no longer
// changes after k rounds (it rests on earlier windows only), so the rounds end, and the only
// decisions that reproduce themselves are the ones the walk takes one after another.  After the
// first round only windows with a net of a window that changed are evaluated.  Two passes over
// 210,000 cells: 76.6 ms, and 5.8 so, of which the uploads take 1.5 and the kernels 2.5.

constexpr int kMaxRounds = 1000;
constexpr int kRoundsPerCheck = 4;  // launched before the host looks whether the last one changed anything
constexpr double kSegmentEpsilon = 1e-6;

int threadBlocks(std::size_t count) { return static_cast<int>((std::max<std::size_t>(count, 1) + kThreads - 1) / kThreads); }

// The rows on the device: in bottom order for the search, and by index.
struct DeviceRows {
    int count = 0;
    const double* centre = nullptr;  // sorted
    const int* index = nullptr;      // sorted -> row
    const double* bottom = nullptr;
    const double* spacing = nullptr;
    const int* turn = nullptr;       // orientation a moved cell takes, kOrientationUnknown: its own
};

// Counts of a pass that the host needs.
struct PassCounts {
    int windows = 0;
    int ties = 0;  // cells at the same x of a row: the host sort's order of them is not ours to know
    int four = 0;
    int tails = 0;
    unsigned long long permutations = 0;
    unsigned long long accepted = 0;
};

__device__ __forceinline__ double lowerLeft(double centre, double extent) {
    return __dsub_rn(centre, __dmul_rn(extent, 0.5));
}

// The caller's arrays on the device.
struct RawDesign {
    int modules = 0, nets = 0, pins = 0;
    const double* x = nullptr;
    const double* y = nullptr;
    const double* width = nullptr;
    const double* height = nullptr;
    const int* flags = nullptr;
    const int* orientation = nullptr;  // null: all N
    const long long* net_start = nullptr;
    const double* net_weight = nullptr;
    const int* pin_module = nullptr;
    const double* offset_x = nullptr;
    const double* offset_y = nullptr;
};

// Kernels that walk the nets give each eight lanes, and a net of more than kLongNet pins a block
// of kLongThreads in a launch of its own: eight lanes follow one chain of dependent loads after
// another.  Two passes over 210,000 cells with a net of 420,000 pins beside the others took 95 ms
// with eight lanes (72 from the host's lists) and take 5-6, with one of 210,000 pins 15 and 4-4.6.
constexpr int kLongNet = 512;
constexpr int kLongThreads = 1024;

// Sets flags[0] where validateDesign, or the check of the orientations, would refuse an entry, and
// lists the long nets (flags[1] of them; their list has room for one per kLongNet pins).
__global__ void __launch_bounds__(kThreads) checkDesignKernel(RawDesign d, int* flags, int* long_nets) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool good = true;
    if (i < d.nets) {
        const long long degree = d.net_start[i + 1] - d.net_start[i];
        good = degree >= 0 && isfinite(d.net_weight[i]);
        if (degree > kLongNet) {
            const int at = atomicAdd(flags + 1, 1);
            if (at <= d.pins / kLongNet) long_nets[at] = i;  // more only of offsets that are refused
        }
    }
    if (i < d.pins) {
        const int m = d.pin_module[i];
        good = good && m >= 0 && m < d.modules && isfinite(d.offset_x[i]) && isfinite(d.offset_y[i]);
    }
    if (i < d.modules) {
        const double w = d.width[i], h = d.height[i];
        good = good && w >= 0.0 && h >= 0.0 && isfinite(w) && isfinite(h) && isfinite(d.x[i]) && isfinite(d.y[i]);
        if (d.orientation != nullptr) good = good && d.orientation[i] >= 0 && d.orientation[i] <= kOrientationUnknown;
    }
    if (!good) flags[0] = 1;
}

// A thread's part of a net: pins first + lane, first + lane + lanes, ... below last.  In the form
// for long nets a block's, otherwise eight lanes', whose long nets are empty here.
struct NetShare {
    int net = -1;  // none: nothing to write either
    int first = 0, last = 0;
    int lane = 0;
};
template <bool kLong>
constexpr int kNetLanes = kLong ? kLongThreads : 8;
template <bool kLong, class Start>
__device__ __forceinline__ NetShare netShare(int count, const Start* start, const int* long_nets) {
    NetShare s;
    const int n = kLong ? long_nets[blockIdx.x] : static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 3);
    s.lane = static_cast<int>(kLong ? threadIdx.x : threadIdx.x & 7);
    if (n >= count) return s;
    s.first = static_cast<int>(start[n]);
    s.last = static_cast<int>(start[n + 1]);
    if (!kLong && s.last - s.first > kLongNet) {
        s.last = s.first;
    } else {
        s.net = n;
    }
    return s;
}

// Joins the parts of the net's threads; the first lane has the whole.
template <bool kLong, class T>
__device__ __forceinline__ void joinNet(T& v) {
#pragma unroll
    for (int lanes = kLong ? 16 : 4; lanes > 0; lanes >>= 1) v.joinLane(lanes);
    if constexpr (kLong) {
        static_assert(kLongThreads == 32 * 32, "a warp joins the warps' parts");
        __shared__ __align__(16) unsigned char parts[32 * sizeof(T)];
        T* const of_warp = reinterpret_cast<T*>(parts);
        const int lane = threadIdx.x & 31;
        if (lane == 0) of_warp[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x < 32) {
            v = of_warp[lane];
#pragma unroll
            for (int lanes = 16; lanes > 0; lanes >>= 1) v.joinLane(lanes);
        }
    }
}

// Calls launch(whether the form for long nets, blocks, threads) for the nets of at most kLongNet pins and,
// if there are any, for the longer ones.
template <class Launch>
void launchNets(int nets, int long_nets, const Launch& launch) {
    launch(std::false_type{}, threadBlocks(8 * (static_cast<std::size_t>(nets) + 1)), kThreads);
    if (long_nets > 0) launch(std::true_type{}, long_nets, kLongThreads);
}

// deriveDesign's fixed and macro rules: a standard cell is neither.
__global__ void __launch_bounds__(kThreads) detailedModulesKernel(RawDesign d, double nominal_row_height, double2* center,
                                                                  double2* size, int8_t* turn, uint8_t* standard) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= d.modules) return;
    const double height = d.height[m];
    center[m] = make_double2(d.x[m], d.y[m]);
    size[m] = make_double2(d.width[m], height);
    turn[m] = d.orientation != nullptr ? static_cast<int8_t>(d.orientation[m]) : 0;
    const bool terminal = (d.flags[m] & MPGP_MODULE_TERMINAL) != 0;
    const bool fixed = terminal || (d.flags[m] & MPGP_MODULE_FIXED) != 0;
    const bool macro = !terminal && nominal_row_height > kEpsilon && fabs(height - nominal_row_height) > kEpsilon;
    standard[m] = !fixed && !macro ? 1 : 0;
}

template <bool kLong>
__global__ void __launch_bounds__(kNetLanes<kLong> * (kLong ? 1 : kThreads / 8))
    detailedNetsKernel(int count, const long long* start, const int* long_nets, int* start32, int* pin_net,
                       int* pin_index) {
    const NetShare s = netShare<kLong>(count, start, long_nets);
    if constexpr (!kLong) {
        const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
        if (s.lane == 0 && n <= count) start32[n] = static_cast<int>(start[n]);
    }
    for (int p = s.first + s.lane; p < s.last; p += kNetLanes<kLong>) {
        pin_net[p] = s.net;
        pin_index[p] = p;
    }
}

__global__ void __launch_bounds__(kThreads) rawOffsetsKernel(int count, const double* x, const double* y, double2* raw) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < count) raw[p] = make_double2(x[p], y[p]);
}

__global__ void __launch_bounds__(kThreads) turnedOffsetsKernel(int count, const double2* raw, const int* pin_module,
                                                                const int8_t* turn, double2* offset) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < count) offset[p] = transformed(raw[p], turn[pin_module[p]]);
}

// The least value of a set of pins, its owner and the least value of other owners' pins.  (An
// unowned pin may count as the others' owner too: no window asks without it.)
struct LeastTwo {
    double first = kLargest;
    double next = kLargest;
    int owner = -2;
    __device__ __forceinline__ void join(double f, double n, int o) {
        if (o == owner) {
            next = n < next ? n : next;
            first = f < first ? f : first;
        } else if (f < first) {
            next = first < n ? first : n;
            first = f;
            owner = o;
        } else {
            next = f < next ? f : next;
        }
    }
    __device__ __forceinline__ void joinLane(int lanes) {
        const double f = __shfl_xor_sync(0xffffffffu, first, lanes);
        const double n = __shfl_xor_sync(0xffffffffu, next, lanes);
        join(f, n, __shfl_xor_sync(0xffffffffu, owner, lanes));
    }
};

// The greatest values as the least negated ones.  Nets of more than `longest` pins are left out: a
// window with one of them is not evaluated.
struct LeastFour {
    LeastTwo low_x, low_y, high_x, high_y;
    __device__ __forceinline__ void joinLane(int lanes) {
        low_x.joinLane(lanes);
        low_y.joinLane(lanes);
        high_x.joinLane(lanes);
        high_y.joinLane(lanes);
    }
};
template <bool kLong>
__global__ void __launch_bounds__(kNetLanes<kLong> * (kLong ? 1 : kThreads / 8))
    netExtremesKernel(int count, const int* start, const int* long_nets, int longest, const int* pin_module,
                      const double2* offset, const double2* center, const int* owner, NetExtremes* out) {
    const NetShare s = netShare<kLong>(count, start, long_nets);
    if (kLong && s.last - s.first > longest) return;  // the whole block
    const int last = s.last - s.first > longest ? s.first : s.last;
    LeastFour v;
#pragma unroll (kLong ? 4 : 1)
    for (int p = s.first + s.lane; p < last; p += kNetLanes<kLong>) {
        const int m = pin_module[p];
        const double2 c = center[m];
        const double2 o = offset[p];
        const int w = owner[m];
        const double x = c.x + o.x;
        const double y = c.y + o.y;
        v.low_x.join(x, kLargest, w);
        v.low_y.join(y, kLargest, w);
        v.high_x.join(-x, kLargest, w);
        v.high_y.join(-y, kLargest, w);
    }
    joinNet<kLong>(v);
    if (s.net >= 0 && s.lane == 0) {
        out[s.net] = NetExtremes{make_double2(v.low_x.first, v.low_y.first),
                                 make_double2(-v.high_x.first, -v.high_y.first),
                                 make_double2(v.low_x.next, v.low_y.next),
                                 make_double2(-v.high_x.next, -v.high_y.next),
                                 make_int2(v.low_x.owner, v.low_y.owner),
                                 make_int2(v.high_x.owner, v.high_y.owner)};
    }
}

// One net's weighted HPWL (Placement::netTerm; zero below two pins).
struct NetBox {
    double min_x = INFINITY, max_x = -INFINITY, min_y = INFINITY, max_y = -INFINITY;
    __device__ __forceinline__ void joinLane(int lanes) {
        min_x = fmin(min_x, __shfl_xor_sync(0xffffffffu, min_x, lanes));
        max_x = fmax(max_x, __shfl_xor_sync(0xffffffffu, max_x, lanes));
        min_y = fmin(min_y, __shfl_xor_sync(0xffffffffu, min_y, lanes));
        max_y = fmax(max_y, __shfl_xor_sync(0xffffffffu, max_y, lanes));
    }
};
template <bool kLong>
__global__ void __launch_bounds__(kNetLanes<kLong> * (kLong ? 1 : kThreads / 8))
    netTermsKernel(int count, const int* start, const int* long_nets, const int* pin_module, const double2* offset,
                   const double2* center, const double* weight, double* term) {
    const NetShare s = netShare<kLong>(count, start, long_nets);
    NetBox box;
#pragma unroll (kLong ? 4 : 1)
    for (int p = s.first + s.lane; p < s.last; p += kNetLanes<kLong>) {
        const double2 c = center[pin_module[p]];
        const double2 o = offset[p];
        const double x = c.x + o.x;
        const double y = c.y + o.y;
        box.min_x = x < box.min_x ? x : box.min_x;
        box.max_x = box.max_x < x ? x : box.max_x;
        box.min_y = y < box.min_y ? y : box.min_y;
        box.max_y = box.max_y < y ? y : box.max_y;
    }
    joinNet<kLong>(box);
    if (s.net >= 0 && s.lane == 0) {
        const double span = (box.max_x - box.min_x) + (box.max_y - box.min_y);
        term[s.net] = s.last - s.first < 2 ? 0.0 : __dmul_rn(weight[s.net], span);
    }
}

// Each standard cell's row (buildWindows: the nearest row by centre, if the cell sits on its
// bottom) and sort keys; the other modules sort behind every row.
__global__ void __launch_bounds__(kThreads) cellRowsKernel(int count, const uint8_t* standard, const double2* center,
                                                           const double2* size, DeviceRows rows, double* x_key,
                                                           int* cell, int* row) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= count) return;
    int r = rows.count;
    const double2 c = center[m];
    const double2 s = size[m];
    if (standard[m] != 0) {
        int lo = 0, hi = rows.count;  // first sorted row whose centre is not below the cell's
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (rows.centre[mid] < c.y) {
                lo = mid + 1;
            } else {
                hi = mid;
            }
        }
        int at = lo;
        if (lo == rows.count) {
            at = rows.count - 1;
        } else if (lo > 0 && fabs(rows.centre[lo - 1] - c.y) <= fabs(rows.centre[lo] - c.y)) {
            at = lo - 1;
        }
        const int nearest = rows.index[at];
        if (fabs(lowerLeft(c.y, s.y) - rows.bottom[nearest]) <= kSegmentEpsilon) r = nearest;
    }
    x_key[m] = lowerLeft(c.x, s.x);
    cell[m] = m;
    row[m] = r;
}

__global__ void __launch_bounds__(kThreads) rowKeysKernel(int count, const int* cell, const int* row, unsigned* key) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) key[i] = static_cast<unsigned>(row[cell[i]]);
}

// first[i] = i where a segment begins (the row's first cell, or one that does not abut the cell
// before it), else 0; a running maximum then gives every cell its segment's first position.
__global__ void __launch_bounds__(kThreads) segmentsKernel(int count, const int* cell, const unsigned* row,
                                                           const double2* center, const double2* size, DeviceRows rows,
                                                           int* first, PassCounts* counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const unsigned r = row[i];
    bool begins = true;
    if (i > 0 && row[i - 1] == r && r < static_cast<unsigned>(rows.count)) {
        const int previous = cell[i - 1];
        const int m = cell[i];
        const double left = lowerLeft(center[previous].x, size[previous].x);
        const double mine = lowerLeft(center[m].x, size[m].x);
        const double expected = __dadd_rn(left, roundedWidthDevice(size[previous].x, rows.spacing[r]));
        begins = fabs(mine - expected) > kSegmentEpsilon;
        if (mine == left) counts->ties = 1;
    }
    first[i] = begins ? i : 0;
}

__device__ __forceinline__ bool sameSegment(const int* first, const unsigned* row, int i, int j) {
    return first[i] == first[j] && row[i] == row[j];
}

// begins[i] = 1 where a window begins: every kWindow-th cell of a segment from `phase` on that
// has a cell after it; begins[count] = 0.
__global__ void __launch_bounds__(kThreads) windowBeginsKernel(int count, int phase, int rows, const int* first,
                                                               const unsigned* row, int* begins) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > count) return;
    int b = 0;
    if (i + 1 < count && row[i] < static_cast<unsigned>(rows)) {
        const int q = i - first[i] - phase;
        b = q >= 0 && q % kWindow == 0 && sameSegment(first, row, i, i + 1) ? 1 : 0;
    }
    begins[i] = b;
}

// A pass's windows in the reference's order (rows, then x), whatever their kind.
struct DeviceWindows {
    int4* modules = nullptr;  // unused slots -1
    int* count = nullptr;
    double* start_x = nullptr;
    double* bottom = nullptr;
    double* spacing = nullptr;
    int* net_start = nullptr;
    int* nets = nullptr;
    int* own = nullptr;       // per entry of nets: its first own pin among the sorted pins
    uint8_t* kind = nullptr;
    int* owner = nullptr;              // per module: its window, or -1
    int8_t* moved_orientation = nullptr;  // per module: the orientation it takes when its window is reordered
};

__global__ void __launch_bounds__(kThreads) fillWindowsKernel(int count, const int* cell, const unsigned* row,
                                                              const int* first, const int* begins, const int* id,
                                                              const double2* center, const double2* size,
                                                              const int8_t* turn, DeviceRows rows, DeviceWindows out,
                                                              PassCounts* counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) counts->windows = id[count];
    if (i >= count || begins[i] == 0) return;
    const int w = id[i];
    const unsigned r = row[i];
    int module[kWindow] = {-1, -1, -1, -1};
    int n = 0;
#pragma unroll
    for (int k = 0; k < kWindow; ++k) {
        if (n == k && i + k < count && sameSegment(first, row, i, i + k)) {
            module[k] = cell[i + k];
            ++n;
        }
    }
    out.modules[w] = make_int4(module[0], module[1], module[2], module[3]);
    out.count[w] = n;
    out.start_x[w] = lowerLeft(center[module[0]].x, size[module[0]].x);
    out.bottom[w] = rows.bottom[r];
    out.spacing[w] = rows.spacing[r];
    const int turned = rows.turn[r];
#pragma unroll
    for (int k = 0; k < kWindow; ++k) {
        if (module[k] < 0) continue;
        out.owner[module[k]] = w;
        out.moved_orientation[module[k]] = turned != kOrientationUnknown ? static_cast<int8_t>(turned) : turn[module[k]];
    }
}

__global__ void __launch_bounds__(kThreads) pinWindowsKernel(int pins, const int* pin_module, const int* owner,
                                                             const PassCounts* counts, unsigned* key) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pins) return;
    const int w = owner[pin_module[p]];
    key[p] = static_cast<unsigned>(w >= 0 ? w : counts->windows);  // behind every window
}

// head[i] = 1 where a net of a window appears first among the sorted pins; head[pins] = 0.
__global__ void __launch_bounds__(kThreads) netHeadsKernel(int pins, const unsigned* key, const int* pin,
                                                           const int* net, const PassCounts* counts, int* head) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > pins) return;
    head[i] = i < pins && key[i] < static_cast<unsigned>(counts->windows) &&
                      (i == 0 || key[i - 1] != key[i] || net[pin[i - 1]] != net[pin[i]])
                  ? 1
                  : 0;
}

__global__ void __launch_bounds__(kThreads) windowNetsKernel(int pins, const unsigned* key, const int* pin,
                                                             const int* net, const int* head, const int* at, const PassCounts* counts,
                                                             DeviceWindows out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > pins) return;
    const int windows = counts->windows;
    if (i < pins && head[i] != 0) {
        out.nets[at[i]] = net[pin[i]];
        out.own[at[i]] = i;
    }
    // The windows after the previous pin's up to this one's begin here (those between have no pins).
    const int mine = i < pins ? static_cast<int>(key[i]) : windows;
    const int before = i > 0 ? static_cast<int>(key[i - 1]) : -1;
    for (int w = before + 1; w <= mine; ++w) out.net_start[w] = at[i];
    if (mine == windows && before < windows) out.own[at[i]] = i;  // the end of the last entry
}

// Each window's kind: none without nets or with one above the degree limit.
__global__ void __launch_bounds__(kThreads) windowKindsKernel(const int* net_pin_start, unsigned long long maximum_degree,
                                                              DeviceWindows out, PassCounts* counts) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    int four = 0, tail = 0, orders = 0;
    if (w < counts->windows) {
        const int first = out.net_start[w];
        const int last = out.net_start[w + 1];
        bool takes = last > first;
        for (int e = first; e < last && takes; ++e) {
            const int n = out.nets[e];
            takes = static_cast<unsigned long long>(net_pin_start[n + 1] - net_pin_start[n]) <= maximum_degree;
        }
        four = takes && out.count[w] == kWindow ? 1 : 0;
        tail = takes && four == 0 ? 1 : 0;
        orders = takes ? factorialOf(out.count[w]) : 0;
        out.kind[w] = four != 0 ? kFourCells : (tail != 0 ? kTail : kNotEvaluated);
    }
    four = __reduce_add_sync(0xffffffffu, four);
    tail = __reduce_add_sync(0xffffffffu, tail);
    orders = __reduce_add_sync(0xffffffffu, orders);
    if ((threadIdx.x & 31) == 0 && orders > 0) {
        if (four > 0) atomicAdd(&counts->four, four);
        if (tail > 0) atomicAdd(&counts->tails, tail);
        atomicAdd(&counts->permutations, static_cast<unsigned long long>(orders));
    }
}

// Moves the cells of the accepted windows of a kind (four-cell: decided, tails: an order taken).
__global__ void __launch_bounds__(kThreads) applyWindowsKernel(int windows, WindowKind kind, const uint8_t* decided,
                                                               const int8_t* order, DeviceWindows w,
                                                               const double2* moved_center, double2* center,
                                                               int8_t* turn, PassCounts* counts) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool accepted = k < windows && w.kind[k] == kind && (kind == kTail ? order[k] >= 0 : decided[k] != 0);
    if (accepted) {
        const int4 m4 = w.modules[k];
        const int module[kWindow] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
        for (int i = 0; i < kWindow; ++i) {
            if (module[i] < 0) continue;
            center[module[i]] = moved_center[module[i]];
            turn[module[i]] = w.moved_orientation[module[i]];
        }
    }
    const unsigned all = __ballot_sync(0xffffffffu, accepted ? 1 : 0);
    if ((threadIdx.x & 31) == 0 && all != 0u) {
        atomicAdd(&counts->accepted, static_cast<unsigned long long>(__popc(all)));
    }
}

__global__ void __launch_bounds__(kThreads) resultKernel(int count, const double2* center, const int8_t* turn, double* x,
                                                         double* y, int* orientation) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= count) return;
    const double2 c = center[m];
    x[m] = c.x;
    y[m] = c.y;
    orientation[m] = turn[m];
}

struct LargerOf {
    __device__ __forceinline__ int operator()(int a, int b) const { return a < b ? b : a; }
};

// What the passes on the device hold: the arrays below (176 bytes per module, 88 per pin, 120 per
// net, 32 per row) and the sorts' workspace (12 bytes per module or 8 per pin), with slack.
uint64_t devicePassBytes(const mpgp_design& d) {
    const uint64_t modules = static_cast<uint64_t>(d.module_count);
    const uint64_t pins = static_cast<uint64_t>(d.pin_count);
    const uint64_t nets = static_cast<uint64_t>(d.net_count);
    return modules * 240 + pins * 112 + nets * 128 + static_cast<uint64_t>(d.row_count) * 32 + (uint64_t{8} << 20);
}

// The passes' arrays out of one block of the device's pool.  The pool keeps up to kKeptBytes
// of what is free for the next call; a larger design's memory goes back to the device.
constexpr uint64_t kKeptBytes = uint64_t{1} << 29;
class PassMemory {
public:
    PassMemory(cudaStream_t stream, uint64_t bytes) : stream_(stream), bytes_(bytes) {
        scratch_ = std::make_unique<Scratch>(stream, [bytes] { return bytes; });
        block_ = scratch_->array<unsigned char>(bytes);
    }
    ~PassMemory() {
        scratch_.reset();
        int device = 0;
        if (bytes_ <= kKeptBytes || cudaStreamSynchronize(stream_) != cudaSuccess || cudaGetDevice(&device) != cudaSuccess) {
            return;
        }
        cudaMemPoolTrimTo(devicePool(device), kKeptBytes);
    }
    PassMemory(const PassMemory&) = delete;
    PassMemory& operator=(const PassMemory&) = delete;
    template <typename T>
    T* array(std::size_t count) {
        const std::size_t at = (used_ + 255) / 256 * 256;
        require(at + count * sizeof(T) <= bytes_, "The detailed-placement arrays exceed their block.");
        used_ = at + count * sizeof(T);
        return reinterpret_cast<T*>(block_ + at);
    }

private:
    cudaStream_t stream_;
    std::unique_ptr<Scratch> scratch_;
    unsigned char* block_ = nullptr;
    std::size_t bytes_;
    std::size_t used_ = 0;
};

// Every pass on the device.  False, with nothing written, where the host has to look: an entry
// that validation refuses, rows of which cells share an x (the host's sort decides their
// order), rounds that do not end in kMaxRounds, or no memory for the arrays.
bool placeOnDevice(const mpgp_design& d, const int32_t* row_orientation, const mpgp_detailed_options& options,
                   double* module_x, double* module_y, int32_t* module_orientation, mpgp_detailed_result& result) {
    for (int32_t r = 0; r < d.row_count; ++r) {
        const bool good = std::isfinite(d.row_bottom[r]) && std::isfinite(d.row_height[r]) &&
                          std::isfinite(d.row_site_spacing[r]) && std::isfinite(d.row_x_start[r]) &&
                          d.row_site_count[r] >= 0 &&
                          (row_orientation == nullptr ||
                           (row_orientation[r] >= 0 && row_orientation[r] <= kOrientationUnknown));
        if (!good) return false;
    }
    const auto started = std::chrono::steady_clock::now();
    const int modules = d.module_count;
    const int pins = static_cast<int>(d.pin_count);
    const int nets = d.net_count;
    const std::size_t rows = static_cast<std::size_t>(d.row_count);
    Stream owned_stream;
    const cudaStream_t stream = owned_stream.get();
    Stream side;  // the HPWL terms' way to the host
    Event terms;
    std::unique_ptr<PassMemory> memory;
    try {
        memory = std::make_unique<PassMemory>(stream, devicePassBytes(d));
    } catch (const Error&) {
        cudaGetLastError();
        return false;  // the host's path says what is missing
    }
    PassMemory& scratch = *memory;
    const auto put = [&](const auto* host, std::size_t count) {
        using T = std::remove_const_t<std::remove_pointer_t<decltype(host)>>;
        T* device = scratch.array<T>(count);
        checkCuda(cudaMemcpyAsync(device, host, count * sizeof(T), cudaMemcpyHostToDevice, stream), "upload the design");
        return device;
    };

    // The rows in bottom order (buildWindows).
    std::vector<std::size_t> sorted_rows(rows);
    std::iota(sorted_rows.begin(), sorted_rows.end(), 0U);
    std::sort(sorted_rows.begin(), sorted_rows.end(),
              [&](std::size_t a, std::size_t b) { return d.row_bottom[a] < d.row_bottom[b]; });
    std::vector<double> centres(rows);
    std::vector<int> indices(rows), turns(rows);
    for (std::size_t k = 0; k < rows; ++k) {
        const std::size_t r = sorted_rows[k];
        centres[k] = d.row_bottom[r] + d.row_height[r] * 0.5;
        indices[k] = static_cast<int>(r);
        turns[k] = row_orientation != nullptr ? row_orientation[k] : 0;
    }
    DeviceRows row_data;
    row_data.count = d.row_count;
    row_data.centre = put(centres.data(), rows);
    row_data.index = put(indices.data(), rows);
    row_data.bottom = put(d.row_bottom, rows);
    row_data.spacing = put(d.row_site_spacing, rows);
    row_data.turn = put(turns.data(), rows);

    const std::size_t m_count = static_cast<std::size_t>(modules);
    const std::size_t p_count = static_cast<std::size_t>(pins);
    const std::size_t n_count = static_cast<std::size_t>(nets);
    const std::size_t w_count = m_count / 2 + 1;  // every window holds two cells at least
    static_assert(sizeof(long long) == sizeof(int64_t), "net offsets are 64-bit");
    RawDesign raw;
    raw.modules = modules;
    raw.nets = nets;
    raw.pins = pins;
    double* x = put(d.module_x, m_count);
    double* y = put(d.module_y, m_count);
    raw.x = x;
    raw.y = y;
    raw.width = put(d.module_width, m_count);
    raw.height = put(d.module_height, m_count);
    raw.flags = put(d.module_flags, m_count);
    if (d.module_orientation != nullptr) raw.orientation = put(d.module_orientation, m_count);
    raw.net_start = put(reinterpret_cast<const long long*>(d.net_pin_start), n_count + 1);
    raw.net_weight = put(d.net_weight, n_count);
    raw.pin_module = put(d.pin_module, p_count);
    raw.offset_x = put(d.pin_offset_x, p_count);
    raw.offset_y = put(d.pin_offset_y, p_count);
    const int* pin_module = raw.pin_module;
    const double* net_weight = raw.net_weight;
    int* changed = scratch.array<int>(kMaxRounds + kRoundsPerCheck + 1);
    PassCounts* counts = scratch.array<PassCounts>(1);
    int* long_nets = scratch.array<int>(p_count / kLongNet + 1);
    const PinnedBlock readback(sizeof(PassCounts) + 2 * sizeof(int), "detailed-placement counters");
    PassCounts* const host_counts = reinterpret_cast<PassCounts*>(readback.data());
    int* const host_changed = reinterpret_cast<int*>(readback.data() + sizeof(PassCounts));
    // The checks, before any kernel follows an index.
    checkCuda(cudaMemsetAsync(changed, 0, 2 * sizeof(int), stream), "check the design");
    checkDesignKernel<<<threadBlocks(std::max({m_count, n_count, p_count})), kThreads, 0, stream>>>(raw, changed,
                                                                                                       long_nets);
    checkCuda(cudaMemcpyAsync(host_changed, changed, 2 * sizeof(int), cudaMemcpyDeviceToHost, stream), "check the design");
    checkCuda(cudaStreamSynchronize(stream), "check the design");
    if (host_changed[0] != 0) return false;
    const int long_count = host_changed[1];

    double2* center = scratch.array<double2>(m_count);
    double2* moved_center = scratch.array<double2>(m_count);
    double2* size = scratch.array<double2>(m_count);
    int8_t* turn = scratch.array<int8_t>(m_count);
    uint8_t* is_standard = scratch.array<uint8_t>(m_count);
    detailedModulesKernel<<<threadBlocks(m_count), kThreads, 0, stream>>>(raw, nominalRowHeight(d), center, size, turn,
                                                                          is_standard);
    checkCuda(cudaGetLastError(), "detailed placement on the device");
    int* net_pin_start = scratch.array<int>(n_count + 1);
    int* pin_net = scratch.array<int>(p_count);
    int* pin_index = scratch.array<int>(p_count);
    launchNets(nets, long_count, [&](auto is_long, int blocks, int threads) {
        detailedNetsKernel<decltype(is_long)::value><<<blocks, threads, 0, stream>>>(nets, raw.net_start, long_nets,
                                                                                    net_pin_start, pin_net, pin_index);
    });
    double2* raw_offset = scratch.array<double2>(p_count);
    double2* pin_offset = scratch.array<double2>(p_count);
    rawOffsetsKernel<<<threadBlocks(p_count), kThreads, 0, stream>>>(pins, raw.offset_x, raw.offset_y, raw_offset);
    double* term_before = scratch.array<double>(n_count);
    double* term_after = scratch.array<double>(n_count);
    const auto turnOffsets = [&] {
        turnedOffsetsKernel<<<threadBlocks(p_count), kThreads, 0, stream>>>(pins, raw_offset, pin_module, turn, pin_offset);
    };
    const auto netTerms = [&](double* term) {
        launchNets(nets, long_count, [&](auto is_long, int blocks, int threads) {
            netTermsKernel<decltype(is_long)::value><<<blocks, threads, 0, stream>>>(
                nets, net_pin_start, long_nets, pin_module, pin_offset, center, net_weight, term);
        });
        checkCuda(cudaGetLastError(), "net terms");
    };
    turnOffsets();
    netTerms(term_before);
    checkCuda(cudaEventRecord(terms.get(), stream), "net terms");
    checkCuda(cudaStreamWaitEvent(side.get(), terms.get(), 0), "net terms");

    double* x_key = scratch.array<double>(m_count);
    double* x_sorted = scratch.array<double>(m_count);
    int* cell = scratch.array<int>(m_count);
    int* cell_by_x = scratch.array<int>(m_count);
    int* row = scratch.array<int>(m_count);
    unsigned* row_key = scratch.array<unsigned>(m_count);
    unsigned* row_sorted = scratch.array<unsigned>(m_count);
    int* first = scratch.array<int>(m_count);
    int* segment = scratch.array<int>(m_count);
    int* begins = scratch.array<int>(m_count + 1);
    int* window_id = scratch.array<int>(m_count + 1);
    unsigned* pin_key = scratch.array<unsigned>(p_count);
    unsigned* pin_key_sorted = scratch.array<unsigned>(p_count);
    int* pin_sorted = scratch.array<int>(p_count);
    int* head = scratch.array<int>(p_count + 1);
    int* head_at = scratch.array<int>(p_count + 1);
    DeviceWindows windows;
    windows.modules = scratch.array<int4>(w_count);
    windows.count = scratch.array<int>(w_count);
    windows.start_x = scratch.array<double>(w_count);
    windows.bottom = scratch.array<double>(w_count);
    windows.spacing = scratch.array<double>(w_count);
    windows.net_start = scratch.array<int>(w_count + 1);
    windows.nets = scratch.array<int>(p_count);
    windows.own = scratch.array<int>(p_count + 1);
    windows.kind = scratch.array<uint8_t>(w_count);
    windows.owner = scratch.array<int>(m_count);
    windows.moved_orientation = scratch.array<int8_t>(m_count);
    int* best_order = scratch.array<int>(w_count);
    uint8_t* decided[2] = {scratch.array<uint8_t>(w_count), scratch.array<uint8_t>(w_count)};
    int8_t* taken[2] = {scratch.array<int8_t>(w_count), scratch.array<int8_t>(w_count)};
    NetExtremes* extremes = scratch.array<NetExtremes>(n_count);
    int* stamp = scratch.array<int>(n_count);

    const auto bitsFor = [](uint64_t largest) {
        int bits = 1;
        while ((largest >> bits) != 0) ++bits;
        return bits;
    };
    const int row_bits = bitsFor(rows);
    const int window_bits = bitsFor(w_count);
    std::size_t workspace_bytes = 0;
    const auto grow = [&](cudaError_t status, std::size_t bytes) {
        checkCuda(status, "size a sort's workspace");
        workspace_bytes = std::max(workspace_bytes, bytes);
    };
    std::size_t bytes = 0;
    grow(cub::DeviceRadixSort::SortPairs(nullptr, bytes, x_key, x_sorted, cell, cell_by_x, modules, 0, 64, stream), bytes);
    grow(cub::DeviceRadixSort::SortPairs(nullptr, bytes, row_key, row_sorted, cell_by_x, cell, modules, 0, row_bits, stream),
         bytes);
    grow(cub::DeviceRadixSort::SortPairs(nullptr, bytes, pin_key, pin_key_sorted, pin_index, pin_sorted, pins, 0, window_bits,
                                         stream),
         bytes);
    grow(cub::DeviceScan::InclusiveScan(nullptr, bytes, first, segment, LargerOf{}, modules, stream), bytes);
    grow(cub::DeviceScan::ExclusiveSum(nullptr, bytes, head, head_at, pins + 1, stream), bytes);
    grow(cub::DeviceScan::ExclusiveSum(nullptr, bytes, begins, window_id, modules + 1, stream), bytes);
    void* workspace = scratch.array<unsigned char>(workspace_bytes);
    result.cuda_reserved_memory_bytes = devicePassBytes(d);
    const auto readCounts = [&] {
        checkCuda(cudaMemcpyAsync(host_counts, counts, sizeof(PassCounts), cudaMemcpyDeviceToHost, stream), "pass counts");
        checkCuda(cudaStreamSynchronize(stream), "detailed-placement pass");
    };
    // Rounds until one changes nothing; launch(rounds, in) launches round `rounds.round` from
    // decisions `in` (0 or 1) into the other.
    const auto settle = [&](const auto& launch) {
        checkCuda(cudaMemsetAsync(stamp, 0, n_count * sizeof(int), stream), "clear the rounds");
        checkCuda(cudaMemsetAsync(changed, 0, (kMaxRounds + kRoundsPerCheck + 1) * sizeof(int), stream), "clear the rounds");
        for (int round = 1; round <= kMaxRounds; round += kRoundsPerCheck) {
            for (int k = round; k < round + kRoundsPerCheck; ++k) launch(Rounds{k, stamp, changed}, (k - 1) & 1);
            checkCuda(cudaGetLastError(), "re-decide the windows");
            checkCuda(cudaMemcpyAsync(host_changed, changed + round + kRoundsPerCheck - 1, sizeof(int),
                                      cudaMemcpyDeviceToHost, stream),
                      "read the rounds");
            checkCuda(cudaStreamSynchronize(stream), "re-decide the windows");
            if (*host_changed == 0) return true;
        }
        return false;
    };

    // calculateHpwl (Metrics.cpp:128-147): the nets' terms in net order.
    const auto sum = [&](const double* term, cudaStream_t on) {
        double total = 0.0;
        readDown(term, n_count,
                 [&](const double* v, std::size_t count) {
                     for (std::size_t k = 0; k < count; ++k) total += v[k];
                 },
                 on);
        return total;
    };
    const int longest = static_cast<int>(
        std::min<uint64_t>(options.maximum_net_degree, static_cast<uint64_t>(std::numeric_limits<int>::max())));
    double hpwl_before = 0.0;
    uint64_t evaluated = 0, permutations = 0, accepted = 0;
    for (int pass = 0; pass < options.passes; ++pass) {
        const int phase = (pass % 2) * (kWindow / 2);
        checkCuda(cudaMemsetAsync(counts, 0, sizeof(PassCounts), stream), "clear the counts");
        checkCuda(cudaMemsetAsync(windows.owner, 0xFF, m_count * sizeof(int), stream), "clear the owners");
        const int module_blocks = threadBlocks(m_count + 1);
        const int pin_blocks = threadBlocks(p_count + 1);
        cellRowsKernel<<<module_blocks, kThreads, 0, stream>>>(modules, is_standard, center, size, row_data, x_key, cell, row);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceRadixSort::SortPairs(workspace, bytes, x_key, x_sorted, cell, cell_by_x, modules, 0, 64, stream),
                  "sort the cells by x");
        rowKeysKernel<<<module_blocks, kThreads, 0, stream>>>(modules, cell_by_x, row, row_key);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceRadixSort::SortPairs(workspace, bytes, row_key, row_sorted, cell_by_x, cell, modules, 0, row_bits,
                                                  stream),
                  "sort the cells by row");
        segmentsKernel<<<module_blocks, kThreads, 0, stream>>>(modules, cell, row_sorted, center, size, row_data, first, counts);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceScan::InclusiveScan(workspace, bytes, first, segment, LargerOf{}, modules, stream), "segments");
        windowBeginsKernel<<<module_blocks, kThreads, 0, stream>>>(modules, phase, row_data.count, segment, row_sorted, begins);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceScan::ExclusiveSum(workspace, bytes, begins, window_id, modules + 1, stream), "windows");
        fillWindowsKernel<<<module_blocks, kThreads, 0, stream>>>(modules, cell, row_sorted, segment, begins, window_id, center,
                                                                  size, turn, row_data, windows, counts);
        pinWindowsKernel<<<pin_blocks, kThreads, 0, stream>>>(pins, pin_module, windows.owner, counts, pin_key);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceRadixSort::SortPairs(workspace, bytes, pin_key, pin_key_sorted, pin_index, pin_sorted, pins, 0,
                                                  window_bits, stream),
                  "sort the pins by window");
        netHeadsKernel<<<pin_blocks, kThreads, 0, stream>>>(pins, pin_key_sorted, pin_sorted, pin_net, counts, head);
        bytes = workspace_bytes;
        checkCuda(cub::DeviceScan::ExclusiveSum(workspace, bytes, head, head_at, pins + 1, stream), "window nets");
        windowNetsKernel<<<pin_blocks, kThreads, 0, stream>>>(pins, pin_key_sorted, pin_sorted, pin_net, head, head_at, counts,
                                                              windows);
        windowKindsKernel<<<threadBlocks(w_count), kThreads, 0, stream>>>(net_pin_start, options.maximum_net_degree, windows,
                                                                          counts);
        checkCuda(cudaGetLastError(), "build the windows");
        if (pass == 0) hpwl_before = sum(term_before, side.get());  // while the device builds the windows
        readCounts();
        if (host_counts->ties != 0) return false;
        const int total = host_counts->windows;
        evaluated += static_cast<uint64_t>(total);
        permutations += host_counts->permutations;
        const unsigned warps = static_cast<unsigned>((total + kWindowsPerBlock - 1) / kWindowsPerBlock);
        if (host_counts->four > 0) {
            if (pass > 0) turnOffsets();
            const WindowArrays arrays{windows.modules, windows.start_x, windows.bottom,
                                      windows.spacing, windows.net_start, windows.nets};
            launchNets(nets, longest > kLongNet ? long_count : 0, [&](auto is_long, int blocks, int threads) {
                netExtremesKernel<decltype(is_long)::value><<<blocks, threads, 0, stream>>>(
                    nets, net_pin_start, long_nets, longest, pin_module, pin_offset, center, windows.owner, extremes);
            });
            windowOrdersKernel<true><<<warps, 32 * kWindowsPerBlock, 0, stream>>>(
                center, size, pin_module, pin_offset, net_pin_start, net_weight, arrays, total, windows.kind,
                options.improvement_epsilon, best_order, decided[0], moved_center,
                OwnPins{windows.own, pin_sorted, extremes});
            const bool settled = settle([&](const Rounds& rounds, int in) {
                speculativeValuesKernel<<<warps, 32 * kWindowsPerBlock, 0, stream>>>(
                    center, moved_center, windows.owner, windows.moved_orientation, raw_offset, pin_offset, pin_module,
                    net_pin_start, net_weight, arrays, total, best_order, options.improvement_epsilon, decided[in],
                    decided[in ^ 1], nullptr, nullptr, rounds);
            });
            if (!settled) return false;
            applyWindowsKernel<<<threadBlocks(static_cast<std::size_t>(total)), kThreads, 0, stream>>>(
                total, kFourCells, decided[0], nullptr, windows, moved_center, center, turn, counts);
        }
        if (host_counts->tails > 0) {
            const TailArrays tail{windows.modules, windows.count, windows.start_x, windows.bottom,
                                  windows.spacing, windows.net_start, windows.nets};
            checkCuda(cudaMemsetAsync(taken[0], 0xFF, static_cast<std::size_t>(total), stream), "tail orders");
            const bool settled = settle([&](const Rounds& rounds, int in) {
                if (rounds.round > 1) {
                    tailPlacementKernel<<<threadBlocks(static_cast<std::size_t>(total)), kThreads, 0, stream>>>(
                        tail, total, size, taken[in], moved_center, rounds);
                }
                tailOrdersKernel<<<warps, 32 * kWindowsPerBlock, 0, stream>>>(
                    center, turn, moved_center, windows.owner, 0, windows.moved_orientation, raw_offset, size, pin_module,
                    net_pin_start, net_weight, tail, total, windows.kind, options.improvement_epsilon, taken[in],
                    taken[in ^ 1], rounds);
            });
            if (!settled) return false;
            applyWindowsKernel<<<threadBlocks(static_cast<std::size_t>(total)), kThreads, 0, stream>>>(
                total, kTail, nullptr, taken[0], windows, moved_center, center, turn, counts);
        }
        checkCuda(cudaGetLastError(), "detailed-placement pass");
        if (pass + 1 == options.passes) break;
        readCounts();
        accepted += host_counts->accepted;
    }
    turnOffsets();
    netTerms(term_after);
    int* orientation_out = row;  // the arrays of the cell sort are free again
    resultKernel<<<threadBlocks(m_count), kThreads, 0, stream>>>(modules, center, turn, x, y, orientation_out);
    checkCuda(cudaGetLastError(), "detailed-placement result");
    readCounts();
    accepted += host_counts->accepted;
    result.hpwl_before = hpwl_before;
    result.hpwl_after = sum(term_after, side.get());
    const auto bring = [&](const auto* device, auto* host) {
        checkCuda(cudaMemcpyAsync(host, device, m_count * sizeof(*host), cudaMemcpyDeviceToHost, stream), "detailed-placement result");
    };
    bring(x, module_x);
    bring(y, module_y);
    if (module_orientation != nullptr) bring(orientation_out, module_orientation);
    checkCuda(cudaStreamSynchronize(stream), "detailed-placement result");
    result.cuda_device_used = options.cuda_device;
    result.evaluated_windows = evaluated;
    result.evaluated_permutations = permutations;
    result.accepted_operations = accepted;
    result.completed_passes = options.passes;
    result.elapsed_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - started).count();
    return true;
}

// The bytes the host's lists reserve on the device (detailedPlace).
uint64_t hostListBytes(const mpgp_design& d) {
    const auto of = [](uint64_t count, uint64_t size) { return std::max<uint64_t>(count, 1) * size; };
    const uint64_t modules = static_cast<uint64_t>(d.module_count);
    const uint64_t pins = static_cast<uint64_t>(d.pin_count);
    const uint64_t nets = static_cast<uint64_t>(d.net_count);
    const uint64_t windows = modules / kWindow + 1;
    const uint64_t tails = modules / 2 + 1;
    return of(modules, 16 + 16 + 4 + 1 + 16 + 1) + of(pins, 16 + 16 + 4 + 4) + of(nets + 1, 4) + of(nets, 8) +
           windows * (16 + 3 * 8 + 4 + 2 * 8 + 2) + (windows + 1) * 4 + tails * (16 + 4 + 3 * 8 + 2) + (tails + 1) * 4;
}

}  // namespace

bool detailedPlace(const mpgp_design& d, const int32_t* row_orientation, const mpgp_detailed_options& options,
                   double* module_x, double* module_y, int32_t* module_orientation, mpgp_detailed_result& result,
                   std::string& reason) {
    reason.clear();
    // The checks of tryRunCudaDetailedPlacement (:493-523), without the home
    // server's device allow-list and free-memory reserve.
    if (options.method != MPGP_DETAILED_WINDOW_REORDER || options.window_size != kWindow) {
        reason = "CUDA detailed placement currently supports window reordering with a four-cell window only.";
        return false;
    }
    if (options.passes <= 0 || options.maximum_net_degree < 2U || options.improvement_epsilon < 0.0 ||
        options.maximum_cuda_memory_bytes == 0U) {
        reason = "CUDA detailed-placement options are outside their valid range.";
        return false;
    }
    validateDesignShape(d);
    const auto validate = [&] {
        validateDesign(d);
        for (int32_t m = 0; d.module_orientation != nullptr && m < d.module_count; ++m) {
            require(d.module_orientation[m] >= 0 && d.module_orientation[m] <= kOrientationUnknown,
                    "Module orientations must be Orientation values (0-8).");
        }
        for (int32_t r = 0; row_orientation != nullptr && r < d.row_count; ++r) {
            require(row_orientation[r] >= 0 && row_orientation[r] <= kOrientationUnknown,
                    "Row orientations must be Orientation values (0-8).");
        }
    };
    int device_count = 0;
    if (cudaGetDeviceCount(&device_count) != cudaSuccess || options.cuda_device < 0 ||
        options.cuda_device >= device_count) {
        cudaGetLastError();
        validate();
        reason = "Requested CUDA device is unavailable on this host.";
        return false;
    }
    int previous_device = 0;
    cudaGetDevice(&previous_device);
    if (cudaSetDevice(options.cuda_device) != cudaSuccess) {
        cudaGetLastError();
        validate();
        reason = "Unable to select the requested CUDA device.";
        return false;
    }
    struct RestoreDevice {
        int device;
        ~RestoreDevice() { cudaSetDevice(device); }
    } restore{previous_device};
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, options.cuda_device) != cudaSuccess || major < 6) {
        validate();
        reason = "Requested CUDA device lacks required double-precision support.";
        return false;
    }
    // The device takes every design it can (the rules above placeOnDevice) whose arrays, and
    // those of the host's lists, the caller's budget allows.  Two passes, host's lists against
    // device, a B200 with 16 host CPUs: 50 cells 1.9 / 0.8 ms, 500 2.2 / 1.0, 2,000 3.0 / 1.1, 8,000
    // 5.3 / 1.4, 30,000 12.9 / 2.0, 210,000 61 / 5.3.
    result = mpgp_detailed_result{};
    const uint64_t budget = options.maximum_cuda_memory_bytes;
    if (d.module_count > 0 && d.pin_count > 0 && d.net_count > 0 && d.row_count > 0 && hostListBytes(d) <= budget &&
        devicePassBytes(d) <= budget &&
        placeOnDevice(d, row_orientation, options, module_x, module_y, module_orientation, result)) {
        return true;
    }
    result = mpgp_detailed_result{};
    validate();
    std::size_t free_bytes = 0;
    std::size_t total_bytes = 0;
    checkCuda(cudaMemGetInfo(&free_bytes, &total_bytes), "cudaMemGetInfo");
    const uint64_t limit = std::min<uint64_t>(budget, free_bytes);

    const DerivedDesign derived = deriveDesign(d, false);
    std::vector<uint8_t> standard(static_cast<std::size_t>(d.module_count));
    for (int32_t m = 0; m < d.module_count; ++m) standard[m] = derived.is_fixed[m] == 0 && derived.is_macro[m] == 0;
    const auto rowOrientation = [&](int r) { return row_orientation != nullptr ? row_orientation[r] : 0; };
    const Workers workers = Workers::all(16);
    Placement s(d);
    result.hpwl_before = s.hpwl(workers);
    result.cuda_device_used = options.cuda_device;
    const auto started = std::chrono::steady_clock::now();

    // Device copies of the design: sizes, pin modules and net CSR once; centres
    // and orientation-transformed pin offsets at the start of every pass.
    const std::size_t modules = static_cast<std::size_t>(d.module_count);
    const std::size_t pins = static_cast<std::size_t>(d.pin_count);
    const std::size_t nets = static_cast<std::size_t>(d.net_count);
    const std::size_t window_capacity = modules / kWindow + 1;
    uint64_t reserved = 0;
    DeviceArray<double2> center, moved_center, size, pin_offset, raw_offset;
    DeviceArray<int> pin_module, net_pin_start, owner;
    DeviceArray<int8_t> moved_orientation;
    DeviceArray<double> net_weight;
    DeviceArray<int4> window_modules;
    DeviceArray<double> window_start, window_bottom, window_spacing, value_before, value_after;
    DeviceArray<int> window_net_start, window_nets, best_order;
    DeviceArray<uint8_t> decided[2];
    center.allocate(modules, reserved, limit, "CUDA detailed module centers");
    moved_center.allocate(modules, reserved, limit, "CUDA detailed moved centers");
    owner.allocate(modules, reserved, limit, "CUDA detailed window owners");
    moved_orientation.allocate(modules, reserved, limit, "CUDA detailed moved orientations");
    size.allocate(modules, reserved, limit, "CUDA detailed module sizes");
    pin_offset.allocate(pins, reserved, limit, "CUDA detailed pin offsets");
    raw_offset.allocate(pins, reserved, limit, "CUDA detailed raw pin offsets");
    pin_module.allocate(pins, reserved, limit, "CUDA detailed pin modules");
    net_pin_start.allocate(nets + 1, reserved, limit, "CUDA detailed net offsets");
    net_weight.allocate(nets, reserved, limit, "CUDA detailed net weights");
    window_modules.allocate(window_capacity, reserved, limit, "CUDA detailed window modules");
    window_start.allocate(window_capacity, reserved, limit, "CUDA detailed window start x");
    window_bottom.allocate(window_capacity, reserved, limit, "CUDA detailed window bottoms");
    window_spacing.allocate(window_capacity, reserved, limit, "CUDA detailed window spacing");
    window_net_start.allocate(window_capacity + 1, reserved, limit, "CUDA detailed window net offsets");
    window_nets.allocate(std::max<std::size_t>(pins, 1), reserved, limit, "CUDA detailed window net ids");
    best_order.allocate(window_capacity, reserved, limit, "CUDA detailed best orders");
    value_before.allocate(window_capacity, reserved, limit, "CUDA detailed window values");
    value_after.allocate(window_capacity, reserved, limit, "CUDA detailed window values");
    decided[0].allocate(window_capacity, reserved, limit, "CUDA detailed decisions");
    decided[1].allocate(window_capacity, reserved, limit, "CUDA detailed decisions");
    const std::size_t tail_capacity = modules / 2 + 1;  // every window holds two cells at least
    DeviceArray<int4> tail_modules;
    DeviceArray<int> tail_count, tail_net_start;
    DeviceArray<double> tail_start, tail_bottom, tail_spacing;
    DeviceArray<int8_t> tail_decided[2], orientation_now;
    tail_modules.allocate(tail_capacity, reserved, limit, "CUDA detailed tail windows");
    tail_count.allocate(tail_capacity, reserved, limit, "CUDA detailed tail windows");
    tail_start.allocate(tail_capacity, reserved, limit, "CUDA detailed tail windows");
    tail_bottom.allocate(tail_capacity, reserved, limit, "CUDA detailed tail windows");
    tail_spacing.allocate(tail_capacity, reserved, limit, "CUDA detailed tail windows");
    tail_net_start.allocate(tail_capacity + 1, reserved, limit, "CUDA detailed tail window net offsets");
    tail_decided[0].allocate(tail_capacity, reserved, limit, "CUDA detailed tail orders");
    tail_decided[1].allocate(tail_capacity, reserved, limit, "CUDA detailed tail orders");
    orientation_now.allocate(modules, reserved, limit, "CUDA detailed orientations");
    result.cuda_reserved_memory_bytes = reserved;

    Stream stream;
    {
        std::vector<double2> sizes(modules);
        for (std::size_t m = 0; m < modules; ++m) sizes[m] = make_double2(d.module_width[m], d.module_height[m]);
        const std::vector<int> modules_of_pins(d.pin_module, d.pin_module + pins);
        std::vector<int> starts(nets + 1);
        for (std::size_t n = 0; n <= nets; ++n) starts[n] = static_cast<int>(d.net_pin_start[n]);
        const std::vector<double> weights(d.net_weight, d.net_weight + nets);
        std::vector<double2> raw(pins);
        for (std::size_t q = 0; q < pins; ++q) raw[q] = make_double2(d.pin_offset_x[q], d.pin_offset_y[q]);
        raw_offset.upload(raw, stream.get());
        size.upload(sizes, stream.get());
        pin_module.upload(modules_of_pins, stream.get());
        net_pin_start.upload(starts, stream.get());
        net_weight.upload(weights, stream.get());
        checkCuda(cudaStreamSynchronize(stream.get()), "detailed-placement upload");
    }

    Windows windows;
    std::vector<double2> host_center(modules);
    std::vector<double2> host_offset(pins);
    std::vector<int4> host_modules;
    std::vector<double> host_start, host_bottom, host_spacing, before, after;
    std::vector<int> host_net_start, host_nets, best, host_owner(modules);
    std::vector<int8_t> host_moved_orientation(modules);
    std::vector<uint8_t> assumed, divergent(nets);
    std::vector<int4> tail_host_modules;
    std::vector<int> tail_host_count, tail_host_net_start, tail_host_nets, tail_of_window;
    std::vector<double> tail_host_start, tail_host_bottom, tail_host_spacing;
    std::vector<int8_t> tail_result, tail_assumed, host_orientation_now(modules);
    for (int pass = 0; pass < options.passes; ++pass) {
        buildWindows(s, standard, (pass % 2) * (kWindow / 2), options.maximum_net_degree, workers, windows);
        const std::size_t total = windows.row.size();
        host_modules.clear();
        host_start.clear();
        host_bottom.clear();
        host_spacing.clear();
        host_net_start.assign(1, 0);
        host_nets.clear();
        std::vector<std::size_t> on_device;
        for (std::size_t k = 0; k < total; ++k) {
            if (windows.device[k] == 0) continue;
            on_device.push_back(k);
            const int32_t* m = &windows.modules[k * kWindow];
            host_modules.push_back(make_int4(m[0], m[1], m[2], m[3]));
            host_start.push_back(s.lowerLeftX(m[0]));
            host_bottom.push_back(d.row_bottom[windows.row[k]]);
            host_spacing.push_back(d.row_site_spacing[windows.row[k]]);
            for (int64_t e = windows.net_start[k]; e < windows.net_start[k + 1]; ++e) host_nets.push_back(windows.nets[e]);
            host_net_start.push_back(static_cast<int>(host_nets.size()));
        }
        const std::size_t count = on_device.size();
        require(count <= window_capacity && host_nets.size() <= std::max<std::size_t>(pins, 1),
                "Detailed-placement window arrays exceed their capacity.");
        // The host-rule windows with nets to evaluate (optimizeCpuWindow returns
        // at once for the others).
        tail_host_modules.clear();
        tail_host_count.clear();
        tail_host_start.clear();
        tail_host_bottom.clear();
        tail_host_spacing.clear();
        tail_host_net_start.assign(1, 0);
        tail_host_nets.clear();
        tail_of_window.assign(total, -1);
        for (std::size_t k = 0; k < total; ++k) {
            if (windows.device[k] != 0 || windows.net_start[k + 1] == windows.net_start[k]) continue;
            bool too_wide = false;
            for (int64_t e = windows.net_start[k]; e < windows.net_start[k + 1]; ++e) {
                const int32_t net = windows.nets[e];
                too_wide |= static_cast<uint64_t>(d.net_pin_start[net + 1] - d.net_pin_start[net]) >
                            options.maximum_net_degree;
            }
            if (too_wide) continue;
            tail_of_window[k] = static_cast<int>(tail_host_count.size());
            const int32_t* m = &windows.modules[k * kWindow];
            tail_host_modules.push_back(make_int4(m[0], m[1], m[2], m[3]));
            tail_host_count.push_back(windows.count[k]);
            tail_host_start.push_back(s.lowerLeftX(m[0]));
            tail_host_bottom.push_back(d.row_bottom[windows.row[k]]);
            tail_host_spacing.push_back(d.row_site_spacing[windows.row[k]]);
            for (int64_t e = windows.net_start[k]; e < windows.net_start[k + 1]; ++e) {
                tail_host_nets.push_back(windows.nets[e]);
            }
            tail_host_net_start.push_back(static_cast<int>(tail_host_nets.size()));
        }
        const std::size_t tails = tail_host_count.size();
        require(tails <= tail_capacity && tail_host_nets.size() <= std::max<std::size_t>(pins, 1),
                "Detailed-placement tail window arrays exceed their capacity.");
        if (count > 0 || tails > 0) {
            // Owners: device window j as j, tail window t as count + t; and the
            // orientation a moved cell takes.
            std::fill(host_owner.begin(), host_owner.end(), -1);
            for (std::size_t m = 0; m < modules; ++m) host_moved_orientation[m] = static_cast<int8_t>(s.orientation[m]);
            const auto own = [&](std::size_t k, int value) {
                const int32_t* m = &windows.modules[k * kWindow];
                const int r = windows.row[k];
                for (int i = 0; i < windows.count[k]; ++i) {
                    host_owner[m[i]] = value;
                    if (rowOrientation(r) != kOrientationUnknown) {
                        host_moved_orientation[m[i]] = static_cast<int8_t>(rowOrientation(r));
                    }
                }
            };
            for (std::size_t j = 0; j < count; ++j) own(on_device[j], static_cast<int>(j));
            for (std::size_t k = 0; k < total; ++k) {
                if (tail_of_window[k] >= 0) own(k, static_cast<int>(count) + tail_of_window[k]);
            }
            owner.upload(host_owner, stream.get());
            moved_orientation.upload(host_moved_orientation, stream.get());
        }
        best.assign(count, 0);
        before.assign(count, 0.0);
        after.assign(count, 0.0);
        assumed.assign(count, 0);
        if (count > 0) {
            for (std::size_t m = 0; m < modules; ++m) host_center[m] = make_double2(s.cx[m], s.cy[m]);
            workers.blocks(pins, 65536, [&](std::size_t b, std::size_t e) {
                for (std::size_t p = b; p < e; ++p) {
                    double ox = 0.0;
                    double oy = 0.0;
                    transform(d.pin_offset_x[p], d.pin_offset_y[p], s.orientation[d.pin_module[p]], ox, oy);
                    host_offset[p] = make_double2(ox, oy);
                }
            });
            center.upload(host_center, stream.get());
            pin_offset.upload(host_offset, stream.get());
            window_modules.upload(host_modules, stream.get());
            window_start.upload(host_start, stream.get());
            window_bottom.upload(host_bottom, stream.get());
            window_spacing.upload(host_spacing, stream.get());
            window_net_start.upload(host_net_start, stream.get());
            window_nets.upload(host_nets, stream.get());
            const WindowArrays arrays{window_modules.get(), window_start.get(), window_bottom.get(),
                                      window_spacing.get(), window_net_start.get(), window_nets.get()};
            const int n = static_cast<int>(count);
            const unsigned blocks = static_cast<unsigned>((count + kWindowsPerBlock - 1) / kWindowsPerBlock);
            windowOrdersKernel<false><<<blocks, 32 * kWindowsPerBlock, 0, stream.get()>>>(
                center.get(), size.get(), pin_module.get(), pin_offset.get(), net_pin_start.get(), net_weight.get(),
                arrays, n, nullptr, options.improvement_epsilon, best_order.get(), decided[0].get(), moved_center.get(),
                OwnPins{});
            checkCuda(cudaGetLastError(), "windowOrdersKernel launch");
            // Each iteration re-decides every window on the previous iteration's
            // decisions; the last one's input is the assumption its values rest on.
            int in = 0;
            for (int iteration = 0; iteration < kSpeculations; ++iteration, in ^= 1) {
                speculativeValuesKernel<<<blocks, 32 * kWindowsPerBlock, 0, stream.get()>>>(
                    center.get(), moved_center.get(), owner.get(), moved_orientation.get(), raw_offset.get(),
                    pin_offset.get(), pin_module.get(), net_pin_start.get(), net_weight.get(), arrays, n,
                    best_order.get(), options.improvement_epsilon, decided[in].get(), decided[in ^ 1].get(),
                    value_before.get(), value_after.get(), Rounds{});
                checkCuda(cudaGetLastError(), "speculativeValuesKernel launch");
            }
            best_order.download(best, stream.get());
            decided[in ^ 1].download(assumed, stream.get());
            value_before.download(before, stream.get());
            value_after.download(after, stream.get());
            checkCuda(cudaStreamSynchronize(stream.get()), "windowOrdersKernel");
        }

        // The device's windows in order (:649-677), then the host's (:680-688).
        std::fill(divergent.begin(), divergent.end(), 0);
        double wx[kWindow];
        double wy[kWindow];
        for (std::size_t j = 0; j < count; ++j) {
            const std::size_t k = on_device[j];
            ++result.evaluated_windows;
            result.evaluated_permutations += kOrders;
            const int order_index = best[j];
            if (order_index <= 0 || order_index >= kOrders) continue;
            const int32_t* m = &windows.modules[k * kWindow];
            const int32_t* window_nets_k = &windows.nets[windows.net_start[k]];
            const int net_count = static_cast<int>(windows.net_start[k + 1] - windows.net_start[k]);
            int order[kWindow];
            orderOf(order_index, order);
            const int r = windows.row[k];
            // The device's values rest on the assumed decisions of the earlier
            // windows; they are exact unless one whose cells sit on these nets
            // decided otherwise.
            double value_now = before[j];
            double value_then = after[j];
            bool stale = false;
            for (int e = 0; e < net_count && !stale; ++e) stale = divergent[window_nets_k[e]] != 0;
            if (stale) {
                for (int i = 0; i < kWindow; ++i) {
                    wx[i] = s.cx[m[i]];
                    wy[i] = s.cy[m[i]];
                }
                value_now = s.windowHpwl(m, kWindow, window_nets_k, net_count, wx, wy);
                s.centersForOrder(m, order, kWindow, d.row_bottom[r], d.row_site_spacing[r], wx, wy);
                value_then = s.windowHpwl(m, kWindow, window_nets_k, net_count, wx, wy);
            }
            const bool accept = value_then < value_now - options.improvement_epsilon;
            if (accept) {
                s.applyOrder(m, order, kWindow, d.row_bottom[r], d.row_site_spacing[r], rowOrientation(r));
                ++result.accepted_operations;
            }
            if (accept != (assumed[j] != 0)) {
                for (int e = 0; e < net_count; ++e) divergent[window_nets_k[e]] = 1;
            }
        }
        // The host-rule windows: evaluated on the device the same speculative
        // way, from the placement the four-cell windows left.
        tail_result.assign(tails, -1);
        tail_assumed.assign(tails, -1);
        if (tails > 0) {
            for (std::size_t m = 0; m < modules; ++m) {
                host_center[m] = make_double2(s.cx[m], s.cy[m]);
                host_orientation_now[m] = static_cast<int8_t>(s.orientation[m]);
            }
            center.upload(host_center, stream.get());
            orientation_now.upload(host_orientation_now, stream.get());
            tail_modules.upload(tail_host_modules, stream.get());
            tail_count.upload(tail_host_count, stream.get());
            tail_start.upload(tail_host_start, stream.get());
            tail_bottom.upload(tail_host_bottom, stream.get());
            tail_spacing.upload(tail_host_spacing, stream.get());
            tail_net_start.upload(tail_host_net_start, stream.get());
            window_nets.upload(tail_host_nets, stream.get());
            checkCuda(cudaMemsetAsync(tail_decided[0].get(), 0xFF, tails, stream.get()), "tail orders");
            const TailArrays tail{tail_modules.get(), tail_count.get(), tail_start.get(), tail_bottom.get(),
                                  tail_spacing.get(), tail_net_start.get(), window_nets.get()};
            const int n = static_cast<int>(tails);
            const unsigned blocks = static_cast<unsigned>((tails + 255) / 256);
            const unsigned warp_blocks = static_cast<unsigned>((tails + kWindowsPerBlock - 1) / kWindowsPerBlock);
            int in = 0;
            for (int iteration = 0; iteration < kSpeculations; ++iteration, in ^= 1) {
                if (iteration > 0) {
                    tailPlacementKernel<<<blocks, 256, 0, stream.get()>>>(tail, n, size.get(), tail_decided[in].get(),
                                                                         moved_center.get(), Rounds{});
                    checkCuda(cudaGetLastError(), "tailPlacementKernel launch");
                }
                tailOrdersKernel<<<warp_blocks, 32 * kWindowsPerBlock, 0, stream.get()>>>(
                    center.get(), orientation_now.get(), moved_center.get(), owner.get(), static_cast<int>(count),
                    moved_orientation.get(), raw_offset.get(), size.get(), pin_module.get(), net_pin_start.get(),
                    net_weight.get(), tail, n, nullptr, options.improvement_epsilon, tail_decided[in].get(),
                    tail_decided[in ^ 1].get(), Rounds{});
                checkCuda(cudaGetLastError(), "tailOrdersKernel launch");
            }
            tail_decided[in].download(tail_result, stream.get());
            tail_decided[in ^ 1].download(tail_assumed, stream.get());
            checkCuda(cudaStreamSynchronize(stream.get()), "tailOrdersKernel");
        }
        std::fill(divergent.begin(), divergent.end(), 0);
        for (std::size_t k = 0; k < total; ++k) {
            if (windows.device[k] != 0) continue;
            ++result.evaluated_windows;
            const int t = tail_of_window[k];
            if (t < 0) continue;  // no nets, or one above the degree limit: nothing to evaluate
            // optimizeCpuWindow (:328-354).
            const int32_t* m = &windows.modules[k * kWindow];
            const int n = windows.count[k];
            const int32_t* window_nets_k = &windows.nets[windows.net_start[k]];
            const int net_count = static_cast<int>(windows.net_start[k + 1] - windows.net_start[k]);
            const int r = windows.row[k];
            result.evaluated_permutations += static_cast<uint64_t>(factorialOf(n));
            bool stale = false;
            for (int e = 0; e < net_count && !stale; ++e) stale = divergent[window_nets_k[e]] != 0;
            int taken = tail_result[t];
            if (stale) {
                for (int i = 0; i < n; ++i) {
                    wx[i] = s.cx[m[i]];
                    wy[i] = s.cy[m[i]];
                }
                double best_value = s.windowHpwl(m, n, window_nets_k, net_count, wx, wy);
                taken = -1;
                for (int candidate = 0; candidate < factorialOf(n); ++candidate) {
                    int order[kWindow];
                    orderOf(candidate, order, n);
                    s.centersForOrder(m, order, n, d.row_bottom[r], d.row_site_spacing[r], wx, wy);
                    const double value = s.windowHpwl(m, n, window_nets_k, net_count, wx, wy);
                    if (value < best_value - options.improvement_epsilon) {
                        best_value = value;
                        taken = candidate;
                    }
                }
            }
            if (taken >= 0) {
                int order[kWindow];
                orderOf(taken, order, n);
                s.applyOrder(m, order, n, d.row_bottom[r], d.row_site_spacing[r], rowOrientation(r));
                ++result.accepted_operations;
            }
            if (taken != tail_assumed[t]) {
                for (int e = 0; e < net_count; ++e) divergent[window_nets_k[e]] = 1;
            }
        }
        result.completed_passes = pass + 1;
    }
    result.hpwl_after = s.hpwl(workers);
    result.elapsed_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - started).count();
    std::copy(s.cx.begin(), s.cx.end(), module_x);
    std::copy(s.cy.begin(), s.cy.end(), module_y);
    if (module_orientation != nullptr) std::copy(s.orientation.begin(), s.orientation.end(), module_orientation);
    return true;
}

}  // namespace mpgp
