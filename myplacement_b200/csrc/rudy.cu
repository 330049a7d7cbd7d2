// RUDY routing-demand map, hotspot penalty and its subgradient on the device.
//
// Restates evaluateRudy (Rudy.cpp:227-456) for the adaptive controller's
// routability term (AdaptiveGlobalPlacer.cpp:149-172, 201-331).  A net's
// rectangle-overlap demand is separable: the overlap of its (expanded, clipped)
// box with bin (c, r) is ox(c) * oy(r), where ox is a partial width in the box's
// first and last columns and the bin width in between, and the same along y.
// So a net's demand is at most 3 x 3 constant blocks, and the passes are:
//   deposit   one thread per two-pin net, G lanes per larger one: the pin box,
//             expanded to minimum_span_in_bins where a net is thinner
//             (calculateNetBox, Rudy.cpp:120-152), each block's horizontal demand
//             w * overlap / y_span and vertical demand w * overlap / x_span
//             quantized to int64 (units of bin_w * 2^-32 and bin_h * 2^-32) and
//             added at the block's corners of a 2-D difference array with integer
//             atomics, neighbouring blocks' corners combined: at most 32 atomics a
//             net instead of two per covered bin, in a shared-memory copy of the
//             arrays where that pays, and the maps stay bit-exact.  Bound by the
//             issue of its FP64 and address arithmetic: 220,000 nets on 64 x 64
//             bins took 241 us with 72 global atomics a net and a thread per net,
//             52 us now (B200, cold).
//   prefix    two scans (rows, then columns) turn the difference arrays into the
//             demand maps and clear them.
//   metrics   one thread per bin: utilisation against the frozen capacities,
//             the penalty model (hinge L2 / softplus L2 / hinge L4,
//             evaluatePenalty Rudy.cpp:83-100), its adjoint, the energy, the
//             proxy overflow, the maximum utilisation and the demand totals
//             (FP64 block partials, reduced in a fixed order).
//   tables    two scans build summed-area tables of the two adjoints.
//   gradient  G >= 2 lanes per net, an axis of the box per lane: the Clarke
//             subgradient with respect to the four box edges (Rudy.cpp:320-400);
//             the same nets 142 us with a thread per net, 113 us now.  Four lanes
//             per net with an edge each took 157 us: each repeated the box's
//             set-up.  An edge's term only involves
//             the one or two columns (rows) its derivative is non-zero in, and
//             the span terms a box-weighted adjoint sum: with the tables each is
//             O(1), not O(box area).  The edge gradients are split over the pins
//             on each extremal edge (Rudy.cpp:402-452) and written to the pins'
//             particle-ordered slots for the gather.
// Arithmetic is FP64; interior bins take the bin width and height as their
// overlap, which the reference's per-bin differences reproduce to the last bit
// or one unit in it.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "kernels.cuh"

namespace mpgp {
namespace {

struct Box {
    double left, right, bottom, top;
    double raw_left, raw_right, raw_bottom, raw_top;
    double x_span, y_span;
    bool x_physical, y_physical;
};

__device__ __forceinline__ double2 pinPosition(const RudyArgs& a, int pin) {
    const int particle = a.pin_particle[pin];
    if (particle >= 0) {
        const double2 c = a.positions[particle];
        const float2 o = a.pin_offset[pin];
        return make_double2(c.x + static_cast<double>(o.x), c.y + static_cast<double>(o.y));
    }
    return a.static_pins[-particle - 1];
}

// The box of pins whose extremes are given (calculateNetBox, Rudy.cpp:120-152).
__device__ __forceinline__ Box boxOf(const RudyArgs& a, double left, double right, double bottom, double top) {
    Box b;
    b.left = left;
    b.right = right;
    b.bottom = bottom;
    b.top = top;
    const double raw_x_span = b.right - b.left;
    const double raw_y_span = b.top - b.bottom;
    b.raw_left = b.left;
    b.raw_right = b.right;
    b.raw_bottom = b.bottom;
    b.raw_top = b.top;
    b.x_physical = true;
    b.y_physical = true;
    if (raw_x_span < a.minimum_x_span) {
        const double center = (b.left + b.right) * 0.5;
        b.left = center - a.minimum_x_span * 0.5;
        b.right = center + a.minimum_x_span * 0.5;
        b.x_physical = false;
    }
    if (raw_y_span < a.minimum_y_span) {
        const double center = (b.bottom + b.top) * 0.5;
        b.bottom = center - a.minimum_y_span * 0.5;
        b.top = center + a.minimum_y_span * 0.5;
        b.y_physical = false;
    }
    b.x_span = fmax(b.right - b.left, kEpsilon);
    b.y_span = fmax(b.top - b.bottom, kEpsilon);
    return b;
}

__device__ __forceinline__ int startBin(double coordinate, double lower, double length, int count) {
    return max(0, min(count - 1, static_cast<int>(floor((coordinate - lower) / length))));
}

__device__ __forceinline__ int endBin(double coordinate, double lower, double length, int count) {
    return max(0, min(count - 1, static_cast<int>(ceil((coordinate - lower) / length) - 1.0)));
}

__device__ __forceinline__ double overlapLength(double lower_a, double upper_a, double lower_b, double upper_b) {
    return fmax(0.0, fmin(upper_a, upper_b) - fmax(lower_a, lower_b));
}

__device__ __forceinline__ bool approximatelyEqual(double left, double right) {
    return fabs(left - right) <= 1e-10 * fmax(1.0, fmax(fabs(left), fabs(right)));
}

__device__ __forceinline__ double upperDerivative(double upper, double bin_lower, double bin_upper, double overlap) {
    if (upper > bin_lower + kEpsilon && upper < bin_upper - kEpsilon && overlap > kEpsilon) return 1.0;
    if (approximatelyEqual(upper, bin_lower) || approximatelyEqual(upper, bin_upper)) return 0.5;
    return 0.0;
}

__device__ __forceinline__ double lowerDerivative(double lower, double bin_lower, double bin_upper, double overlap) {
    if (lower > bin_lower + kEpsilon && lower < bin_upper - kEpsilon && overlap > kEpsilon) return -1.0;
    if (approximatelyEqual(lower, bin_lower) || approximatelyEqual(lower, bin_upper)) return -0.5;
    return 0.0;
}

__device__ __forceinline__ bool onInteriorGridLine(double coordinate, double lower, double length, int count) {
    const double relative = (coordinate - lower) / length;
    const double nearest = round(relative);
    return nearest > 0.0 && nearest < static_cast<double>(count) && approximatelyEqual(relative, nearest);
}

// Whether the net counts (two or more pins, positive weight) and its clipped box has area.
__device__ __forceinline__ bool clippedRange(const RudyArgs& a, const Box& b, int& c0, int& c1, int& r0, int& r1) {
    const double cl = fmax(b.left, a.llx), cr = fmin(b.right, a.urx);
    const double cb = fmax(b.bottom, a.lly), ct = fmin(b.top, a.ury);
    if (fmax(0.0, cr - cl) * fmax(0.0, ct - cb) <= kEpsilon) return false;
    c0 = startBin(cl, a.llx, a.bin_w, a.columns);
    c1 = endBin(cr, a.llx, a.bin_w, a.columns);
    r0 = startBin(cb, a.lly, a.bin_h, a.rows);
    r1 = endBin(ct, a.lly, a.bin_h, a.rows);
    return true;
}

// The parts of a clipped box along one axis, in three fixed slots: the first cell (partial),
// the interior cells (full), the last cell (partial); an absent part has overlap zero.  Part i
// covers cells [bound[i], bound[i + 1]).
struct AxisParts {
    int bound[4];
    double overlap[3];
};

__device__ __forceinline__ AxisParts axisParts(double lower, double upper, double origin, double length, int first,
                                               int last) {
    AxisParts p;
    const auto cell = [&](int i) {
        const double begin = origin + static_cast<double>(i) * length;
        return overlapLength(lower, upper, begin, begin + length);
    };
    const bool several = last > first;
    p.bound[0] = first;
    p.bound[1] = first + 1;
    p.bound[2] = several ? last : first + 1;
    p.bound[3] = last + 1;
    p.overlap[0] = cell(first);
    p.overlap[1] = last > first + 1 ? length : 0.0;
    p.overlap[2] = several ? cell(last) : 0.0;
    return p;
}

// A net's extremes over G lanes, a pin per lane (in a loop for nets of more than G pins; the
// 32-lane form only).  Every lane of the group returns them.
struct Extremes {
    double left = DBL_MAX, right = -DBL_MAX, bottom = DBL_MAX, top = -DBL_MAX;
    __device__ __forceinline__ void add(double2 p) {
        left = fmin(left, p.x);
        right = fmax(right, p.x);
        bottom = fmin(bottom, p.y);
        top = fmax(top, p.y);
    }
};

template <int G>
__device__ __forceinline__ Extremes groupExtremes(Extremes e) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        e.left = fmin(e.left, __shfl_xor_sync(0xffffffffu, e.left, o, G));
        e.right = fmax(e.right, __shfl_xor_sync(0xffffffffu, e.right, o, G));
        e.bottom = fmin(e.bottom, __shfl_xor_sync(0xffffffffu, e.bottom, o, G));
        e.top = fmax(e.top, __shfl_xor_sync(0xffffffffu, e.top, o, G));
    }
    return e;
}

// Adds a net's demand to one of the two difference arrays: q[i][j], the quantized demand of
// the block of row part i and column part j, at the block's four corners.  Neighbouring blocks
// share corners, so their terms are combined: at most sixteen adds a map (four row bounds
// times four column bounds) instead of thirty-six.  Handles row bounds first .. last - 1.
// `density` is the demand of a unit of area in the map's units: weight / span of the box.
template <class Add>
__device__ __forceinline__ void addDemand(const AxisParts& rows, const AxisParts& cols, double density, int first,
                                          int last, const Add& add) {
    const auto row = [&](int i, long long (&q)[3]) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            q[j] = 0;
            if (i < 0 || i > 2) continue;
            const double overlap_y = i == 0 ? rows.overlap[0] : i == 1 ? rows.overlap[1] : rows.overlap[2];
            const double overlap = cols.overlap[j] * overlap_y;
            if (overlap_y <= kEpsilon || overlap <= kEpsilon) continue;
            q[j] = __double2ll_rn(overlap * density);
        }
    };
    long long above[3];
    row(first - 1, above);
    for (int k = first; k < last; ++k) {
        long long here[3];
        row(k, here);
        const int bound = k == 0 ? rows.bound[0] : k == 1 ? rows.bound[1] : k == 2 ? rows.bound[2] : rows.bound[3];
        const long long d0 = here[0] - above[0], d1 = here[1] - above[1], d2 = here[2] - above[2];
        if (d0 != 0) add(bound, cols.bound[0], d0);
        if (d1 != d0) add(bound, cols.bound[1], d1 - d0);
        if (d2 != d1) add(bound, cols.bound[2], d2 - d1);
        if (d2 != 0) add(bound, cols.bound[3], -d2);
#pragma unroll
        for (int j = 0; j < 3; ++j) above[j] = here[j];
    }
}

// Nets [first, first + count) on the calling sub-block of 256 threads (thread `t`, warp
// `t / 32`): one thread per two-pin net, G lanes per net of degree <= G, a warp per larger net.
template <int G, class Adder>
__device__ __forceinline__ void depositNets(const RudyArgs& a, int first, int count, int t, const Adder& adder) {
    const int lane = t & 31;
    const int sub = lane % G;
    constexpr int kPerWarp = 32 / G;
    constexpr int kWarps = kThreads / 32;
    for (int base = (t >> 5) * kPerWarp; base < count; base += kWarps * kPerWarp) {
        const int local = base + lane / G;
        const bool net_ok = local < count;
        const int net = first + (net_ok ? local : 0);
        const int begin = a.net_start[net];
        const int end = a.net_start[net + 1];
        const double weight = a.net_weight[net];
        Extremes e;
        if constexpr (G == 1) {
            for (int pin = begin; pin < end; ++pin) e.add(pinPosition(a, pin));
        } else {
            for (int pin = begin + sub; pin < end; pin += G) e.add(pinPosition(a, pin));
            e = groupExtremes<G>(e);
        }
        if (!net_ok || end - begin < 2 || weight <= 0.0) continue;
        const Box b = boxOf(a, e.left, e.right, e.bottom, e.top);
        int c0, c1, r0, r1;
        if (!clippedRange(a, b, c0, c1, r0, r1)) continue;
        const AxisParts cols = axisParts(b.left, b.right, a.llx, a.bin_w, c0, c1);
        const AxisParts rows = axisParts(b.bottom, b.top, a.lly, a.bin_h, r0, r1);
        if constexpr (G == 1) {
            addDemand(rows, cols, weight / b.y_span * a.inv_unit_h, 0, 4,
                      [&](int r, int c, long long q) { adder(0, r, c, q); });
            addDemand(rows, cols, weight / b.x_span * a.inv_unit_v, 0, 4,
                      [&](int r, int c, long long q) { adder(1, r, c, q); });
        } else if (sub < 4) {
            // Four lanes: each one map and two of its row bounds.
            const int map = sub & 1;
            const int half = sub & 2;
            addDemand(rows, cols, weight / (map == 0 ? b.y_span : b.x_span) * (map == 0 ? a.inv_unit_h : a.inv_unit_v),
                      half, half + 2, [&](int r, int c, long long q) { adder(map, r, c, q); });
        }
    }
}

// The wirelength pass's work items ({lanes per net, first net, nets}, RudyArgs::work), a
// sub-block of 256 threads each.
template <class Adder>
__device__ __forceinline__ void depositItems(const RudyArgs& a, const Adder& adder) {
    const int t = static_cast<int>(threadIdx.x) % kThreads;
    const int sub_blocks = static_cast<int>(blockDim.x) / kThreads;
    const int stride = static_cast<int>(gridDim.x) * sub_blocks;
    for (int item = static_cast<int>(blockIdx.x) * sub_blocks + static_cast<int>(threadIdx.x) / kThreads;
         item < a.work_count; item += stride) {
        const int4 work = a.work[item];
        switch (work.x) {
            case 1: depositNets<1>(a, work.y, work.z, t, adder); break;
            case 4: depositNets<4>(a, work.y, work.z, t, adder); break;
            case 8: depositNets<8>(a, work.y, work.z, t, adder); break;
            case 16: depositNets<16>(a, work.y, work.z, t, adder); break;
            default: depositNets<32>(a, work.y, work.z, t, adder); break;
        }
    }
}

// Straight to the difference arrays with global atomics.
__global__ void __launch_bounds__(kThreads) rudyDepositKernel(RudyArgs a) {
    releaseNext();
    waitForPrior();
    const int stride = a.columns + 1;
    const size_t map_cells = static_cast<size_t>(a.rows + 1) * stride;
    depositItems(a, [&](int map, int r, int c, long long q) {
        atomicAdd(a.diff + map * map_cells + static_cast<size_t>(r) * stride + c, static_cast<unsigned long long>(q));
    });
}

constexpr int kDepositThreads = 1024;

// Through a copy of both difference arrays in shared memory, one block per SM: a value is kept
// as two 32-bit words, each added with a native shared atomic (the low word's carry goes to the
// high one), and the block's non-zero values are added to the global arrays at its end,
// neighbouring threads at neighbouring cells.  The sums are integers: the maps are the same.
__global__ void __launch_bounds__(kDepositThreads, 1) rudyDepositSharedKernel(RudyArgs a) {
    extern __shared__ unsigned int words[];
    releaseNext();
    const int stride = a.columns + 1;
    const int map_cells = (a.rows + 1) * stride;
    const int cells = 2 * map_cells;
    unsigned int* low = words;
    unsigned int* high = words + cells;
    for (int k = threadIdx.x; k < 2 * cells; k += blockDim.x) words[k] = 0u;
    waitForPrior();
    __syncthreads();
    depositItems(a, [&](int map, int r, int c, long long q) {
        const int k = map * map_cells + r * stride + c;
        const unsigned int q_low = static_cast<unsigned int>(q);
        unsigned int q_high = static_cast<unsigned int>(static_cast<unsigned long long>(q) >> 32);
        const unsigned int before = atomicAdd(low + k, q_low);
        if (before + q_low < before) ++q_high;
        if (q_high != 0u) atomicAdd(high + k, q_high);
    });
    __syncthreads();
    for (int k = threadIdx.x; k < cells; k += blockDim.x) {
        const unsigned long long q = static_cast<unsigned long long>(low[k]) |
                                     (static_cast<unsigned long long>(high[k]) << 32);
        if (q != 0ULL) atomicAdd(a.diff + k, q);
    }
}

// Inclusive scan of `length` values (load(i) / store(i, v)) by the whole block,
// in chunks of blockDim.x, always in index order (the sums are deterministic).
template <typename T, class Load, class Store>
__device__ void scanLine(int length, Load load, Store store) {
    __shared__ T warp_sums[32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5;
    T carry = T(0);
    for (int base = 0; base < length; base += blockDim.x) {
        const int i = base + static_cast<int>(threadIdx.x);
        T v = i < length ? load(i) : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) warp_sums[warp] = v;
        __syncthreads();
        if (warp == 0) {
            T w = lane < warps ? warp_sums[lane] : T(0);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const T u = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += u;
            }
            if (lane < warps) warp_sums[lane] = w;
        }
        __syncthreads();
        const T before = warp > 0 ? warp_sums[warp - 1] : T(0);
        if (i < length) store(i, carry + before + v);
        carry += warp_sums[warps - 1];
        __syncthreads();
    }
}

// Difference arrays -> demand maps.  Pass 0 scans each row of both arrays in
// place; pass 1 scans each column, writes the map and clears the array.
__global__ void __launch_bounds__(kThreads) rudyPrefixKernel(RudyArgs a, int pass) {
    releaseNext();
    waitForPrior();
    const int stride = a.columns + 1;
    unsigned long long* diff = a.diff + static_cast<size_t>(blockIdx.y) * (a.rows + 1) * stride;
    unsigned long long* map = blockIdx.y == 0 ? a.horizontal : a.vertical;
    if (pass == 0) {
        unsigned long long* row = diff + static_cast<size_t>(blockIdx.x) * stride;
        scanLine<unsigned long long>(
            stride, [&](int i) { return row[i]; }, [&](int i, unsigned long long v) { row[i] = v; });
    } else {
        const int c = blockIdx.x;
        scanLine<unsigned long long>(
            a.rows + 1,
            [&](int i) {
                const unsigned long long v = diff[static_cast<size_t>(i) * stride + c];
                diff[static_cast<size_t>(i) * stride + c] = 0ULL;
                return v;
            },
            [&](int i, unsigned long long v) {
                if (i < a.rows && c < a.columns) map[static_cast<size_t>(i) * a.columns + c] = v;
            });
    }
}

// Summed-area tables of the two adjoints: table[(r + 1) * (columns + 1) + c + 1]
// = sum over r' <= r, c' <= c (row 0 and column 0 stay zero).
__global__ void __launch_bounds__(kThreads) rudyTableKernel(RudyArgs a, int pass) {
    releaseNext();
    waitForPrior();
    const int stride = a.columns + 1;
    double* table = a.table + static_cast<size_t>(blockIdx.y) * (a.rows + 1) * stride;
    const double* adjoint = blockIdx.y == 0 ? a.adjoint_h : a.adjoint_v;
    if (pass == 0) {
        const int r = blockIdx.x;
        const double* in = adjoint + static_cast<size_t>(r) * a.columns;
        double* out = table + static_cast<size_t>(r + 1) * stride + 1;
        scanLine<double>(a.columns, [&](int i) { return in[i]; }, [&](int i, double v) { out[i] = v; });
    } else {
        const int c = blockIdx.x + 1;
        scanLine<double>(
            a.rows, [&](int i) { return table[static_cast<size_t>(i + 1) * stride + c]; },
            [&](int i, double v) { table[static_cast<size_t>(i + 1) * stride + c] = v; });
    }
}

// evaluatePenalty (Rudy.cpp:83-100): value and derivative of the model at utilisation u.
__device__ __forceinline__ double2 penalty(double u, int model, double temperature) {
    const double overflow = fmax(0.0, u - 1.0);
    if (model == MPGP_RUDY_HINGE_L2) return make_double2(0.5 * overflow * overflow, overflow);
    if (model == MPGP_RUDY_HINGE_L4) {
        const double square = overflow * overflow;
        return make_double2(0.25 * square * square, overflow * square);
    }
    if (model == MPGP_RUDY_SOFTPLUS_L2) {
        const double t = fmax(temperature, kEpsilon);
        const double scaled = (u - 1.0) / t;
        const double softplus = scaled > 30.0 ? scaled : (scaled < -30.0 ? exp(scaled) : log1p(exp(scaled)));
        double sigmoid;
        if (scaled >= 0.0) {
            sigmoid = 1.0 / (1.0 + exp(-scaled));
        } else {
            const double e = exp(scaled);
            sigmoid = e / (1.0 + e);
        }
        const double softened = t * softplus;
        return make_double2(0.5 * softened * softened, softened * sigmoid);
    }
    return make_double2(0.0, 0.0);
}

__global__ void __launch_bounds__(kThreads) rudyMetricsKernel(RudyArgs a) {
    releaseNext();
    waitForPrior();
    const int bins = a.columns * a.rows;
    const double unit_h = 1.0 / a.inv_unit_h, unit_v = 1.0 / a.inv_unit_v;
    const bool with_capacity = a.capacity_h > 0.0 && a.capacity_v > 0.0;
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // energy, H total, V total, proxy overflow, max utilisation
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < bins; b += gridDim.x * blockDim.x) {
        const double h = static_cast<double>(static_cast<long long>(a.horizontal[b])) * unit_h;
        const double w = static_cast<double>(static_cast<long long>(a.vertical[b])) * unit_v;
        v[1] += h;
        v[2] += w;
        if (!with_capacity) continue;
        const double uh = h / a.capacity_h;
        const double uv = w / a.capacity_v;
        const double2 ph = penalty(uh, a.model, a.temperature);
        const double2 pv = penalty(uv, a.model, a.temperature);
        v[0] += (ph.x + pv.x) / static_cast<double>(bins);
        a.adjoint_h[b] = ph.y / (static_cast<double>(bins) * a.capacity_h);
        a.adjoint_v[b] = pv.y / (static_cast<double>(bins) * a.capacity_v);
        v[3] += fmax(0.0, uh - 1.0) + fmax(0.0, uv - 1.0);
        const double u = fmax(uh, uv);
        v[4] = fmax(v[4], u);
        if (a.utilization != nullptr) a.utilization[b] = u;
    }
    const bool is_max[5] = {false, false, false, false, true};
    blockReduce<5>(v, is_max);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 5; ++k) a.partials[k * gridDim.x + blockIdx.x] = v[k];
    }
}

// The subgradient of nets [first, first + count), G >= 2 lanes per net.  The lanes share the
// pins; even lanes take the box's x axis (its left and right edges), odd lanes its y axis, and
// an axis' cells and overlaps go to the other axis by shuffles, so that no lane forms both.
template <int G>
__device__ __forceinline__ void gradientNets(const RudyArgs& a, int first, int count) {
    constexpr unsigned int kAll = 0xffffffffu;
    constexpr unsigned int kGroup = G == 32 ? kAll : (1u << G) - 1u;
    constexpr int kPerWarp = 32 / G;
    constexpr int kWarps = kThreads / 32;
    const int lane = threadIdx.x & 31;
    const int sub = lane % G;
    const int base_lane = lane - sub;
    const bool along_x = (sub & 1) == 0;
    const int stride = a.columns + 1;
    const double origin = along_x ? a.llx : a.lly;
    const double limit = along_x ? a.urx : a.ury;
    const double length = along_x ? a.bin_w : a.bin_h;
    const double minimum_span = along_x ? a.minimum_x_span : a.minimum_y_span;
    const int cells = along_x ? a.columns : a.rows;
    const int step = along_x ? 1 : stride;        // table step along the axis
    const int cross_step = along_x ? stride : 1;  // and across it
    const double* table_h = a.table;
    const double* table_v = a.table + static_cast<size_t>(a.rows + 1) * stride;
    for (int base = (threadIdx.x >> 5) * kPerWarp; base < count; base += kWarps * kPerWarp) {
        const int local = base + lane / G;
        const bool net_ok = local < count;
        const int net = first + (net_ok ? local : 0);
        const int begin = a.net_start[net];
        const int end = a.net_start[net + 1];
        const double weight = a.net_weight[net];
        Extremes e;
        double2 own = make_double2(0.0, 0.0);  // this lane's first pin
        for (int pin = begin + sub; pin < end; pin += G) {
            const double2 p = pinPosition(a, pin);
            if (pin == begin + sub) own = p;
            e.add(p);
        }
        e = groupExtremes<G>(e);
        // The axis of calculateNetBox (boxOf) and of clippedRange.
        const double raw_low = along_x ? e.left : e.bottom, raw_high = along_x ? e.right : e.top;
        double low = raw_low, high = raw_high;
        const bool physical = !(high - low < minimum_span);
        if (!physical) {
            const double center = (raw_low + raw_high) * 0.5;
            low = center - minimum_span * 0.5;
            high = center + minimum_span * 0.5;
        }
        const double span = fmax(high - low, kEpsilon);
        const double clip_low = fmax(low, origin), clip_high = fmin(high, limit);
        const double extent = fmax(0.0, clip_high - clip_low);
        const double cross_extent = __shfl_xor_sync(kAll, extent, 1);
        const bool counted = net_ok && end - begin >= 2 && weight > 0.0 && extent * cross_extent > kEpsilon;
        const int first_cell = startBin(clip_low, origin, length, cells);
        const int last_cell = endBin(clip_high, origin, length, cells);
        const AxisParts parts = axisParts(low, high, origin, length, first_cell, last_cell);
        AxisParts cross;
        {
            const int cross_first = __shfl_xor_sync(kAll, first_cell, 1);
            const int cross_last = __shfl_xor_sync(kAll, last_cell, 1);
            cross.bound[0] = cross_first;
            cross.bound[1] = cross_first + 1;
            cross.bound[2] = cross_last > cross_first ? cross_last : cross_first + 1;
            cross.bound[3] = cross_last + 1;
#pragma unroll
            for (int i = 0; i < 3; ++i) cross.overlap[i] = __shfl_xor_sync(kAll, parts.overlap[i], 1);
        }
        const double inv_span = 1.0 / span;
        const double cross_inv_span = __shfl_xor_sync(kAll, inv_span, 1);
        const double inv_x_span = along_x ? inv_span : cross_inv_span;
        const double inv_y_span = along_x ? cross_inv_span : inv_span;
        // Edge terms (Rudy.cpp:360-400): the cells next to an edge are the only ones whose
        // derivative can be non-zero; each adds d * (adj_h / y_span + adj_v / x_span) weighted
        // by the other axis' overlaps.
        double gradient_low = 0.0, gradient_high = 0.0;
        if (counted && sub < 2) {
            // Sum over the cross parts of overlap * (the adjoint summed over the part) at cell u;
            // a part's four table entries are added in the order of rows, then columns.
            const auto line_sum = [&](const double* t, int u) {
                const double* near_line = t + static_cast<size_t>(u) * step;
                const double* far_line = near_line + step;
                double sum = 0.0;
                double near_from = near_line[cross.bound[0] * cross_step], far_from = far_line[cross.bound[0] * cross_step];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const double near_to = near_line[cross.bound[i + 1] * cross_step];
                    const double far_to = far_line[cross.bound[i + 1] * cross_step];
                    const double second = along_x ? far_from : near_to;
                    const double third = along_x ? near_to : far_from;
                    if (cross.overlap[i] != 0.0) sum += cross.overlap[i] * (far_to - second - third + near_from);
                    near_from = near_to;
                    far_from = far_to;
                }
                return sum;
            };
            const auto cell_sum = [&](int u) { return line_sum(table_h, u) * inv_y_span + line_sum(table_v, u) * inv_x_span; };
            double edge_sum[2];
#pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                const bool lower = side == 0;
                const double edge = lower ? low : high;
                const int own_cell = lower ? first_cell : last_cell;
                const double cell_low = origin + static_cast<double>(own_cell) * length;
                const double cell_high = cell_low + length;
                // The tolerances of the two derivatives (kEpsilon, and 1e-10 relative), with room.
                const double margin = 2.0 * kEpsilon + 2e-10 * (fabs(cell_low) + fabs(cell_high) + 1.0);
                double sum = 0.0;
                if (edge - cell_low > margin && cell_high - edge > margin) {
                    // Inside its cell, away from the grid lines (nearly every edge): the derivative
                    // is one there and zero in the neighbours.
                    const double overlap = overlapLength(low, high, cell_low, cell_high);
                    if (overlap > kEpsilon) sum = cell_sum(own_cell);
                    if (lower) sum = -sum;
                } else {
                    const int g0 = max(0, first_cell - (onInteriorGridLine(low, origin, length, cells) ? 1 : 0));
                    const int g1 = min(cells - 1, last_cell + (onInteriorGridLine(high, origin, length, cells) ? 1 : 0));
                    const int near = static_cast<int>(floor((edge - origin) / length));
                    for (int u = max(g0, near - 1); u <= min(g1, near + 1); ++u) {
                        const double bin_low = origin + static_cast<double>(u) * length;
                        const double bin_high = bin_low + length;
                        const double overlap = overlapLength(low, high, bin_low, bin_high);
                        const double d = lower ? lowerDerivative(edge, bin_low, bin_high, overlap)
                                               : upperDerivative(edge, bin_low, bin_high, overlap);
                        if (d != 0.0) sum += d * cell_sum(u);
                    }
                }
                edge_sum[side] = weight * sum;
            }
            gradient_low = edge_sum[0];
            gradient_high = edge_sum[1];
            if (physical) {
                // The span term: the adjoint weighted by the box's overlaps with every bin.
                const double* t = along_x ? table_v : table_h;
                double box = 0.0;
                double from[4], to[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) from[j] = t[cross.bound[0] * cross_step + parts.bound[j] * step];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) to[j] = t[cross.bound[i + 1] * cross_step + parts.bound[j] * step];
                    if (cross.overlap[i] != 0.0) {
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            box += cross.overlap[i] * parts.overlap[j] * ((to[j + 1] - from[j + 1]) - (to[j] - from[j]));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) from[j] = to[j];
                }
                const double term = weight * box * inv_span * inv_span;
                gradient_low += term;
                gradient_high -= term;
            }
        }
        // The edge gradients split over the pins on each extremal edge (Rudy.cpp:402-452).  A
        // widened axis (not physical) gives half of both to the pins of either raw edge.
        if (!physical) gradient_low = gradient_high = 0.5 * (gradient_low + gradient_high);
        const double at_low = physical ? low : raw_low, at_high = physical ? high : raw_high;
        const double cross_at_low = __shfl_xor_sync(kAll, at_low, 1), cross_at_high = __shfl_xor_sync(kAll, at_high, 1);
        const double at_left = along_x ? at_low : cross_at_low, at_right = along_x ? at_high : cross_at_high;
        const double at_bottom = along_x ? cross_at_low : at_low, at_top = along_x ? cross_at_high : at_high;
        const double g_left = __shfl_sync(kAll, gradient_low, base_lane);
        const double g_right = __shfl_sync(kAll, gradient_high, base_lane);
        const double g_bottom = __shfl_sync(kAll, gradient_low, base_lane + 1);
        const double g_top = __shfl_sync(kAll, gradient_high, base_lane + 1);
        int n_left = 0, n_right = 0, n_bottom = 0, n_top = 0;
        const auto onEdges = [&](double2 p) {
            return (approximatelyEqual(p.x, at_left) ? 1 : 0) | (approximatelyEqual(p.x, at_right) ? 2 : 0) |
                   (approximatelyEqual(p.y, at_bottom) ? 4 : 0) | (approximatelyEqual(p.y, at_top) ? 8 : 0);
        };
        int own_on = 0;
        // Uniform trips: every lane of the warp takes part in the ballots.
        int trips = 1;
        if constexpr (G == 32) trips = __shfl_sync(kAll, (end - begin + G - 1) / G, 0);
        for (int k = 0; k < trips; ++k) {
            const int pin = begin + sub + k * G;
            int on = 0;
            if (counted && pin < end) on = onEdges(k == 0 ? own : pinPosition(a, pin));
            if (k == 0) own_on = on;
            n_left += __popc((__ballot_sync(kAll, on & 1) >> base_lane) & kGroup);
            n_right += __popc((__ballot_sync(kAll, on & 2) >> base_lane) & kGroup);
            n_bottom += __popc((__ballot_sync(kAll, on & 4) >> base_lane) & kGroup);
            n_top += __popc((__ballot_sync(kAll, on & 8) >> base_lane) & kGroup);
        }
        if (!net_ok) continue;
        const auto part = [](double g, int n) { return n == 1 ? g : g / static_cast<double>(n); };
        for (int pin = begin + sub; pin < end; pin += G) {
            if (a.pin_particle[pin] < 0) continue;  // fixed modules take no gradient
            double gx = 0.0, gy = 0.0;
            if (counted) {
                const int on = pin == begin + sub ? own_on : onEdges(pinPosition(a, pin));
                if (on & 1) gx += part(g_left, n_left);
                if (on & 2) gx += part(g_right, n_right);
                if (on & 4) gy += part(g_bottom, n_bottom);
                if (on & 8) gy += part(g_top, n_top);
            }
            a.pin_gradient[a.pin_slot[pin]] = make_double2(gx, gy);
        }
    }
}

// One block per work item of the wirelength pass.
__global__ void __launch_bounds__(kThreads, 3) rudyGradientKernel(RudyArgs a) {
    releaseNext();
    waitForPrior();
    const int4 work = a.work[blockIdx.x];
    switch (work.x) {
        case 1: gradientNets<2>(a, work.y, work.z); break;
        case 4: gradientNets<4>(a, work.y, work.z); break;
        case 8: gradientNets<8>(a, work.y, work.z); break;
        case 16: gradientNets<16>(a, work.y, work.z); break;
        default: gradientNets<32>(a, work.y, work.z); break;
    }
}

// The RUDY subgradient of every particle from its pins' slots (in slot order).
__global__ void __launch_bounds__(kThreads) rudyGatherKernel(const int* particle_pin_start, const double2* pin_gradient,
                                                            int movable_count, int particle_count, double2* out) {
    releaseNext();
    waitForPrior();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= particle_count) return;
    double2 sum = make_double2(0.0, 0.0);
    if (i < movable_count) {
        for (int j = particle_pin_start[i]; j < particle_pin_start[i + 1]; ++j) {
            const double2 g = pin_gradient[j];
            sum.x += g.x;
            sum.y += g.y;
        }
    }
    out[i] = sum;
}

// The deposit goes through shared memory where both difference arrays fit and the nets pay
// for the copy that every block clears and adds to the global arrays.  Measured on a B200,
// cold, shared against direct, us: 32 x 32 cells 23.9 / 19.4 for 10,500 nets, 23.6 / 27.8 for
// 21,000, 39 / 101 for 105,000; 64 x 64 25.0 / 18.8 for 21,000, 24.7 / 36.2 for 42,000;
// 110 x 110 28.3 / 18.1 for 21,000, 29.1 / 28.7 for 42,000, 43.8 / 48.1 for 105,000.  The
// crossing lies near 14,000 nets plus one per cell of the two arrays.
constexpr int kDepositSharedBytes = 200 * 1024;
constexpr int kDepositSharedNets = 14000;

void configureDeposit() {
    constexpr int kMaxDevices = 64;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attribute[kMaxDevices] = {};
    int device = 0;
    checkCuda(cudaGetDevice(&device), "Query the current device");
    require(device >= 0 && device < kMaxDevices, "Device index out of range.");
    std::call_once(once[device], [device] {
        attribute[device] = cudaFuncSetAttribute(rudyDepositSharedKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kDepositSharedBytes);
    });
    checkCuda(attribute[device], "Configure the RUDY deposit");
}

}  // namespace

void launchRudyDeposit(const RudyArgs& args, cudaStream_t stream) {
    if (args.work_count <= 0) return;
    const int cells = 2 * (args.rows + 1) * (args.columns + 1);
    const size_t bytes = static_cast<size_t>(cells) * 2 * sizeof(unsigned int);
    if (bytes <= static_cast<size_t>(kDepositSharedBytes) && args.net_count >= kDepositSharedNets + cells) {
        configureDeposit();
        constexpr int kSubBlocks = kDepositThreads / kThreads;
        const int blocks = std::min(148, ceilDiv(args.work_count, kSubBlocks));
        launchChained("Launch the RUDY deposit", rudyDepositSharedKernel, dim3(blocks), dim3(kDepositThreads), bytes,
                      stream, args);
        return;
    }
    launchChained("Launch the RUDY deposit", rudyDepositKernel, dim3(args.work_count), dim3(kThreads), 0, stream, args);
}

void launchRudyPrefix(const RudyArgs& args, cudaStream_t stream) {
    launchChained("Launch the RUDY row scan", rudyPrefixKernel, dim3(args.rows + 1, 2), dim3(kThreads), 0, stream,
                  args, 0);
    launchChained("Launch the RUDY column scan", rudyPrefixKernel, dim3(args.columns + 1, 2), dim3(kThreads), 0,
                  stream, args, 1);
}

void launchRudyTables(const RudyArgs& args, cudaStream_t stream) {
    launchChained("Launch the RUDY adjoint row scan", rudyTableKernel, dim3(args.rows, 2), dim3(kThreads), 0, stream,
                  args, 0);
    launchChained("Launch the RUDY adjoint column scan", rudyTableKernel, dim3(args.columns, 2), dim3(kThreads), 0,
                  stream, args, 1);
}

void launchRudyMetrics(const RudyArgs& args, int blocks, cudaStream_t stream) {
    launchChained("Launch the RUDY metrics", rudyMetricsKernel, dim3(blocks), dim3(kThreads), 0, stream, args);
}

void launchRudyGradient(const RudyArgs& args, cudaStream_t stream) {
    if (args.work_count <= 0) return;
    launchChained("Launch the RUDY gradient", rudyGradientKernel, dim3(args.work_count), dim3(kThreads), 0, stream,
                  args);
}

void launchRudyGather(const int* particle_pin_start, const double2* pin_gradient, int movable_count,
                      int particle_count, double2* out, cudaStream_t stream) {
    if (particle_count <= 0) return;
    launchChained("Launch the RUDY gather", rudyGatherKernel, dim3(ceilDiv(particle_count, kThreads)), dim3(kThreads), 0,
                  stream, particle_pin_start, pin_gradient, movable_count, particle_count, out);
}

}  // namespace mpgp
