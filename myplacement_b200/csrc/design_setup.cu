// The device's part of a session's set-up (design_setup.cuh).
//
// Compiled without fused multiply-add: every expression rounds as setup.cpp's does.
#include "design_setup.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <limits>

#include "common.cuh"
#include "pinned.hpp"

namespace mpgp {
namespace {

int blocksFor(long long count) { return std::max(1, ceilDiv(std::max(1LL, count), kThreads)); }

__global__ void __launch_bounds__(kThreads) mapModulesKernel(const int* movable, int count, int* particle) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < count) particle[movable[p]] = p;
}

__global__ void __launch_bounds__(kThreads) countPinsKernel(const int* pin_module, int pins, int* count) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < pins) atomicAdd(count + pin_module[p], 1);
}

// A row or fixed module that overlaps a bin row, with the columns its clipped rectangle spans.
struct StaticEntry {
    double llx, lly, urx, ury;
    int first_column, last_column;
};

struct StaticGrid {
    double llx, lly, bin_width, bin_height;
    int columns, rows;
    bool with_rows;       // the design has SiteRows: bins are dark where no row covers them
    double target_density;
};

__device__ __forceinline__ double positive(double v) { return v > 0.0 ? v : 0.0; }

// One thread per bin: the entries of its bin row in the design's order (rows, then fixed
// modules), as setPlaceableRegions and addRectangle visit the bin (Metrics.cpp:42-99).  The
// threads of a warp read the same entry at once.  262,144 bins of the 210,000-cell design: the
// host loops over rows and macros took 3 ms.
__global__ void __launch_bounds__(kThreads) staticLayersKernel(StaticGrid g, const StaticEntry* rows,
                                                              const int* row_start, const StaticEntry* modules,
                                                              const int* module_start, double2* fixed_dark,
                                                              double* static_charge, int* error) {
    const int column = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = blockIdx.y;
    if (column >= g.columns) return;
    const double left = g.llx + static_cast<double>(column) * g.bin_width;
    const double bottom = g.lly + static_cast<double>(row) * g.bin_height;
    const double right = left + g.bin_width;
    const double top = bottom + g.bin_height;
    const double area = positive(right - left) * positive(top - bottom);
    const auto overlap = [&](const StaticEntry& e) {
        const double l = e.llx < left ? left : e.llx;
        const double b = e.lly < bottom ? bottom : e.lly;
        const double r = right < e.urx ? right : e.urx;
        const double t = top < e.ury ? top : e.ury;
        return positive(r - l) * positive(t - b);
    };
    double d = 0.0;
    if (g.with_rows) {
        d = area;
        for (int k = row_start[row]; k < row_start[row + 1]; ++k) {
            const StaticEntry e = rows[k];
            if (column >= e.first_column && column <= e.last_column) d -= overlap(e);
        }
        const double tolerance = (area < 1.0 ? 1.0 : area) * 1e-10;
        if (d < -tolerance) atomicExch(error, 1);
        d = positive(d);
    }
    double f = 0.0;
    for (int k = module_start[row]; k < module_start[row + 1]; ++k) {
        const StaticEntry e = modules[k];
        if (column < e.first_column || column > e.last_column) continue;
        const double a = overlap(e);
        if (a > kEpsilon) f += a;
    }
    const size_t bin = static_cast<size_t>(row) * g.columns + column;
    fixed_dark[bin] = make_double2(f, d);
    static_charge[bin] = g.target_density * (f + d);
}

__global__ void __launch_bounds__(kThreads) areasKernel(DeviceModules m, int movable, Rect2 core, double* areas) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= movable) return;
    const int k = m.movable[p];
    const double w = m.width[k], h = m.height[k], x = m.x[k], y = m.y[k];
    const double l = x - w * 0.5, b = y - h * 0.5, r = x + w * 0.5, t = y + h * 0.5;
    const double width = (core.urx < r ? core.urx : r) - (l < core.llx ? core.llx : l);
    const double height = (core.ury < t ? core.ury : t) - (b < core.lly ? core.lly : b);
    const double area = positive(width) * positive(height);
    areas[p] = area > kEpsilon ? area : INFINITY;
}

__global__ void __launch_bounds__(kThreads) particlesKernel(DeviceModules m, ParticleArrays a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.count) return;
    double width, height, charge;
    double2 position;
    int layer, pins = 0;
    if (p < a.movable) {
        const int k = m.movable[p];
        width = m.width[k];
        height = m.height[k];
        // deriveDesign's macro rule (a movable module is no terminal).
        const bool macro = a.nominal_row_height > kEpsilon && fabs(height - a.nominal_row_height) > kEpsilon;
        layer = macro ? MPGP_LAYER_MACRO : MPGP_LAYER_STANDARD;
        const double area = width * height;
        charge = macro ? a.target_density * area : area;
        pins = m.pins[k];
        position = make_double2(m.x[k], m.y[k]);
    } else {
        width = a.filler_width;
        height = a.filler_height;
        layer = MPGP_LAYER_FILLER;
        charge = a.target_density * (width * height);
        position = a.filler_position[p - a.movable];
    }
    // initializePreconditioner (AdaptiveGlobalPlacer.cpp:358-375).
    const double area = width * height;
    const double ratio = area / (a.average_area < kEpsilon ? kEpsilon : a.average_area);
    const double area_ratio = ratio < 0.1 ? 0.1 : ratio;
    const double pin_factor = sqrt(1.0 + static_cast<double>(pins));
    const double area_factor = 1.0 + sqrt(area_ratio);
    a.size[p] = make_double2(width, height);
    a.layer[p] = static_cast<unsigned char>(layer);
    a.charge[p] = charge;
    a.precond[p] = 1.0 / (pin_factor * area_factor);
    a.position[p] = position;
}

// A bin row's entries in list order.
struct EntryLists {
    std::vector<StaticEntry> entries;
    std::vector<int> start;
};

struct Rectangle {
    double llx, lly, urx, ury;
};

// A rectangle's entry and the bin rows it goes to: those it spans (Grid::span).
struct Span {
    StaticEntry entry;
    int first_row, last_row;
};

// False for a rectangle that does not overlap the region.
bool spanOf(const Rectangle& r, const Rect2& region, int columns, int rows, Span& s) {
    const double bin_width = region.width() / static_cast<double>(columns);
    const double bin_height = region.height() / static_cast<double>(rows);
    const Rectangle c{std::max(r.llx, region.llx), std::max(r.lly, region.lly), std::min(r.urx, region.urx),
                      std::min(r.ury, region.ury)};
    const double area = std::max(0.0, c.urx - c.llx) * std::max(0.0, c.ury - c.lly);
    if (area <= kEpsilon) return false;
    const auto first = [](double offset, double length, int count) {
        return std::max(0, std::min(count - 1, static_cast<int>(std::floor(offset / length))));
    };
    const auto last = [](double offset, double length, int count) {
        return std::max(0, std::min(count - 1, static_cast<int>(std::ceil(offset / length) - 1.0)));
    };
    s.entry = StaticEntry{c.llx, c.lly, c.urx, c.ury, first(c.llx - region.llx, bin_width, columns),
                          last(c.urx - region.llx, bin_width, columns)};
    s.first_row = first(c.lly - region.lly, bin_height, rows);
    s.last_row = last(c.ury - region.lly, bin_height, rows);
    return true;
}

// The rectangles' entries by bin row, in the given order.
EntryLists entryLists(const std::vector<Rectangle>& rectangles, const Rect2& region, int columns, int rows) {
    std::vector<Span> spans;
    spans.reserve(rectangles.size());
    EntryLists out;
    out.start.assign(static_cast<std::size_t>(rows) + 1, 0);
    for (const Rectangle& r : rectangles) {
        Span s{};
        if (!spanOf(r, region, columns, rows, s)) continue;
        for (int row = s.first_row; row <= s.last_row; ++row) ++out.start[static_cast<std::size_t>(row) + 1];
        spans.push_back(s);
    }
    for (int row = 0; row < rows; ++row) out.start[static_cast<std::size_t>(row) + 1] += out.start[static_cast<std::size_t>(row)];
    out.entries.resize(static_cast<std::size_t>(out.start.back()));
    std::vector<int> at(out.start.begin(), out.start.end() - 1);
    for (const Span& s : spans) {
        for (int row = s.first_row; row <= s.last_row; ++row) {
            out.entries[static_cast<std::size_t>(at[static_cast<std::size_t>(row)]++)] = s.entry;
        }
    }
    return out;
}

Rectangle rowRectangle(const mpgp_design& d, int r) {
    const double x_end = d.row_x_start[r] + static_cast<double>(d.row_site_count[r]) * d.row_site_spacing[r];
    return {d.row_x_start[r], d.row_bottom[r], x_end, d.row_bottom[r] + d.row_height[r]};
}

Rectangle moduleRectangle(const mpgp_design& d, int32_t m) {
    const double x = d.module_x[m], y = d.module_y[m], w = d.module_width[m], h = d.module_height[m];
    return {x - w * 0.5, y - h * 0.5, x + w * 0.5, y + h * 0.5};
}

}  // namespace

uint64_t staticEntryCount(const mpgp_design& d, const DerivedDesign& derived, int bins_x, int bins_y) {
    uint64_t entries = 0;
    Span s{};
    const auto add = [&](const Rectangle& r) {
        if (spanOf(r, derived.core, bins_x, bins_y, s)) entries += static_cast<uint64_t>(s.last_row - s.first_row) + 1;
    };
    for (int r = 0; r < d.row_count; ++r) add(rowRectangle(d, r));
    if (derived.movable.size() < static_cast<std::size_t>(d.module_count)) {
        for (int32_t m = 0; m < d.module_count; ++m) {
            if (derived.is_fixed[m]) add(moduleRectangle(d, m));
        }
    }
    return entries;
}

uint64_t deviceSetupBytes(const mpgp_design& d, uint64_t static_entries, int bins_x, int bins_y) {
    const uint64_t pins = static_cast<uint64_t>(d.pin_count), modules = static_cast<uint64_t>(d.module_count);
    const uint64_t nets = static_cast<uint64_t>(d.net_count);
    const uint64_t bins = static_cast<uint64_t>(bins_x) * static_cast<uint64_t>(bins_y);
    // Per pin: the design's arrays (20), the layout's staging and sorting scratch (88) and its
    // lasting arrays (24); per module: geometry and maps, and the area sort (24); per net: the
    // offsets and weights, the net sort and the lasting arrays; the static layers and lists.
    return 160 * pins + 96 * modules + 128 * nets + 64 * bins + sizeof(StaticEntry) * static_entries +
           8 * (static_cast<uint64_t>(bins_y) + 1) + (uint64_t{32} << 20);
}

void launchMapModules(const DeviceModules& m, int movable, cudaStream_t stream) {
    checkCuda(cudaMemsetAsync(m.particle, 0xff, static_cast<std::size_t>(std::max(1, m.count)) * sizeof(int), stream),
              "Clear the module map");
    if (movable <= 0) return;
    mapModulesKernel<<<blocksFor(movable), kThreads, 0, stream>>>(m.movable, movable, m.particle);
    checkCuda(cudaGetLastError(), "Launch the module map");
}

void launchCountPins(const int* pin_module, int pins, int* count, cudaStream_t stream) {
    if (pins <= 0) return;
    countPinsKernel<<<blocksFor(pins), kThreads, 0, stream>>>(pin_module, pins, count);
    checkCuda(cudaGetLastError(), "Launch the pin count");
}

StaticSums staticLayersOnDevice(const mpgp_design& d, const DerivedDesign& derived, int bins_x, int bins_y,
                                double target_density, double* static_charge, const BudgetHeadroom& headroom,
                                cudaStream_t stream) {
    const Rect2& region = derived.core;
    require(region.width() >= -kEpsilon && region.height() >= -kEpsilon &&
                std::max(0.0, region.width()) * std::max(0.0, region.height()) > kEpsilon,
            "DensityMap requires a valid region, positive dimensions, and target density.");
    std::vector<Rectangle> rectangles;
    rectangles.reserve(static_cast<std::size_t>(d.row_count));
    for (int r = 0; r < d.row_count; ++r) rectangles.push_back(rowRectangle(d, r));
    const EntryLists rows = entryLists(rectangles, region, bins_x, bins_y);
    rectangles.clear();
    for (int32_t m = 0; m < d.module_count; ++m) {
        if (derived.is_fixed[m]) rectangles.push_back(moduleRectangle(d, m));
    }
    const EntryLists modules = entryLists(rectangles, region, bins_x, bins_y);

    const std::size_t bins = static_cast<std::size_t>(bins_x) * static_cast<std::size_t>(bins_y);
    Scratch scratch(stream, headroom);
    const auto put = [&](const auto& host) {
        using T = typename std::decay_t<decltype(host)>::value_type;
        T* device = scratch.array<T>(host.size());
        if (!host.empty()) {
            checkCuda(cudaMemcpyAsync(device, host.data(), host.size() * sizeof(T), cudaMemcpyHostToDevice, stream),
                      "static layer lists");
        }
        return static_cast<const T*>(device);
    };
    const StaticEntry* row_entries = put(rows.entries);
    const int* row_start = put(rows.start);
    const StaticEntry* module_entries = put(modules.entries);
    const int* module_start = put(modules.start);
    double2* fixed_dark = scratch.array<double2>(bins);
    int* error = scratch.array<int>(1);
    checkCuda(cudaMemsetAsync(error, 0, sizeof(int), stream), "static layers");
    const StaticGrid grid{region.llx,
                          region.lly,
                          region.width() / static_cast<double>(bins_x),
                          region.height() / static_cast<double>(bins_y),
                          bins_x,
                          bins_y,
                          d.row_count > 0,
                          target_density};
    const dim3 blocks(static_cast<unsigned>(ceilDiv(bins_x, kThreads)), static_cast<unsigned>(bins_y));
    staticLayersKernel<<<blocks, kThreads, 0, stream>>>(grid, row_entries, row_start, module_entries, module_start,
                                                        fixed_dark, static_charge, error);
    checkCuda(cudaGetLastError(), "Launch the static layers");
    int failed = 0;
    checkCuda(cudaMemcpyAsync(&failed, error, sizeof(int), cudaMemcpyDeviceToHost, stream), "static layers");
    StaticSums sums;
    int row = 0, column = 0;
    readDown(reinterpret_cast<const double*>(fixed_dark), 2 * bins,
             [&](const double* v, std::size_t count) {
                 for (const double* end = v + count; v != end; v += 2) {
                     const double left = region.llx + static_cast<double>(column) * grid.bin_width;
                     const double bottom = region.lly + static_cast<double>(row) * grid.bin_height;
                     const double area = std::max(0.0, (left + grid.bin_width) - left) *
                                         std::max(0.0, (bottom + grid.bin_height) - bottom);
                     sums.fixed += v[0];
                     sums.dark += v[1];
                     sums.placeable += area - v[1];
                     const double scaled_area = v[0] + 0.0 + v[1] + 0.0;
                     sums.charge += 0.0 + target_density * scaled_area;
                     if (++column == bins_x) {
                         column = 0;
                         ++row;
                     }
                 }
             },
             stream);
    require(failed == 0, "Overlapping SiteRows cannot define a density placeable-area mask.");
    return sums;
}

void sortAreasOnDevice(const DeviceModules& modules, int movable, const Rect2& core, double* sorted,
                       const BudgetHeadroom& headroom, cudaStream_t stream) {
    if (movable == 0) return;
    Scratch scratch(stream, headroom);
    double* areas = scratch.array<double>(static_cast<std::size_t>(movable));
    areasKernel<<<blocksFor(movable), kThreads, 0, stream>>>(modules, movable, core, areas);
    checkCuda(cudaGetLastError(), "Launch the area pass");
    std::size_t bytes = 0;
    checkCuda(cub::DeviceRadixSort::SortKeys(nullptr, bytes, areas, sorted, movable, 0, 64, stream), "area sort size");
    void* temp = scratch.array<unsigned char>(bytes);
    checkCuda(cub::DeviceRadixSort::SortKeys(temp, bytes, areas, sorted, movable, 0, 64, stream), "area sort");
}

void readDown(const double* device, std::size_t count, const std::function<void(const double*, std::size_t)>& consume,
              cudaStream_t stream) {
    constexpr std::size_t kPiece = std::size_t{1} << 17;  // doubles: 1 MB
    const PinnedBlock block(2 * kPiece * sizeof(double), "pinned read-back slots");
    double* slots = reinterpret_cast<double*>(block.data());
    cudaEvent_t arrived[2] = {};
    struct Events {
        cudaEvent_t* e;
        cudaStream_t stream;
        ~Events() {
            cudaStreamSynchronize(stream);  // no copy uses the slots any more
            for (int k = 0; k < 2; ++k) {
                if (e[k] != nullptr) cudaEventDestroy(e[k]);
            }
        }
    } events{arrived, stream};
    for (cudaEvent_t& e : arrived) checkCuda(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "Create event");
    const std::size_t pieces = (count + kPiece - 1) / kPiece;
    const auto size = [&](std::size_t k) { return std::min(kPiece, count - k * kPiece); };
    const auto fetch = [&](std::size_t k) {
        checkCuda(cudaMemcpyAsync(slots + (k % 2) * kPiece, device + k * kPiece, size(k) * sizeof(double),
                                  cudaMemcpyDeviceToHost, stream),
                  "Read back");
        checkCuda(cudaEventRecord(arrived[k % 2], stream), "Read back");
    };
    for (std::size_t k = 0; k < std::min<std::size_t>(2, pieces); ++k) fetch(k);
    for (std::size_t k = 0; k < pieces; ++k) {
        checkCuda(cudaEventSynchronize(arrived[k % 2]), "Read back");
        consume(slots + (k % 2) * kPiece, size(k));
        if (k + 2 < pieces) fetch(k + 2);
    }
}

void launchParticles(const DeviceModules& modules, const ParticleArrays& arrays, cudaStream_t stream) {
    if (arrays.count <= 0) return;
    particlesKernel<<<blocksFor(arrays.count), kThreads, 0, stream>>>(modules, arrays);
    checkCuda(cudaGetLastError(), "Launch the particle arrays");
}

}  // namespace mpgp
