// Host-side setup of one global-placement problem: the engine's input model.
//
// A Problem is what the device engine needs: particles (movable modules in
// module order, then density fillers), the netlist flattened to pin CSR, the
// bin grid and the static density layers.  It is built either from the
// drop-in layout (mpgp_layout, i.e. what tryCreateCudaPlacementBackend
// receives) or from a whole design, in which case the reference's session
// setup is restated here operation for operation so that fillers, static
// layers and preconditioner are bit-identical to the reference's.
#pragma once

#include <cstddef>
#include <cstdint>
#include <functional>
#include <random>
#include <vector>

#include "mpgp.h"

namespace mpgp {

struct Rect2 {
    double llx = 0.0, lly = 0.0, urx = 0.0, ury = 0.0;
    [[nodiscard]] double width() const { return urx - llx; }
    [[nodiscard]] double height() const { return ury - lly; }
};

struct Problem {
    int64_t particle_count = 0;
    int64_t movable_count = 0;
    std::vector<double> width;         // P
    std::vector<double> height;        // P
    std::vector<int32_t> layer;        // P, MPGP_LAYER_*
    std::vector<double> charge;        // P, densityChargeArea
    std::vector<double> precond_base;  // P, empty for the drop-in backend
    std::vector<int32_t> pin_count;    // P (module pins; 0 for fillers)

    std::vector<double> net_weight;        // N
    std::vector<int64_t> net_pin_start;    // N + 1
    std::vector<int32_t> pin_particle;     // I, -1 for static pins
    std::vector<double> pin_x, pin_y;      // I: transformed offset, or absolute static position

    int bins_x = 0;
    int bins_y = 0;
    Rect2 region;
    double target_density = 0.0;
    std::vector<double> static_fixed;  // B
    std::vector<double> static_dark;   // B
};

// What refreshDerivedData (PlacementDatabase.cpp:162-200) derives from a design.
struct DerivedDesign {
    double nominal_row_height = 0.0;
    Rect2 core;
    std::vector<uint8_t> is_fixed;
    std::vector<uint8_t> is_macro;
    std::vector<int32_t> movable;    // module ids in module order
    std::vector<int32_t> pin_count;  // per module
};

// Without `with_pins` the pin counts stay empty.
DerivedDesign deriveDesign(const mpgp_design& design, bool with_pins = true);
// The pins per module.
std::vector<int32_t> countPins(const mpgp_design& design);
// The median row height (zero without rows): a standard cell's height.
double nominalRowHeight(const mpgp_design& design);

// Validates the design arrays (sizes, indices, finiteness).
void validateDesign(const mpgp_design& design);
// Its first part: counts, missing arrays and the pin total, without a pass over the arrays.
void validateDesignShape(const mpgp_design& design);

// validateAdaptiveOptions (AdaptiveGlobalPlacer.cpp:413-454) plus the engine's own limits.
void validateOptions(const mpgp_options& options);

// The static density layers of DensityMap after initializeStaticDensity
// (GlobalPlacementSupport.cpp:21-30 -> Metrics.cpp:42-99).
void staticDensity(const mpgp_design& design, const DerivedDesign& derived, int bins_x, int bins_y,
                   double target_density, std::vector<double>& fixed, std::vector<double>& dark);

struct Filler {
    double x, y, width, height;
};

// createDensityFillers (GlobalPlacementSupport.cpp:52-103).
std::vector<Filler> createFillers(const mpgp_design& design, const DerivedDesign& derived,
                                  const std::vector<double>& fixed, const std::vector<double>& dark,
                                  int bins_x, int bins_y, const mpgp_options& options);

// Its parts: the movable modules' areas summed in module order, the fillers' number and size
// from the areas inside the core in ascending order (those above kEpsilon), and their seeded
// centres in order.
struct MovableAreas {
    double standard = 0.0, macro = 0.0;  // inside the core
    double total = 0.0;                  // of the whole modules (initializePreconditioner)
    std::size_t positive = 0;            // modules with more than kEpsilon inside the core
};
MovableAreas movableAreas(const mpgp_design& design, const DerivedDesign& derived);
struct FillerPlan {
    std::size_t count = 0;
    double width = 0.0, height = 0.0;
};
// trimmed_sum(lower, upper) sums the ascending areas [lower, upper) in order.
FillerPlan planFillers(const Rect2& core, const MovableAreas& areas, double static_charge_area,
                       const std::function<double(std::size_t, std::size_t)>& trimmed_sum,
                       const mpgp_options& options);
// The seeded uniform numbers in [0, 1) of the first `count` fillers (two each), and the centres
// made of them: x0, y0, x1, y1, ...  (uniform_real_distribution's formula; `unit` holds as many
// as are at hand and is extended as needed).
struct FillerNumbers {
    explicit FillerNumbers(uint64_t seed) : generator(seed ^ 0x9e3779b97f4a7c15ULL) {}
    void extend(std::size_t count);
    std::mt19937_64 generator;
    std::vector<double> unit;
};
std::vector<double> fillerCentres(const Rect2& core, const FillerPlan& plan, FillerNumbers& numbers);

// The whole session setup (AdaptiveGlobalPlacer.cpp:114-126 plus buildHostLayout,
// CudaPlacementBackend.cu:784-839).  `fillers` receives the filler geometry.
Problem buildProblem(const mpgp_design& design, const DerivedDesign& derived, const mpgp_options& options,
                     std::vector<Filler>& fillers);
// Its two independent parts, which write disjoint members of `problem` and may run
// on two threads at once: the net and pin arrays (buildHostLayout's CSR part), and
// the grid, the static layers, the fillers and the particle arrays.
void buildProblemPins(const mpgp_design& design, const DerivedDesign& derived, Problem& problem);
void buildProblemParticles(const mpgp_design& design, const DerivedDesign& derived, const mpgp_options& options,
                           Problem& problem, std::vector<Filler>& fillers);

// The drop-in path: a Problem from an mpgp_layout.
Problem problemFromLayout(const mpgp_layout& layout);

// randomPlacement (InitialPlacer.cpp:102-121).
void randomPlacement(const mpgp_design& design, const DerivedDesign& derived, uint64_t seed, double* module_x,
                     double* module_y);

// Fills GlobalPlacementOptions defaults (GlobalPlacer.hpp:26-80).
void defaultOptions(mpgp_options& options);

}  // namespace mpgp
