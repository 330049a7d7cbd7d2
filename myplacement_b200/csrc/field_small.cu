// One-launch tcgen05 field solve of small grids (sm_100a).
//
// On a grid of at most 128 x 128 the six contractions of
// ElectrostaticField::solveNeumann (ElectrostaticField.cpp:205-237) are one to four
// tiles each, and four launches of them spend their time between the tiles: waiting
// for the previous launch, fetching operands the previous launch has just written,
// and writing planes for the next one.  Here one cluster runs the whole chain.
//
// CTA r of the cluster owns columns r * N .. of every result and all (at most 128)
// rows, so that a result's transpose, the K-major B operand of the next contraction
// along y, is its own: it is split into fp16 planes straight into the swizzled operand
// tile in shared memory.  phi_hat and T are also A operands of contractions along x,
// over the columns of every CTA: each CTA writes its columns into the operand tile of
// every CTA of the cluster.  Four operand areas are reused along the chain:
//   data A   S -> phi_hat -> T             data B   X^T -> phi_hat^T -> U^T
//   basis A  Cy -> Dy -> Syw               basis B  Cx -> Dxc -> Sxwt (-> Dxc)
// The next basis is fetched as soon as the contraction that read the last one is done,
// behind its epilogue.  One thread issues the TMA loads and the tcgen05.mma (the products
// of the error-corrected fp16 split, as dct_tc.cu); every K-block has accumulators of
// its own, so one commit covers a step.  All 16 warps run the epilogues: warp w reads
// TMEM lanes 32 (w % 4) .. (tile rows) and the (w / 4)-th quarter of the columns.
//
// Bound by latency: a chain of four products with an epilogue, an operand write and a barrier
// each, on one to four SMs.  As four launches against one (a backend evaluation, and one
// iteration of a placement, microseconds):
//   32 x 32    90.6 ->  76.3   107.9 ->  86.7      65 x 65    101.5 ->  93.6   106.8 ->  91.6
//   64 x 64   101.5 ->  90.2    91.9 ->  74.5      128 x 64   128.7 -> 109.5    99.0 ->  78.2
//   96 x 96   118.6 -> 111.9   113.8 -> 105.3      128 x 128  143.3 -> 135.7   120.1 -> 114.3
// and 24 to 200 placements in shared launches 6 to 13 % faster.  Two K-blocks along an axis
// gain less: the FP64 sums of its epilogues are the larger part then.
//
// The arithmetic is that of dct_tc.cu: K-block partials summed in FP64 and rounded once
// to FP32, the same exponents from the same maxima.  With a single K-block the sum is
// main + 2^-11 corr, which one FP32 fma rounds once as well, and conversions to FP64
// (a quarter of the FP32 rate or less) are saved.
//
// Every mbarrier wait is bounded; a CTA whose wait runs out raises the error flag, skips
// further waits and products but reaches every cluster barrier, and drains its copies.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "field_small.cuh"
#include "split.cuh"
#include "tc_ptx.cuh"

namespace mpgp {
namespace {

using namespace tc;

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kAPlane = kTileM * kBlockK * 2;   // 16 KB: 128 rows of one K-block
constexpr int kABlock = kSplit * kAPlane;       // both planes
// The thread that issues the loads and products: in a warp whose TMEM lanes hold no rows of a
// grid of at most 64, so that it does so beside the epilogues there.
constexpr unsigned kIssuer = 64;
constexpr uint32_t kSecondTask = 128;           // TMEM columns of a step's first task
constexpr uint32_t kSmallTmem = 256;

// Shared memory for N columns per CTA: K-blocks (one at N = 64, up to two at N = 32) of
// the four operand areas, then the barriers and the exchanged maxima.
template <int N>
struct SmallLayout {
    static constexpr int kBlocks = N == 64 ? 1 : 2;
    static constexpr int kBBlock = kSplit * N * kBlockK * 2;
    static constexpr int kDataA = 0;
    static constexpr int kBasisA = kDataA + kBlocks * kABlock;
    static constexpr int kDataB = kBasisA + kBlocks * kABlock;
    static constexpr int kBasisB = kDataB + kBlocks * kBBlock;
    static constexpr int kScale = kBasisB + kBlocks * kBBlock;  // the spectral scale, a column of values per thread
    static constexpr int kTail = kScale + N / 4 * kSmallThreads * 4;  // 4 barriers, TMEM address, 2 maxima, warp energies
    static constexpr int kFieldPitch = 2 * N + 1;  // floats per staged field row (odd: no bank conflicts)
    static constexpr int kBytes = kTail + 4 * 8 + 16 + kSmallWarps * 8 + 1024 /* alignment slack */;
};
static_assert(SmallLayout<32>::kBytes <= 227 * 1024 && SmallLayout<64>::kBytes <= 227 * 1024, "one CTA's shared memory");
static_assert(SmallLayout<64>::kFieldPitch * 4 * 64 <= kABlock + SmallLayout<64>::kBBlock &&
                  SmallLayout<32>::kFieldPitch * 4 * 128 <= 2 * kABlock,
              "the staged field fits where the basis and data operands of the last contraction along y were");
static_assert(SmallLayout<32>::kBBlock % 1024 == 0 && kABlock % 1024 == 0, "swizzled tiles stay 1024-byte aligned");

__device__ __forceinline__ int planeExponentOf(float bound) {
    return min(120, max(-120, exponentOf(bound) - kPlaneTop));
}

__device__ __forceinline__ void loadColumns(uint32_t main_at, uint32_t corr_at, uint32_t (&m)[8], uint32_t (&c)[8]) {
    tmemLoad8(main_at, m);
    tmemLoad8(corr_at, c);
    tmemWait(m, c);
}

// One thread's row of a task's result: the sum of its K-block partials times 2^shift.
// `at` is the TMEM address of the thread's first main column; K-blocks are 2 N columns apart.
template <int N, int kCols>
__device__ __forceinline__ void readResult(uint32_t at, int k_blocks, int shift, float (&v)[kCols]) {
    if (k_blocks == 1) {
        uint32_t m[kCols], c[kCols];
        loadColumns(at, at + N, m, c);
        if (shift >= -126 && shift <= 127) {
            const float unscale = __int_as_float((shift + 127) << 23);
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
                v[j] = __fmaf_rn(__uint_as_float(c[j]), 1.0f / kLoShift, __uint_as_float(m[j])) * unscale;
            }
        } else {
            const double unscale = pow2(shift);
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
                const float part = __fmaf_rn(__uint_as_float(c[j]), 1.0f / kLoShift, __uint_as_float(m[j]));
                v[j] = static_cast<float>(static_cast<double>(part) * unscale);
            }
        }
        return;
    }
    double acc[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.0;
    for (int kb = 0; kb < k_blocks; ++kb) {
        uint32_t m[kCols], c[kCols];
        const uint32_t block = at + static_cast<uint32_t>(kb * 2 * N);
        loadColumns(block, block + N, m, c);
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            acc[j] += __fma_rn(static_cast<double>(__uint_as_float(c[j])), 1.0 / static_cast<double>(kLoShift),
                               static_cast<double>(__uint_as_float(m[j])));
        }
    }
    const double unscale = pow2(shift);
#pragma unroll
    for (int j = 0; j < kCols; ++j) v[j] = static_cast<float>(acc[j] * unscale);
}

// The planes of eight values, packed two halves to a word.
__device__ __forceinline__ void splitEight(const float (&v)[8], float inv_scale, uint4& h, uint4& l) {
    __half hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) splitScaled(v[i], inv_scale, hi[i], lo[i]);
    h = make_uint4(packHalves(hi[0], hi[1]), packHalves(hi[2], hi[3]), packHalves(hi[4], hi[5]), packHalves(hi[6], hi[7]));
    l = make_uint4(packHalves(lo[0], lo[1]), packHalves(lo[2], lo[3]), packHalves(lo[4], lo[5]), packHalves(lo[6], lo[7]));
}

// Writes row r of a result, columns n0 .. n0 + 7 of this CTA's N (n0 a multiple of 8), as
// column r of a K-major operand (128-byte swizzle: chunk c of operand row n sits at chunk
// c ^ (n % 8)).
template <int N>
__device__ __forceinline__ void writeTransposed(unsigned char* operand, int r, int n0, const uint4& h, const uint4& l) {
    unsigned char* tile = operand + (r >> 6) * (kSplit * N * kBlockK * 2) + n0 * 128 + (r & 7) * 2;
    const int chunk = (r & 63) >> 3;
    const uint32_t hi[4] = {h.x, h.y, h.z, h.w};
    const uint32_t lo[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        unsigned char* at = tile + j * 128 + ((chunk ^ j) << 4);
        *reinterpret_cast<unsigned short*>(at) = static_cast<unsigned short>(hi[j / 2] >> (16 * (j & 1)));
        *reinterpret_cast<unsigned short*>(at + N * 128) = static_cast<unsigned short>(lo[j / 2] >> (16 * (j & 1)));
    }
}

__device__ __forceinline__ void storeOwn16(uint32_t address, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

__device__ __forceinline__ void storeCluster16(uint32_t address, const uint4& v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}

// Writes row r, columns column .. column + 7 (of the whole grid, a multiple of 8) of a result
// as a K-major A operand in every CTA of the cluster.
__device__ __forceinline__ void writeRows(uint32_t operand, int rank, int cluster, int r, int column, const uint4& h,
                                          const uint4& l) {
    const int chunk = (column & 63) >> 3;
    const uint32_t at = operand + static_cast<uint32_t>((column >> 6) * kABlock + r * 128 + ((chunk ^ (r & 7)) << 4));
    storeOwn16(at, h);
    storeOwn16(at + kAPlane, l);
    for (int peer = 0; peer < cluster; ++peer) {
        if (peer == rank) continue;
        const uint32_t there = clusterAddress(at, static_cast<uint32_t>(peer));
        storeCluster16(there, h);
        storeCluster16(there + kAPlane, l);
    }
}

// Folds `v` (not negative) into the maximum at `slot` of every CTA of the cluster.
__device__ __forceinline__ void foldMaximum(float v, uint32_t slot, int cluster) {
    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    if ((threadIdx.x & 31) < static_cast<unsigned>(cluster)) {
        asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(
                         clusterAddress(slot, threadIdx.x & 31)),
                     "r"(top)
                     : "memory");
    }
}

// A writer's stores before the barrier that hands them to the tensor cores or the copy engine
// (about 800 cycles: the readers need none of their own).
__device__ __forceinline__ void asyncFence() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void tcBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One CTA of a grid's cluster; `local_block` indexes its energy partial.  The caller has
// released its successor.
template <int N>
__device__ __forceinline__ void fieldSmall(const FieldSmall& f, int mode, int local_block) {
    using L = SmallLayout<N>;
    constexpr int kCols = N / 4;
    constexpr uint32_t kDescriptor = instrDescriptor(N);
    constexpr uint32_t kPairDescriptor = instrDescriptor(2 * N);  // A x [B_hi; B_lo]: main and first correction
    __shared__ __align__(8) uint64_t probe;
    if (f.stall_polls > 0) {
        // Failure-detection probe: a bounded wait on a barrier that nothing completes.
        // Every CTA of every cluster takes this path before any cluster barrier, copy
        // or TMEM allocation, so nothing is in flight when it returns.
        if (threadIdx.x == 0) {
            mbarInit(smemAddress(&probe), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            bool done = false;
            for (long long k = 0; k < f.stall_polls && !done; ++k) done = mbarTryWait(smemAddress(&probe), 0);
            if (!done) atomicExch(f.error_flag, 1);
        }
        waitForPrior();
        __syncthreads();
        return;
    }
    const bool forward = (mode & kSmallForward) != 0;
    const bool gradient = (mode & kSmallGradient) != 0;
    const bool potential = gradient && (mode & kSmallPotential) != 0;
    const int cluster = f.shape.cluster;
    const int rank = static_cast<int>(clusterRank());
    const int n0 = rank * N;
    const int kx_blocks = (f.nx + kBlockK - 1) / kBlockK;
    const int ky_blocks = (f.ny + kBlockK - 1) / kBlockK;
    const int warp = threadIdx.x >> 5;
    const int r = (warp & 3) * 32 + static_cast<int>(threadIdx.x & 31);
    const int c0 = (warp >> 2) * kCols;   // the warp's first column within the CTA's N
    const int column = n0 + c0;
    // Rows past the last K-block of y feed no operand and no output.
    const bool active = (warp & 3) * 32 < ky_blocks * kBlockK;

    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const uint32_t data_a = smemAddress(smem + L::kDataA);
    const uint32_t basis_a = smemAddress(smem + L::kBasisA);
    const uint32_t data_b = smemAddress(smem + L::kDataB);
    const uint32_t basis_b = smemAddress(smem + L::kBasisB);
    uint64_t* barriers = reinterpret_cast<uint64_t*>(smem + L::kTail);
    uint32_t* tail = reinterpret_cast<uint32_t*>(barriers + 4);  // TMEM address, max |X|, max |phi_hat|, -
    double* energies = reinterpret_cast<double*>(tail + 4);
    const uint32_t full_a = smemAddress(barriers);
    const uint32_t full_b = smemAddress(barriers + 1);
    const uint32_t full_data = smemAddress(barriers + 2);
    const uint32_t products = smemAddress(barriers + 3);

    if (threadIdx.x == 0) {
        for (int b = 0; b < 4; ++b) mbarInit(full_a + 8 * b, 1);
        tail[1] = 0u;
        tail[2] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddress(tail)),
                     "r"(kSmallTmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        tcBefore();
    }
    __syncthreads();
    tcAfter();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tail);
    const uint32_t here = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(c0);
    clusterArrive();  // this CTA's maxima are cleared; peers wait for it before their first remote store

    // The issuer's loads and products.  Each barrier completes once per use.
    bool ok = true;
    uint32_t parity_a = 0, parity_b = 0, parity_data = 0, parity_products = 0;
    bool pending_a = false, pending_b = false, pending_data = false, pending_products = false;
    const auto fetchA = [&](const CUtensorMap* map) {
        mbarExpectTx(full_a, static_cast<uint32_t>(ky_blocks * kABlock));
        for (int kb = 0; kb < ky_blocks; ++kb) tmaLoad3d(basis_a + kb * kABlock, map, full_a, kb * kBlockK, 0, 0);
        pending_a = true;
    };
    const auto fetchB = [&](const CUtensorMap* map) {
        mbarExpectTx(full_b, static_cast<uint32_t>(kx_blocks * L::kBBlock));
        for (int kb = 0; kb < kx_blocks; ++kb) tmaLoad3d(basis_b + kb * L::kBBlock, map, full_b, kb * kBlockK, n0, 0);
        pending_b = true;
    };
    const auto landed = [&](uint32_t bar, uint32_t& parity, bool& pending) {
        if (ok) ok = mbarWait(bar, parity, f.error_flag);
        if (ok) {
            parity ^= 1u;
            pending = false;
        }
    };
    const auto multiply = [&](uint32_t a, uint32_t b, int k_blocks, uint32_t to) {
        for (int kb = 0; kb < k_blocks; ++kb) {
            const uint32_t main_acc = to + static_cast<uint32_t>(kb * 2 * N);
            const uint32_t corr_acc = main_acc + N;
            const uint32_t a_base = a + static_cast<uint32_t>(kb * kABlock);
            const uint32_t b_base = b + static_cast<uint32_t>(kb * L::kBBlock);
#pragma unroll
            for (int kk = 0; kk < kBlockK / 16; ++kk) {
                const uint64_t a_hi = smemDescriptor(a_base + kk * 32);
                const uint64_t a_lo = smemDescriptor(a_base + kAPlane + kk * 32);
                const uint64_t b_both = smemDescriptor(b_base + kk * 32);
                ummaF16(main_acc, a_hi, b_both, kPairDescriptor, kk > 0 ? 1u : 0u);
                ummaF16(corr_acc, a_lo, b_both, kDescriptor, 1u);
            }
        }
    };
    // Every thread: this step's products are complete.
    const auto awaitProducts = [&] {
        __syncwarp();
        if (ok) ok = mbarWait(products, parity_products, f.error_flag);
        parity_products ^= 1u;
        if (ok) pending_products = false;
        __syncwarp();
        tcAfter();
    };
    // Every thread, after its stores to shared memory and its TMEM loads.
    const auto exchange = [&] {
        __syncwarp();
        tcBefore();
        if (cluster > 1) {
            clusterArrive();
            clusterWait();
        } else {
            __syncthreads();
        }
        tcAfter();
    };

    if (threadIdx.x == kIssuer) {  // fixed tables: before the predecessor has finished
        fetchA(forward ? &f.map_cy : &f.map_dy);
        fetchB(forward ? &f.map_cx : &f.map_dxc);
        for (const CUtensorMap* map : {&f.map_s, &f.map_dy, &f.map_dxc, &f.map_syw, &f.map_sxwt}) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
        }
    }
    float* const scale = reinterpret_cast<float*>(smem + L::kScale) + threadIdx.x;  // read back by this thread only
    if (forward) {
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            scale[j * kSmallThreads] =
                r < f.ny && column + j < f.nx ? __ldg(f.scale + static_cast<size_t>(r) * f.nx + column + j) : 0.0f;
        }
    }
    waitForPrior();
    __syncwarp();
    clusterWait();
    // The kept phi_hat: its A operand (every K-block), then each CTA's B operand.
    unsigned char* const kept_b = f.phi_store + static_cast<size_t>(kx_blocks) * kABlock +
                                  static_cast<size_t>(rank) * ky_blocks * L::kBBlock;
    if (threadIdx.x == kIssuer) {
        if (forward) {
            mbarExpectTx(full_data, static_cast<uint32_t>(kx_blocks * kABlock));
            for (int kb = 0; kb < kx_blocks; ++kb) {
                tmaLoad3d(data_a + kb * kABlock, &f.map_s, full_data, kb * kBlockK, 0, 0);
            }
        } else {
            mbarExpectTx(full_data, static_cast<uint32_t>(kx_blocks * kABlock + ky_blocks * L::kBBlock));
            bulkFromGlobal(data_a, f.phi_store, static_cast<uint32_t>(kx_blocks * kABlock), full_data);
            bulkFromGlobal(data_b, kept_b, static_cast<uint32_t>(ky_blocks * L::kBBlock), full_data);
        }
        pending_data = true;
    }
    const volatile TcScales* known = f.scales;
    const int exp_cx = known->exp_basis[0], exp_cy = known->exp_basis[1], exp_dy = known->exp_basis[2];
    const int exp_dxc = known->exp_basis[3], exp_sxwt = known->exp_basis[4], exp_syw = known->exp_basis[5];
    const int exp_row = forward && r < f.ny ? __ldg(f.row_exp + r) : 0;
    const int exp_x = forward ? planeExponentOf(__uint_as_float(known->max_source) * f.gain_x) : 0;
    int exp_phi = forward ? 0 : known->exp_phi;
    float top_phi = forward ? 0.0f : __uint_as_float(known->max_phi);
    int exp_t = planeExponentOf(top_phi * f.gain_t);
    int exp_u = planeExponentOf(top_phi * f.gain_u);

    // The steps of the chain share one loop body: code that runs once is fetched as it runs, and
    // a step is a few thousand cycles (X 3,500 for the source, 250 after the last product, 2,400
    // for the epilogue; T and U 5,100 of epilogue).  Unrolled, with a fence on the readers' side
    // and the loads issued by an epilogue warp, an evaluation took 2 us more (94.8 us against 93
    // at 64 x 64, 104.4 against 102.5 at 128 x 128).
    enum { kX = 0, kPhi, kTU, kField, kPotential };
    const int last = !gradient ? kPhi : (potential ? kPotential : kField);
#pragma unroll 1
    for (int step = forward ? kX : kTU; step <= last; ++step) {
        const int tasks = step == kTU || step == kField ? 2 : 1;
        // Task 0 of T/U and phi_hat contract along y: A = basis A, B = data B.  The others
        // contract along x: A = data A, B = basis B.
        const auto alongX = [&](int task) {
            return step == kX || step == kPotential || (step == kTU && task == 1) || (step == kField && task == 0);
        };
        if (threadIdx.x == kIssuer) {
            if (pending_data) landed(full_data, parity_data, pending_data);
            if (step != kX && step != kPotential) landed(full_a, parity_a, pending_a);
            if (step != kPhi) landed(full_b, parity_b, pending_b);
            tcAfter();
            if (ok) {
#pragma unroll 1
                for (int task = 0; task < tasks; ++task) {
                    const bool x = alongX(task);
                    multiply(x ? data_a : basis_a, x ? basis_b : data_b, x ? kx_blocks : ky_blocks,
                             tmem + static_cast<uint32_t>(task) * kSecondTask);
                }
                ummaCommit(products);
                pending_products = true;
            }
            if (step == kPhi && rank == 0) f.scales->max_source = 0u;  // every CTA has read it
        }
        awaitProducts();
        if (threadIdx.x == kIssuer) {
            // The next basis, behind this step's epilogue.
            if (ok && gradient) {
                if (step == kPhi || step == kTU) fetchA(step == kPhi ? &f.map_dy : &f.map_syw);
                if (step == kX || step == kTU) fetchB(step == kX ? &f.map_dxc : &f.map_sxwt);
                if (step == kField && potential) fetchB(&f.map_dxc);
            }
            if (step == kTU) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the kept copies have read the operands
            }
        }
        // T and U replace operands that every CTA's products (and copies) have to have read.
        if (step == kTU) exchange();

        float top = 0.0f;
        double energy = 0.0;
        if (active) {
#pragma unroll 1
            for (int unit = 0; unit < tasks * (kCols / 8); ++unit) {
                const int task = unit / (kCols / 8);
                const int j0 = unit % (kCols / 8) * 8;
                const int shift = step == kX     ? exp_cx + exp_row
                                  : step == kPhi ? exp_cy + exp_x
                                  : step == kTU  ? (task == 0 ? exp_dy : exp_dxc) + exp_phi
                                  : step == kField ? (task == 0 ? exp_t + exp_sxwt : exp_syw + exp_u)
                                                   : exp_t + exp_dxc;
                float v[8];
                readResult<N, 8>(here + static_cast<uint32_t>(task) * kSecondTask + static_cast<uint32_t>(j0),
                                 alongX(task) ? kx_blocks : ky_blocks, shift, v);
                if (step == kPhi) {
                    const double wr = parsevalWeight(r);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float phi = v[j] * scale[(j0 + j) * kSmallThreads];
                        if (r < f.ny && column + j0 + j < f.nx) {
                            energy += static_cast<double>(phi) * static_cast<double>(v[j]) * wr *
                                      parsevalWeight(column + j0 + j);
                        }
                        v[j] = phi;
                    }
                }
                if (step <= kTU) {
                    const int e = step == kX ? exp_x : step == kPhi ? exp_phi : task == 0 ? exp_t : exp_u;
                    const float inv_scale = static_cast<float>(pow2(-e));
#pragma unroll
                    for (int j = 0; j < 8; ++j) top = fmaxf(top, fabsf(v[j]));
                    uint4 h, l;
                    splitEight(v, inv_scale, h, l);
                    if (step != kX && task == 0) writeRows(data_a, rank, cluster, r, column + j0, h, l);
                    if (step != kTU || task == 1) writeTransposed<N>(smem + L::kDataB, r, c0 + j0, h, l);
                } else if (step == kField) {
                    float* staged = reinterpret_cast<float*>(smem + L::kBasisA) + r * L::kFieldPitch + 2 * (c0 + j0) + task;
#pragma unroll
                    for (int j = 0; j < 8; ++j) staged[2 * j] = v[j];
                } else if (r < f.ny) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (column + j0 + j < f.nx) f.potential[static_cast<size_t>(r) * f.nx + column + j0 + j] = v[j];
                    }
                }
            }
            if (step <= kPhi) foldMaximum(top, smemAddress(tail + 1 + step), cluster);
            if (step <= kTU) asyncFence();
        }
        if (step == kPhi) {
            energy = warpSum(energy);
            if ((threadIdx.x & 31) == 0) energies[warp] = energy;
        }
        if (step <= kTU) {
            exchange();
        } else {
            tcBefore();
            __syncthreads();
        }
        if (step == kX) {
            const float top_x = __uint_as_float(*reinterpret_cast<volatile uint32_t*>(tail + 1));
            exp_phi = planeExponentOf(top_x * f.gain_phi);
        } else if (step == kPhi) {
            top_phi = __uint_as_float(*reinterpret_cast<volatile uint32_t*>(tail + 2));
            exp_t = planeExponentOf(top_phi * f.gain_t);
            exp_u = planeExponentOf(top_phi * f.gain_u);
            if (threadIdx.x == kIssuer) {
                // phi_hat is kept for a later launch without the forward transform: each K-block
                // of the A operand by the CTA that owns its first column, the B operand by its CTA.
                if (n0 % kBlockK == 0) {
                    bulkToGlobal(f.phi_store + static_cast<size_t>(n0 / kBlockK) * kABlock,
                                 data_a + n0 / kBlockK * kABlock, kABlock);
                }
                bulkToGlobal(kept_b, data_b, static_cast<uint32_t>(ky_blocks * L::kBBlock));
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            if (threadIdx.x == kIssuer + 32) {
                double sum = 0.0;
                for (int w = 0; w < kSmallWarps; ++w) sum += energies[w];
                if (f.energy_partials != nullptr) f.energy_partials[local_block] = sum;
                if (rank == 0) {
                    f.scales->max_phi = __float_as_uint(top_phi);
                    f.scales->exp_phi = exp_phi;
                }
            }
        } else if (step == kField) {
            // Whole rows of the CTA's columns, a warp per row.
            const int floats = 2 * max(0, min(N, f.nx - n0));
            for (int row = warp; row < f.ny; row += kSmallWarps) {
                const float* staged = reinterpret_cast<const float*>(smem + L::kBasisA) + row * L::kFieldPitch;
                float* out = reinterpret_cast<float*>(f.field + static_cast<size_t>(row) * f.nx + n0);
                for (int c = threadIdx.x & 31; c < floats; c += 32) out[c] = staged[c];
            }
        }
    }
    if (threadIdx.x == kIssuer) {
        // Drain: nothing this CTA issued lands after it exits (all done already unless a wait ran out).
        if (pending_a) mbarWait(full_a, parity_a, nullptr);
        if (pending_b) mbarWait(full_b, parity_b, nullptr);
        if (pending_data) mbarWait(full_data, parity_data, nullptr);
        if (pending_products) mbarWait(products, parity_products ^ 1u, nullptr);
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tcBefore();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kSmallTmem));
    }
}

template <int N>
__global__ void __launch_bounds__(kSmallThreads, 1) fieldSmallKernel(const __grid_constant__ FieldSmall field, int mode) {
    releaseNext();
    fieldSmall<N>(field, mode, static_cast<int>(blockIdx.x));
}

// Batched: cluster c solves the grid items[c].field (a FieldSmall in device memory, whose
// tensor maps the TMA reads there).
template <int N>
__global__ void __launch_bounds__(kSmallThreads, 1) fieldSmallBatchKernel(const FieldSmallItem* items, int cluster) {
    releaseNext();
    const FieldSmallItem item = items[blockIdx.x / static_cast<unsigned>(cluster)];
    const FieldSmall& field = *item.field;
    if (threadIdx.x == kIssuer) {
        // Uploaded by a copy, possibly into memory an earlier engine's maps used: the thread that
        // prefetches them and issues the loads makes the TMA proxy see their current bytes.
        for (const CUtensorMap* map : {&field.map_s, &field.map_cy, &field.map_dy, &field.map_syw, &field.map_cx,
                                       &field.map_dxc, &field.map_sxwt}) {
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
        }
    }
    fieldSmall<N>(field, item.mode, static_cast<int>(blockIdx.x % static_cast<unsigned>(cluster)));
}

// The shared-memory attribute is per device: set it once on each device that launches.
template <int N>
void configureSmall() {
    constexpr int kMaxDevices = 64;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attribute[kMaxDevices] = {};
    int device = 0;
    checkCuda(cudaGetDevice(&device), "Query the current device");
    require(device >= 0 && device < kMaxDevices, "Device index out of range.");
    std::call_once(once[device], [device] {
        attribute[device] = cudaFuncSetAttribute(fieldSmallKernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 SmallLayout<N>::kBytes);
        if (attribute[device] == cudaSuccess) {
            attribute[device] = cudaFuncSetAttribute(
                fieldSmallBatchKernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmallLayout<N>::kBytes);
        }
    });
    checkCuda(attribute[device], "Configure the small-grid field kernel");
}

template <int N>
cudaLaunchConfig_t smallConfig(int blocks, int cluster, cudaStream_t stream, cudaLaunchAttribute* attribute) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(blocks));
    config.blockDim = dim3(kSmallThreads);
    config.dynamicSmemBytes = SmallLayout<N>::kBytes;
    config.stream = stream;
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 2;
    return config;
}

template <int N>
void launchSmallN(const FieldSmall& field, int mode, cudaStream_t stream) {
    configureSmall<N>();
    cudaLaunchAttribute attribute[2] = {};
    const cudaLaunchConfig_t config = smallConfig<N>(field.shape.cluster, field.shape.cluster, stream, attribute);
    checkCuda(cudaLaunchKernelEx(&config, fieldSmallKernel<N>, field, mode), "Launch the small-grid field kernel");
}

template <int N>
void launchSmallBatchN(const FieldSmallItem* items, int count, int cluster, cudaStream_t stream) {
    configureSmall<N>();
    cudaLaunchAttribute attribute[2] = {};
    const cudaLaunchConfig_t config = smallConfig<N>(count * cluster, cluster, stream, attribute);
    checkCuda(cudaLaunchKernelEx(&config, fieldSmallBatchKernel<N>, items, cluster),
              "Launch the batched small-grid field kernel");
}

void checkShape(const FieldSmallShape& s) {
    require((s.share_n == 64 && s.cluster == 1) || (s.share_n == 32 && (s.cluster == 2 || s.cluster == 4)),
            "The one-launch field solve does not take this grid.");
}

}  // namespace

FieldSmallShape fieldSmallShape(int nx, int ny) {
    FieldSmallShape s;
    if (nx <= 0 || ny <= 0 || nx > kFieldSmallMax || ny > kFieldSmallMax) return s;
    // One K-block along both axes: a single CTA.  Two along either: 32 columns per CTA, so
    // that the FP64 sums, which bound the epilogues then, spread over two or four SMs.
    const bool one = nx <= kBlockK && ny <= kBlockK;
    s.share_n = one ? kBlockK : kBlockK / 2;
    s.cluster = (nx + kBlockK - 1) / kBlockK * (kBlockK / s.share_n);
    return s;
}

size_t fieldSmallStoreBytes(int nx, int ny) {
    const FieldSmallShape s = fieldSmallShape(nx, ny);
    const size_t kx = static_cast<size_t>((nx + kBlockK - 1) / kBlockK);
    const size_t ky = static_cast<size_t>((ny + kBlockK - 1) / kBlockK);
    return kx * kABlock + static_cast<size_t>(s.cluster) * ky * kSplit * s.share_n * kBlockK * 2;
}

void launchFieldSmall(const FieldSmall& field, int mode, cudaStream_t stream) {
    checkShape(field.shape);
    if (field.shape.share_n == 64) {
        launchSmallN<64>(field, mode, stream);
    } else {
        launchSmallN<32>(field, mode, stream);
    }
}

void launchFieldSmallBatch(const FieldSmallItem* items, int count, const FieldSmallShape& shape, cudaStream_t stream) {
    if (count <= 0) return;
    checkShape(shape);
    if (shape.share_n == 64) {
        launchSmallBatchN<64>(items, count, shape.cluster, stream);
    } else {
        launchSmallBatchN<32>(items, count, shape.cluster, stream);
    }
}

}  // namespace mpgp
