// Field solve of small grids in one launch (field_small.cu): the forward DCT, the
// spectral divide with its Parseval energy, the inverse transforms and, on request,
// the potential, by one cluster that keeps every intermediate in shared memory.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "dct_tc.cuh"

namespace mpgp {

// Grids of up to this many rows and columns take the one-launch solve.  128 is where
// its operands stop fitting: the data and the basis of one contraction are 64 KB each
// at 128 x 128 (two fp16 planes), and a row block is one UMMA tile of 128 rows.
constexpr int kFieldSmallMax = 128;

struct FieldSmallShape {
    int share_n = 0;  // columns per CTA: 64 for a grid of at most 64 x 64, else 32
    int cluster = 0;  // CTAs per grid (0: the grid is too large)
};
FieldSmallShape fieldSmallShape(int nx, int ny);

// What a launch runs.
enum FieldSmallMode : int {
    kSmallForward = 1,    // phi_hat (kept in phi_store) and the energy partials
    kSmallGradient = 2,   // the field; without kSmallForward from the phi_hat of the last forward launch
    kSmallPotential = 4,  // with kSmallGradient: also the potential
};

// One grid's solve, with the operands and exponent rules of the staged contractions
// (dct_tc.cuh): X = S Cx^T, rho_hat = Cy X, phi_hat = rho_hat .* scale,
// T = Dy phi_hat, U = phi_hat Dxc^T, Ex = T Sxwt^T, Ey = Syw U, phi = T Dxc^T.
struct alignas(64) FieldSmall {
    CUtensorMap map_s, map_cy, map_dy, map_syw;  // 128-row boxes
    CUtensorMap map_cx, map_dxc, map_sxwt;       // share_n-row boxes
    int nx = 0, ny = 0;
    FieldSmallShape shape;
    const int* row_exp = nullptr;  // per-row exponents of S
    TcScales* scales = nullptr;    // max_source (read, then cleared), max_phi and exp_phi (kept), exp_basis
    const float* scale = nullptr;  // spectral scale [ny][nx]
    float gain_x = 0.0f, gain_phi = 0.0f, gain_t = 0.0f, gain_u = 0.0f;  // |output| <= gain * max |data operand|
    double* energy_partials = nullptr;  // one per CTA
    float2* field = nullptr;
    float* potential = nullptr;
    unsigned char* phi_store = nullptr;  // fieldSmallStoreBytes: phi_hat and phi_hat^T as the inverse reads them
    int* error_flag = nullptr;
    long long stall_polls = 0;  // failure-detection probe, as TcBatch::stall_polls
};

size_t fieldSmallStoreBytes(int nx, int ny);

void launchFieldSmall(const FieldSmall& field, int mode, cudaStream_t stream);

// One grid of a batched launch (a FieldSmall in device memory) and its mode.
struct FieldSmallItem {
    const FieldSmall* field;
    int mode;
};
// Launches `count` items, all of grids of the shape `shape`, from device memory.
void launchFieldSmallBatch(const FieldSmallItem* items, int count, const FieldSmallShape& shape, cudaStream_t stream);

}  // namespace mpgp
