// What the mat-mat kernels share: how tiles are dealt out, and the launchers that one file calls in another.
#pragma once
#include "common.cuh"

namespace mlxn {

// How a dense mat-mat's work is dealt out when CTAs share tiles: tiles (weight tile fastest) x raw stages of 256 K values in one row,
// cut into `ctas` contiguous ranges, one for each CTA or pair of CTAs.  No tile is cut twice (a range is at least a tile long, or exactly half a tile): a shared
// tile is the sum of two parts added onto zeros, which is the same in either order.
struct TcShare {
    uint32_t ctas;        // 0: every CTA takes whole tiles
    uint32_t n_wt, nraw;  // weight-row tiles; raw stages of a tile
    uint32_t total;       // tiles x nraw
    uint32_t rows, nt;    // weight and activation rows of a tile
    __host__ __device__ uint32_t begin(uint32_t cta) const { return (uint32_t)((uint64_t)total * cta / ctas); }
};

// Products that share their activations in one launch: their weight tiles one after another.
constexpr uint32_t kMmOps = 4;
struct TcOut {
    float *y[kMmOps];
    uint32_t n[kMmOps], wt_end[kMmOps];   // weight rows; weight-row tiles of the products up to and including this one
    // the product of weight tile `wt`, which becomes that product's own tile number
    __device__ __forceinline__ uint32_t find(uint32_t &wt) const {
        uint32_t o = 0;
        while (wt >= wt_end[o]) o++;
        if (o) wt -= wt_end[o - 1];
        return o;
    }
};

constexpr uint32_t kPackRows = 64;   // rows of a tile that a block of pack_x_kernel packs
template <bool SWIGLU>
__global__ void pack_x_kernel(const QmmArgs a, uint8_t *xpack, uint32_t nchunks, uint32_t nt, const TcShare sh, const __grid_constant__ TcOut res);

int sm_count_of_device();

// The mat-mat on pairs of CTAs (qmm_duo.cu).  Time that it would take, in the units of tc_plan, or ~0 where it does not take the call;
// `nt` as for the other kernel, a multiple of 32.
uint64_t qmm_duo_cost(int ggml_type, const QmmArgs &a, uint32_t nt);
cudaError_t launch_qmm_duo(int ggml_type, const QmmArgs *ops, int nops, uint32_t nt, uint8_t *xpack, cudaStream_t st, int *launches);
constexpr uint32_t kRoutedTile = 64;   // rows of a routed tile
bool qmm_duo_routed_fits(int ggml_type, const QmmArgs &a);
cudaError_t launch_qmm_duo_routed(int ggml_type, const QmmArgs &a, uint32_t tiles, const uint8_t *xpack, cudaStream_t st, int *launches);

}  // namespace mlxn
