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
void note_mat_mat(const char *kernel, uint32_t tile_rows);   // see mlxn_debug_last_mat_mat

// How exact a mat-mat's sums are.  The tensor core cuts off what an addition to an f32 accumulator leaves below its last bit, always towards zero: a
// chain of additions over K values is off by 1.2e-9 K of its result (measured against 64 bits, operands as given: K 2048 2.4e-6, 4096
// 4.8e-6, 6144 7.3e-6), sums outside the tensor core by a rounding.  So chains are to be short: accumulators take turns, tiles are cut
// along K.  (Either way the operands' rounding to f16, 2.8e-4 of the result, is most of a product's error.)  The measure is the mean square of the chains' lengths, in 4096ths of K^2 and weighted with what they hold.
constexpr uint32_t kChainAny = 4096;
// ... of tiles of `nraw` raw stages in `parts` each, `accs` accumulators taking turns, `cut` of the tiles cut once, anywhere, instead.
inline uint32_t chain_mean(uint32_t nraw, uint32_t parts, uint32_t accs, uint64_t tiles, uint64_t cut) {
    const uint32_t seg = (nraw + parts - 1) / parts, last = nraw % seg;
    const double a = (double)seg / nraw, b = (double)last / nraw, whole = nraw / seg * (a * a * a) + b * b * b;
    if (cut > tiles) cut = tiles;
    return (uint32_t)(kChainAny * (whole * (double)(tiles - cut) + 0.5 * (double)cut) / ((double)tiles * accs * accs));
}
// The limit that a dense product's launch is to keep, in this measure: what it has on single SMs, and no less than chains of 512 values have.
uint32_t qmm_chain_limit(const QmmArgs &a, int sm_count);

// The mat-mat on pairs of CTAs (qmm_duo.cu): whether it takes the call, which types, sizes and alignment decide, and the time that it would take
// (~0 where it does not) on the thread's current device, in the units of tc_plan; `nt` as for the other kernel, a multiple of 32.
bool qmm_duo_takes(int ggml_type, const QmmArgs &a);
uint64_t qmm_duo_cost(int ggml_type, const QmmArgs &a, uint32_t nt, uint32_t limit);
cudaError_t launch_qmm_duo(int ggml_type, const QmmArgs *ops, int nops, uint32_t nt, uint32_t limit, uint8_t *xpack, cudaStream_t st, int *launches);
constexpr uint32_t kRoutedTile = 64;   // rows of a routed tile
bool qmm_duo_routed_fits(int ggml_type, const QmmArgs &a);
cudaError_t launch_qmm_duo_routed(int ggml_type, const QmmArgs &a, uint32_t tiles, const uint8_t *xpack, cudaStream_t st, int *launches);

}  // namespace mlxn
