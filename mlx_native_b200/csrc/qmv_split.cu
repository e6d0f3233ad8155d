// Dispatcher of the split mat-vec (qmv_split.cuh).
#include "qmv_split.cuh"

#include "../../include/mlxn_b200.h"

namespace mlxn {

extern template cudaError_t sp_run<GT_Q4_0>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);
extern template cudaError_t sp_run<GT_Q8_0>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);
extern template cudaError_t sp_run<GT_Q4_K>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);
extern template cudaError_t sp_run<GT_Q5_K>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);
extern template cudaError_t sp_run<GT_Q6_K>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);

// Every weight row starts on a 16-byte boundary: the rows arrive by tensor copies.
bool qmv_split_aligned(int ggml_type, const QmvArgs &a) {
    const uint64_t rb = (uint64_t)(a.k / ggml_qk(ggml_type)) * ggml_block_bytes(ggml_type);
    return rb % 16 == 0 && ((uintptr_t)a.w & 15u) == 0 && (!a.ids || a.expert_stride % 16 == 0);
}

static SpPick split_pick(int ggml_type, bool aligned, uint32_t mp, bool routed, uint64_t tiles, uint32_t units, int sm_count) {
    const bool packed = !routed && mp > 2;
    switch (ggml_type) {
    case GT_Q4_0: return sp_pick<GT_Q4_0>(aligned, mp, packed, routed, tiles, units, sm_count);
    case GT_Q8_0: return sp_pick<GT_Q8_0>(aligned, mp, packed, routed, tiles, units, sm_count);
    case GT_Q4_K: return sp_pick<GT_Q4_K>(aligned, mp, packed, routed, tiles, units, sm_count);
    case GT_Q5_K: return sp_pick<GT_Q5_K>(aligned, mp, packed, routed, tiles, units, sm_count);
    default: return sp_pick<GT_Q6_K>(aligned, mp, packed, routed, tiles, units, sm_count);
    }
}

// Sizes, types and addresses that the kernel takes; `pick`: the geometry of a launch of this mat-vec alone.
bool qmv_split_fits(int ggml_type, const QmvArgs &a, int sm_count, SpPick *pick) {
    const bool kq = ggml_type == GT_Q4_K || ggml_type == GT_Q5_K;
    if (ggml_type != GT_Q4_0 && ggml_type != GT_Q8_0 && ggml_type != GT_Q6_K && !kq) return false;
    if (a.m == 0 || a.n == 0 || a.k == 0 || a.k % ggml_qk(ggml_type) != 0) return false;
    // the activations are read as pairs of floats
    if (((uintptr_t)a.x & 7u) || ((uintptr_t)a.x2 & 7u) || ((uintptr_t)a.w & 1u)) return false;
    const bool aligned = qmv_split_aligned(ggml_type, a);
    if (kq && (!aligned || a.x2)) return false;
    if (a.x2 && !a.ids) return false;   // (the fused SwiGLU is expert-routed)
    if (ggml_type == GT_Q5_K && !a.ids) return false;
    if ((uint64_t)(a.k / ggml_qk(ggml_type)) * ggml_block_bytes(ggml_type) >= (1ull << 31)) return false;
    uint32_t mp = a.m <= 1 ? 1u : a.m <= 2 ? 2u : a.m <= 4 ? 4u : 8u, ranks = 8;
    if (a.ids) {
        // K is not split over a cluster here; a pair more and the bucketing of a launch does not fit one block
        if (a.nprob == 0 || a.nprob > (uint32_t)kSpMaxPairs || a.n_experts > 65535u || a.m != 1) return false;
        mp = a.nprob <= 1 ? 1u : 4u;
        ranks = 1;
    }
    if (((uint64_t)a.m + 7) / 8 * ((a.n + 15) / 16) >= (1ull << 31)) return false;
    if ((uint64_t)a.m * a.k >= (1ull << 31)) return false;
    // Up to here the kernel has been compared with the others: the activations of a K slice (272 bytes per 64 values and row) beside
    // 40 KB, which is K = 14336 for five rows and more, 30720 for three and four, 65536 for two and 133120 for one; routed, where one
    // CTA holds all of K, 3840 for several pairs and 16640 for one.
    const uint32_t units = (a.k + 63) / 64, slice = ((units + ranks - 1) / ranks + 3) / 4 * 4 + 2;
    if ((uint64_t)slice * mp * 272 + 40 * 1024 > kSpSmem) return false;
    // (the batch that a mat-vec leaves with takes the geometry of its longest K: that one's own)
    *pick = split_pick(ggml_type, aligned, mp, a.ids != nullptr, (a.n + 15) / 16, units, sm_count);
    return pick->ranks != 0;
}

bool qmv_split_supported(int ggml_type, const QmvArgs &a, int sm_count) {
    SpPick pick;
    return qmv_split_fits(ggml_type, a, sm_count, &pick) && encode_tiled_fn() != nullptr;
}

// Whether mat-vecs that the register-level kernel takes too (dense, aligned, one block type and row class) leave by this kernel,
// where nothing else runs meanwhile.  It
// starts 1 to 3 us later and has the higher rate, and its time grows evenly, where the other one's is a number of passes over the chip:
// what decides is how full those passes are (`fill`, qmv_mma_fill) and how much there is to read.  Graph replay of dependent
// launches, us with the register-level kernel (one mat-vec of three or four rows: the tensor-memory kernel) / with this one:
//   one row    4096 values wide   5120 rows     8192 (fill 0.86)   10240 (0.54)   12288 (0.65)   14336 (0.76)   16384 (0.86)   18432 (0.97)   20480 (0.54)   32768 (0.86)
//     Q4_0                        7.7 / 7.2     8.6 / 8.7          12.7 / 9.6     12.9 / 10.1    13.2 / 10.8    14.0 / 11.6    15.0 / 12.5    23.4 / 14.2    26.2 / 19.9
//     Q8_0                        8.7 / 8.3     10.2 / 10.4        14.8 / 11.9    15.4 / 13.2    16.0 / 15.7    16.6 / 16.7    18.6 / 18.5    27.8 / 20.2    30.9 / 30.1
//     Q6_K                        11.1 / 10.9   11.6 / 12.0        18.4 / 14.5    18.6 / 14.9    18.9 / 16.9    19.3 / 18.1    19.9 / 19.3    32.2 / 22.9    36.5 / 30.9
//     Q4_K                        8.3 / 9.1     9.2 / 10.0         14.1 / 11.3    14.2 / 11.6    14.5 / 13.0    15.4 / 14.0    16.4 / 14.4    26.0 / 17.3    28.6 / 22.1
//   two rows
//     Q4_0                        9.2 / 8.9     9.9 / 10.9         13.9 / 12.8    13.9 / 13.7    14.1 / 14.8    15.1 / 15.4    16.2 / 16.4    26.5 / 18.7    28.1 / 26.2
//     Q8_0                        10.1 / 9.5    11.0 / 11.2        16.0 / 15.0    16.4 / 16.7    17.0 / 17.4    17.5 / 19.1    19.1 / 20.9    29.6 / 23.9    32.6 / 33.4
//     Q6_K                        13.3 / 12.5   13.9 / 14.0        20.3 / 18.4    20.6 / 19.7    20.8 / 21.2    21.3 / 22.3    22.0 / 23.7    37.2 / 26.9    40.4 / 37.9
//     Q4_K                        9.9 / 10.7    10.4 / 14.4        15.3 / 14.8    15.4 / 16.3    15.7 / 18.9    16.5 / 19.8    17.7 / 21.1    28.5 / 22.2    30.7 / 32.6
//   of other widths, one row: 4096 x 12288 (0.86) 13.0 / 11.0, 14.9 / 15.4, 18.9 / 15.9, 15.1 / 13.1; 8192 x 12288 (0.86) 20.9 / 18.5, 24.5 / 27.2, 29.8 / 27.5, 22.8 / 19.8;
//     49152 x 1024 (0.86) 11.9 / 10.6, 13.8 / 13.9, 16.6 / 16.4, 12.7 / 12.6; 128256 x 1024 (0.97) 25.8 / 20.6, 29.7 / 28.6, 36.5 / 36.6, 27.9 / 26.2;
//     24576 x 2048 (0.65) 13.6 / 10.7, 15.6 / 13.9, 19.3 / 15.4, 14.8 / 12.8; three of 4096 x 4096 (0.65) 13.3 / 11.3, 15.4 / 15.2, 19.0 / 15.9, 14.6 / 12.5, of 2048 x 4096 8.1 / 8.2,
//     8.9 / 11.1, 11.5 / 11.6, 8.7 / 9.8
//   of two rows: 4096 x 12288 17.4 / 14.2, 19.3 / 17.2, 25.1 / 19.4, 19.9 / 19.1; 8192 x 8192 (0.86) 17.2 / 16.1, 18.9 / 19.6, 24.4 / 22.8, 18.4 / 21.4; 8192 x 12288 24.0 / 24.3, 27.2 / 29.3,
//     35.7 / 31.3, 26.1 / 28.3; 49152 x 1024 12.5 / 13.2, 14.6 / 15.9, 17.8 / 20.0, 13.5 / 15.1; 24576 x 2048 14.6 / 12.6, 17.3 / 15.3, 21.3 / 19.1, 15.9 / 15.1; twice 14336 x 2048 (0.76)
//     15.1 / 13.4, 17.8 / 16.5, 22.0 / 20.2, 16.5 / 17.2
//   four rows  a mat-vec: 3072 rows 8.6 / 8.8, 4096 9.9 / 9.0, 12288 17.4 / 16.5 (Q4_0); 5120 x 5120 12.7 / 13.5, 4096 x 8192 13.7 / 15.5;
//              several: 4096 + 1024 + 1024 rows (0.65) 11.7 / 10.7, twice 6144 (0.65) 15.8 / 16.6, twice 12288 (0.65) 30.1 / 25.7, twice 8192
//              (0.86) 16.3 / 18.9.  Of different widths, 12288 x 2048 + 12288 x 4096: 19.9 / 22.4, one row of Q6_K 20.4 / 22.5
//   Q4_K, three and four rows: 4096 (0.43) 12.2 / 10.8, 12288 (0.65) 17.3 / 18.8, 24576 (0.65) 32.6 / 28.0, 8192 (0.86) 13.7 / 17.4,
//              5120 x 2048 (0.54) 7.9 / 8.9, 24576 x 2048 (0.65) 18.0 / 17.8
//   Q4_K, five and more: 1024 (0.22) 20.0 / 8.4, 8192 (0.43) 27.6 / 23.8, 10240 (0.54) 28.5 / 28.2, 12288 (0.65) 28.5 / 32.9, 16384 (0.86)
//              28.6 / 41.7.  In groups of eight, one launch against one per group: 16 rows 10240 56.7 / 51.5, 12288 56.2 / 61.1; a last group
//              of one row costs this kernel as much as eight: 9 rows 4096 (0.22) 34.4 / 25.0, 6144 (0.32) 28.6 / 35.2.
//              (More than eight rows come here only where the kernel of qmv_wide.cu does not take them: matrices below 2^20 values, and weights
//              that do not start on 16-byte boundaries.)
bool qmv_split_pays(int ggml_type, const QmvArgs *ops, int nops, double fill) {
    uint64_t values = 0;
    uint32_t m = 0, kmin = 0xFFFFFFFFu, kmax = 0;
    for (int i = 0; i < nops; i++) {
        values += (uint64_t)ops[i].n * ops[i].k;
        m = ops[i].m > m ? ops[i].m : m;
        kmin = ops[i].k < kmin ? ops[i].k : kmin;
        kmax = ops[i].k > kmax ? ops[i].k : kmax;
    }
    constexpr uint64_t M = 1u << 20;
    const bool q4k = ggml_type == GT_Q4_K;
    if (kmin != kmax) return false;   // (the other kernel deals out work by K stages, and its passes are fuller than `fill` says)
    // One and two rows, in integers.  (What is more than 5 percent faster here and still leaves by the other kernel: Q4_K of one row from 40 M on, two rows of
    // 10240 to 20480 x 4096 of the other types below the limits, long rows of few.)
    if (q4k && m <= 2) return fill <= 0.7 && values >= 72 * M && (m == 1 || kmax >= 4096);
    if (m <= 1 && nops > 2) return values >= 40 * M;
    if (m <= 1 && ggml_type == GT_Q6_K && kmax < 2048) return false;
    if (m <= 1 && ggml_type == GT_Q8_0) return fill <= 0.7 ? values >= 30 * M : values >= 60 * M && kmax <= 8192;
    if (m <= 1) return values >= (fill > 0.7 ? 40 * M : 24 * M);
    if (m <= 2 && ggml_type == GT_Q8_0) return fill <= 0.75 && values >= 72 * M && kmax >= 4096;   // (twice 13824 x 5120, 0.73: a layer 88 us, so 83)
    if (m <= 2 && ggml_type == GT_Q6_K) return kmax >= 2048 && values >= (fill > 0.8 && kmax <= 4096 ? 90 * M : 40 * M);
    if (m <= 2) return values >= 60 * M && (fill <= 0.7 || kmax <= 8192);
    if (q4k && m <= 4) return kmax >= 4096 && values >= 14 * M && (fill <= 0.6 || (fill <= 0.7 && values >= 72 * M));
    if (q4k) return fill <= 0.6 && (m <= 8 || fill <= 0.25 || (m + 7) / 8 * 16 <= 3 * m);
    if (m > 4) return false;
    const bool alone = nops == 1 && ops[0].n_peer == 0;
    const bool four_bits = ggml_type == GT_Q4_0 && values >= 32 * M && values < 72 * M;
    return values >= 14 * M && kmax <= (ggml_type == GT_Q6_K ? 6144u : 4096u) && (alone || fill <= (four_bits ? 0.6 : 0.7));
}

// Whether an expert-routed call leaves by this kernel; `mma`: the register-level kernel takes it too (up to 16 pairs).  Between those two
// the matrix decides and not the number of pairs, since a pair's sum must not depend on the pairs that travel with it.  Graph replay of
// dependent launches, 128 experts (two and four pairs: 8 and 16), us with the other kernel / with this one:
//   register-level (a pass over the weights for every pair, 16 pairs a launch), gate and up of a layer, n < k:
//             768 x 2048, pairs: 2           4             8             16            1536 x 2048, 8   16            512 x 1024, 8   16
//     Q4_0                       7.5 / 8.1   9.1 / 9.0     12.2 / 11.4   25.2 / 16.2   19.3 / 16.5      39.9 / 26.9   8.6 / 8.9       11.7 / 10.0
//     Q8_0                       7.6 / 8.4   9.3 / 8.9     12.2 / 11.8   26.0 / 17.3   19.9 / 17.8      41.4 / 29.0   8.6 / 9.0       11.7 / 10.7
//     (the others lose more with few pairs, 1536 x 2048 four: Q4_K 10.2 / 12.4, Q5_K 11.8 / 16.7, Q6_K 12.2 / 13.7, and gain nothing with eight,
//     768 x 2048: 12.7 / 12.8, 14.2 / 17.2, 14.2 / 14.5; their 16 pairs, 26.0 / 18.8 for Q4_K, pay for that)
//   register-level, down projection, n >= k: 2048 x 768 eight pairs 7.7 / 10.2 (Q4_0), 8.7 / 11.0 (Q8_0), 16 pairs 14.4 / 14.1, 14.8 / 14.8;
//     2048 x 1536 eight 10.2 / 14.6, 16 18.6 / 22.2
//   streaming (a pass for every pair as well), Q6_K rows off 16-byte boundaries: 2048 x 768 two pairs 6.6 / 9.9, eight 12.1 / 12.5, 16
//     20.6 / 20.2, 256 267 / 109; 2048 x 1536, whose copies cost this kernel more, 16 pairs of 16 experts 21.4 / 26.8, 64 of 128 72.6 / 74.2, 64
//     of 64 72.1 / 63.4, 64 of 8 68.9 / 40.2; 2048 x 3584 64 of 64 141 / 149, 128 of 128 273 / 269, 256 of 128 540 / 392
//   streaming or plain, the other types, 32 pairs: 2048 x 1536 Q4_0 41 / 31, 768 x 2048 Q4_K 110 / 31.
bool qmv_split_pays_routed(int ggml_type, const QmvArgs &a, bool mma) {
    if (mma) return (ggml_type == GT_Q4_0 || ggml_type == GT_Q8_0) && a.n < a.k && (uint64_t)a.n * a.k >= 5u << 18;
    if (ggml_type == GT_Q6_K && !qmv_split_aligned(ggml_type, a))
        return a.k <= 1024 ? a.nprob > 8 : a.nprob >= 64 && a.nprob >= (a.k > 2560 ? 2ull : 1ull) * a.n_experts;
    return true;
}

// Scratch for the packed activations of a launch (one activation row, and routed rows, are converted inside the kernel).
size_t qmv_split_scratch_bytes(const QmvArgs *ops, int nops) {
    size_t n = 0;
    for (int i = 0; i < nops; i++)
        if (!ops[i].ids && ops[i].m > 2) n += sp_pack_bytes<GT_Q4_K>(ops[i].m, ops[i].k);   // (a type with sums)
    return n;
}

cudaError_t launch_qmv_split(int ggml_type, const QmvArgs *ops, int nops, int sm_count, uint8_t *scratch, int *launches, cudaStream_t st) {
    switch (ggml_type) {
    case GT_Q4_0: return sp_run<GT_Q4_0>(ops, nops, sm_count, scratch, launches, st);
    case GT_Q8_0: return sp_run<GT_Q8_0>(ops, nops, sm_count, scratch, launches, st);
    case GT_Q4_K: return sp_run<GT_Q4_K>(ops, nops, sm_count, scratch, launches, st);
    case GT_Q5_K: return sp_run<GT_Q5_K>(ops, nops, sm_count, scratch, launches, st);
    case GT_Q6_K: return sp_run<GT_Q6_K>(ops, nops, sm_count, scratch, launches, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace mlxn

extern "C" int mlxn_debug_split_geometry(const mlxn_qmm_id_params *p, uint32_t misaligned, uint32_t sm_count, uint32_t *ranks, uint32_t *tiles) {
    using namespace mlxn;
    if (!p || !ranks || !tiles || sm_count == 0) return MLXN_INVALID_ARGUMENT;
    QmvArgs a{};
    const uint32_t none = 0;
    a.w = reinterpret_cast<const uint8_t *>((uintptr_t)1024 + misaligned);   // (addresses are looked at, not read)
    a.n = p->n;
    a.k = p->k;
    a.m = p->n_experts ? 1 : p->n_tokens;
    a.nprob = p->n_experts ? p->n_tokens * p->top_k : 1;
    a.ids = p->n_experts ? &none : nullptr;
    a.n_experts = p->n_experts;
    a.expert_stride = p->expert_stride;
    SpPick pick{0, 0};
    const bool taken = qmv_split_fits((int)p->ggml_type, a, (int)sm_count, &pick);
    *ranks = taken ? pick.ranks : 0;
    *tiles = taken ? pick.tr : 0;
    return MLXN_OK;
}
