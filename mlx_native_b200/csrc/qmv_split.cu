// Dispatcher of the split mat-vec (qmv_split.cuh).
#include "qmv_split.cuh"

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

bool qmv_split_supported(int ggml_type, const QmvArgs &a) {
    const bool kq = ggml_type == GT_Q4_K || ggml_type == GT_Q5_K;
    if (ggml_type != GT_Q4_0 && ggml_type != GT_Q8_0 && ggml_type != GT_Q6_K && !kq) return false;
    if (a.m == 0 || a.n == 0 || a.k == 0 || a.k % ggml_qk(ggml_type) != 0) return false;
    // the activations are read as pairs of floats
    if (((uintptr_t)a.x & 7u) || ((uintptr_t)a.x2 & 7u) || ((uintptr_t)a.w & 1u)) return false;
    if (kq && !qmv_split_aligned(ggml_type, a)) return false;
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
    // the activations of a K slice (256 bytes per 64 values and row, and the bias sums) beside the smallest ring: two stages of
    // one tile (at most 14.1 KB each), the scale table (2 KB) and the partial sums (up to 6 KB)
    const uint32_t slice = (((a.k + 63) / 64 + ranks - 1) / ranks + 3) / 4 * 4 + 2;
    return (uint64_t)slice * mp * (256 + 16) + 40 * 1024 <= kSpSmem && encode_tiled_fn() != nullptr;
}

// Scratch for the packed activations of a launch (one activation row, and routed rows, are converted inside the kernel).
size_t qmv_split_scratch_bytes(const QmvArgs *ops, int nops) {
    size_t n = 0;
    for (int i = 0; i < nops; i++)
        if (!ops[i].ids && ops[i].m > 1) n += sp_pack_bytes<GT_Q6_K>(ops[i].m, ops[i].k);   // (the type with the most bias sums)
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
