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
    const bool packed = !routed && mp > 1;
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
    if (kq && !aligned) return false;
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

// Scratch for the packed activations of a launch (one activation row, and routed rows, are converted inside the kernel).
size_t qmv_split_scratch_bytes(const QmvArgs *ops, int nops) {
    size_t n = 0;
    for (int i = 0; i < nops; i++)
        if (!ops[i].ids && ops[i].m > 1) n += sp_pack_bytes<GT_Q4_K>(ops[i].m, ops[i].k);   // (a type with sums)
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
