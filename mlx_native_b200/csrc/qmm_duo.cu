// Mat-mat of many activation rows on pairs of SMs, dense or grouped by expert: y[m, n] = x[m, k] . W[n, k]^T, weights dequantised on the way.
//
// The kernel of qmm.cu gives every SM a tile of 128 weight rows and up to 256 activation rows.  At 256 its tensor core is held up by
// shared memory: it reads the activation tile (8 KB) for every 16 K values, the bulk copies write as much, and the raw weights come on
// top -- 1070 cycles for 64 K values where the multiplication needs 410.  Here two SMs work on one tile of 256 weight rows
// (tcgen05 cta_group::2): each dequantises its own 128 rows into its own tensor memory and holds half of the activation tile, which the
// hardware reads from both.  Operand semantics as in qmm.cu: exact weights rounded once to f16, activations f32 -> f16, f32 sums.
//
// Graph replay of dependent calls, packing included, us with qmm.cu / here (K 4096 unless said): 4096 weight rows: 9 rows 18.9 / 15.5, 64 20.9 / 17.8,
// 256 24.3 / 20.8, 512 31.1 / 26.8; 12288 x 512 rows 66.7 / 49.0; 1024 x 512 22.4 / 18.8; 4096 x 12288, 2048 rows: Q4_0 205 / 178, Q6_K 229 / 190;
// 256 x 512 x 16 rows 8.6 / 8.0.  So it takes every call it can: what has no 16-byte aligned weights, or a row count that its copies cannot group,
// stays with the other kernel, and the row-sharded form.  What bounds it: up to 192 rows the chain raw block -> tensor memory (0.47 us for a
// K stage of 128, 18 values a cycle and SM; Q6_K 0.66 before its 64 values of a thread were unpacked together: 64 rows 21.0 -> 19.9
// us), above that the multiplication (0.43 us at full clock) beside it.
//
// The items of grouped calls are short (64 rows, K of 6 to 16 stages), and while the dequantising warps read an accumulator back both they and the
// tensor core would stand still; there the read-back has warps of its own and two accumulators.  (Dense calls gain nothing from it, Q4_0 2048 x 4096 x
// 4096 61.4 / 62.4 us, and Q6_K loses, 128 x 4096 x 4096 19.8 / 22.2.)  Layer of 512 tokens, 8 of 128 experts each, Q4_0 768 x 2048 twice and Q6_K
// 2048 x 768: 273 us for the whole pass with two CTAs of qmm.cu's kernel on an SM (half of the dequantising warps each), 228 here; weights once at the
// copy rate 61.  Batches: q, k and v of 512 rows (4096, 1024 and 1024 x 4096) and gate and up (12288 x 4096 each) in one launch took a layer from 274
// to 244 us: one packing instead of three and two, and one last wave.
//
// Sums: chains of additions in an accumulator are kept about as short as on single SMs (qmm.cuh): dense tiles have two accumulators up to 192 rows and
// four up to 64, one K stage each in turn.  Relative error of the sums (64 bits of the operands as rounded to f16), one accumulator / this: 512 and
// 333 x 4096 x 4096 4.8e-6 / 2.4e-6, 60 x 1024 x 4096 2.4e-6 / 1.2e-6, 512 x 12288 x 4096 4.8e-6 / 2.4e-6; a batch may have twice what its
// products have alone (k and v of 512 rows 2.4e-6, 1.2e-6).  It costs 0.6 us a call: 512 x 4096 x 4096 25.8 / 26.6, 64 rows 17.1 / 17.9.  Also tried: a
// tile in parts that are added to y, 3.5 us each at 192 rows (q, k and v 28.3 / 32.4); tiles whose read-back waits for the next one's first
// stages, no gain (64 rows 18.7).
//
// Order: the activations' copies of both CTAs complete on CTA 0's barrier.  With bulk copies onto barriers of their own and a relaxed arrival in between,
// which orders nothing in shared memory, 2048 rows took 1.5 % less (Q6_K 187 / 190), others the same.
//
// What else was tried: unpacking the weights once into f16 tiles, by a kernel of its own.  The product alone then runs at the
// multiplication's rate, but the unpacking is bound by memory (13 us for 4096 x 4096, 58 with 2048 rows of 12288 for 4096 x 12288): 32.2 us in
// all for 512 x 4096 x 4096, 72.8 for 512 x 12288 x 4096.  K in two and four parts over clusters of two and four pairs,
// summed through distributed shared memory instead of atomics: 16.2 us for 128 x 4096 x 4096 where halves with atomics take 15.4 (and only 15
// clusters of eight fit on the chip).  Announcing a stage after the next one's arithmetic instead of waiting for its store: 1 to 4 % slower.
#include <cuda_fp16.h>

#include <atomic>

#include "common.cuh"
#include "dequant.cuh"
#include "ptx.cuh"
#include "qmm.cuh"
#include "tensor_map.cuh"

namespace mlxn {

constexpr uint32_t kDuoRows = 256;                          // weight rows of a pair's tile
constexpr uint32_t kDuoDequantWarps = 16;                   // two sets of eight; set s takes the 128-wide K stages st % 2 == s
// Warps that read the accumulators back: of their own where tiles are short (routed), else the dequantising ones.
__host__ __device__ constexpr uint32_t duo_read_warps(bool routed) { return routed ? 4 : kDuoDequantWarps; }
__host__ __device__ constexpr uint32_t duo_threads(bool routed) { return (4 + kDuoDequantWarps + (routed ? duo_read_warps(true) : 0)) * 32; }
constexpr uint32_t kDuoStages = 4;                          // ring of K stages, activations in shared memory
// Tensor memory: accumulators from column 0 on, weights from the last column down, 64 columns a stage (128 f16 values).
constexpr uint32_t kDuoCols = 512, kDuoACols = 64;
static_assert(kDuoStages % 2 == 0, "a ring of two stages in tensor memory takes every other place of the ring in shared memory");
constexpr uint32_t kDuoMaxRaw = 5;

struct DuoCfg {
    uint32_t nchunks;     // ceil(k / 64)
    uint32_t nt;          // activation rows of a tile (a multiple of 32, at most 256)
    uint32_t n_wt, ntiles;
    uint32_t pairs;
    uint32_t accs;        // dense: accumulators that take turns, nt columns each; a power of two
    TcShare share;        // the pairs' ranges where tiles are shared
    uint32_t seg_stride;  // bytes of a raw row segment in shared memory
    uint32_t raw_off, raw_slots;
    uint32_t row_group;   // log2 of the copies of a raw stage (see launch_tc_tn)
    uint32_t aligned;     // every weight row starts on a 16-byte boundary
    uint32_t beside;      // nothing here depends on the kernel ahead, whose own dependences have been waited for: wait for it in the end
    TcOut out;
};
struct DuoMaps {
    CUtensorMap m[kMmOps];   // weights of the products
    CUtensorMap x;           // packed activations: [64-wide chunks][8-row groups of 1 KB][256 words]
};

namespace duo {
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool elect() {
    uint32_t p = 0;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\t@p mov.u32 %0, 1;\n\t}" : "+r"(p));
    return p != 0;
}
__device__ __forceinline__ uint32_t in_cta_0(uint64_t *bar) {   // the barrier at the same place in CTA 0
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(bar)));
    return a;
}
// Arrives on the barrier at the same place in CTA 0.  Relaxed: what it announces are loads and stores of tensor memory only, which the fences of
// tcgen05 before it and behind the wait for it order (with release the instruction takes a thousand cycles, which then bounded the whole kernel).
// Nothing in shared memory may be announced so: the activations' copies complete on CTA 0's barriers themselves.
__device__ __forceinline__ void arrive_at_0(uint64_t *bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta_0(bar)) : "memory");
}
// Tensor copy into this CTA's shared memory that completes on a barrier of either CTA of the pair.
__device__ __forceinline__ void copy_3d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map),
                 "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void alloc(uint32_t *dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols) : "memory");
}
__device__ __forceinline__ void relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// D (+)= A B^T of the pair: A in the tensor memory of both CTAs (128 rows each), B's halves in their shared memory
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this place in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void commit_both(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
}  // namespace duo

// Clusters of two CTAs, one CTA per SM, persistent.  Per CTA:
//   warp 0        activations: one tensor copy per K stage (two 64-wide chunks of its half of the tile), which completes on CTA 0's barrier
//   warp 1        CTA 0: MMAs of the pair, whose completion frees the stage's places in both CTAs; CTA 1: tells CTA 0 that its stage is ready
//   warp 2        raw weights: tensor copies of 128 rows x 256 K values
//   warps 4..19   dequantise raw blocks into tensor memory; dense: read the accumulator back
//   warps 20..23  routed: read the accumulators back, two in turn, so that the next item's multiplications go on
// Ring places and barrier phases run on across the items of a pair.
//
// ROUTED: the products of a mixture of experts.  The tiles are those of the list that build_tiles_kernel made, 64 rows of one expert each,
// packed whole (a CTA's half are rows 0..31 or 32..63 of each 64-column chunk); the weights' map has the expert as third dimension.
// RING: K stages of weights in tensor memory, 64 columns each.  The accumulators have what is left: two of 129 to 192 columns leave two stages.
// RAW: weight rows lie in tensor memory as in a raw stage (see row_of).
template <int T, bool ROUTED, uint32_t RING, bool RAW>
__global__ void __launch_bounds__(768, 1) __cluster_dims__(2, 1, 1)   // (at most 80 registers: a block of the packing kernel fits beside a CTA)
    qmm_duo_kernel(const QmmArgs a, const __grid_constant__ DuoCfg c, const __grid_constant__ DuoMaps wmaps) {
    constexpr int QK = BlockTraits<T>::QK, BB = BlockTraits<T>::BYTES;
    constexpr uint32_t KR = 256, kReadWarps = duo_read_warps(ROUTED), accs = ROUTED ? 2 : 1;   // (items that are in accumulators, 128 columns apart)
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // (the same in both CTAs)
    __shared__ __align__(8) uint64_t full[kDuoStages], peer_full[kDuoStages], done[kDuoStages], raw_full[kDuoMaxRaw], raw_empty[kDuoMaxRaw];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ volatile uint32_t abort_flag;
    const uint32_t lane = threadIdx.x & 31u, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const uint32_t rank = duo::cluster_rank(), pair = blockIdx.x >> 1;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (uint32_t s = 0; s < kDuoStages; s++) {
            mbar_init(&full[s], rank == 0 ? 9 : 8);   // the eight warps of a set; CTA 0: and the activations' copies, both halves
            mbar_init(&peer_full[s], 1);
            mbar_init(&done[s], 1);
        }
        for (uint32_t s = 0; s < c.raw_slots; s++) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], kDuoDequantWarps);
        }
        for (uint32_t s = 0; s < 2; s++) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 2 * kReadWarps);   // (of CTA 0: the warps of both)
        }
        mbar_init_fence();
    }
    if (warp == 3) {
        duo::alloc(&tmem_s, 512);
        duo::relinquish();
    }
    tc_fence_before();
    __syncthreads();
    duo::cluster_sync();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    if (!c.beside) {
        grid_dependency_wait();   // the packed activations, the tile list and the zeros of shared tiles are complete
    } else {
        // ... which they were for every block of the kernel ahead before it let this one be launched: taken over from it, for loads and for copies
        __threadfence();
        fence_proxy_async();
    }
    allow_dependents();

    // ---- work items: weight tile fastest, so that the pairs working at the same time share an activation tile in L2 ----
    const uint32_t nraw_all = (a.k + KR - 1) / KR, total_items = c.n_wt * (ROUTED ? min(__ldcg(a.tiles), c.ntiles) : c.ntiles);
    const bool shared = !ROUTED && c.share.ctas != 0;
    const uint32_t pos0 = shared ? c.share.begin(pair) : pair, pos1 = shared ? c.share.begin(pair + 1) : total_items;
    struct Item {
        uint32_t tt, op, n0, r_lo, nraw, nst, kc_lo, nck, next;
    };
    auto load_item = [&](uint32_t pos) {
        Item it;
        const uint32_t item = shared ? pos / nraw_all : pos;
        it.r_lo = shared ? pos - item * nraw_all : 0u;
        const uint32_t r_hi = shared ? min(nraw_all, it.r_lo + (pos1 - pos)) : nraw_all;
        it.next = shared ? pos + (r_hi - it.r_lo) : pos + c.pairs;
        it.tt = item / c.n_wt;
        uint32_t wt = item - it.tt * c.n_wt;
        it.op = c.out.find(wt);
        it.n0 = wt * kDuoRows + rank * 128u;
        it.nraw = r_hi - it.r_lo;
        it.kc_lo = it.r_lo * (KR / 64);
        it.nst = min((a.k + 127) / 128, r_hi * (KR / 128)) - it.r_lo * (KR / 128);   // K stages of 128
        it.nck = min(c.nchunks, r_hi * (KR / 64)) - it.kc_lo;                         // 64-wide chunks
        return it;
    };
    const uint32_t h = c.nt / 2, b_chunk = h * 128u, b_stage = 2 * b_chunk;
    const uint32_t smem_base = smem_u32(smem), raw_bytes = 128u * c.seg_stride;
    constexpr uint32_t kSpin = 0xFFFFFFFFu;
    bool ok = true;

    // The weight row (of the CTA's 128) in tensor-memory lane p.  RAW, for Q6_K whose rows do not all start on 16-byte boundaries: as in a raw stage,
    // those that start alike one after another, so that a warp's rows are neighbours in shared memory and, with two ways to start, start
    // alike (in the matrix's order every second, fourth or eighth row of a warp meets in the same banks, and extraction is by 4-byte loads).
    auto row_of = [&](uint32_t p) { return RAW ? ((p & ((128u >> c.row_group) - 1u)) << c.row_group) + (p >> (7 - c.row_group)) : p; };

    // The read-back of the pair's `nitem`-th item, by group g of four warps: lane = weight row, 32 activation rows at a time, the groups in turn.
    auto read_back = [&](const Item &it, uint32_t nitem, uint32_t q4, uint32_t g) {
        const uint32_t buf = accs == 2 ? nitem & 1u : 0u, turn = accs == 2 ? nitem >> 1 : nitem, n = c.out.n[it.op], rr = row_of(q4 * 32 + lane);
        const bool row_ok = it.n0 + rr < n;
        int32_t mine[2] = {-1, -1};   // ROUTED: the output rows of activation rows lane and 32 + lane of the tile
        if constexpr (ROUTED) {
            const uint32_t ex = __ldcg(a.tiles + 1 + 2 * it.tt), at0 = __ldcg(a.tiles + 2 + 2 * it.tt) * c.nt + lane;
            const uint32_t rows = min(__ldcg(a.htpe + ex), a.hids_stride);
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) {
                if (at0 + 32 * i < rows) {
                    mine[i] = __ldcg(a.hids + (size_t)ex * a.hids_stride + at0 + 32 * i);
                    if ((uint32_t)mine[i] >= a.total_rows) mine[i] = -1;
                }
            }
        }
        if (!mbar_wait(&acc_full[buf], turn & 1u, &abort_flag, a.status, ST_WAIT_MMA_TIMEOUT, 0u)) return false;
        tc_fence_after();
        [[maybe_unused]] const bool some = it.nraw < nraw_all;   // another pair has the rest of this tile's K
        [[maybe_unused]] const uint32_t used = min(c.accs, it.nst);
#pragma unroll 1
        for (uint32_t col = g * 32; col < c.nt; col += kReadWarps / 4 * 32) {
            uint32_t v[32];
            tmem_ld_32x32(tmem + ((q4 * 32) << 16) + buf * 128 + col, v);
            tmem_ld_wait();
            if constexpr (ROUTED) {   // (tiles of 64 rows: two turns)
                const int32_t rows = col ? mine[1] : mine[0];
                float *y = c.out.y[0] + it.n0 + rr;
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) {
                    const int32_t o = __shfl_sync(0xffffffffu, rows, j);
                    if (row_ok && o >= 0) y[(size_t)o * n] = __uint_as_float(v[j]);
                }
            } else {
#pragma unroll 1
                for (uint32_t i = 1; i < used; i++) {
#pragma unroll
                    for (uint32_t h = 0; h < 32; h += 16) {   // (16 at a time: with more registers the packing kernel's blocks do not fit beside a CTA)
                        uint32_t z[16];
                        tmem_ld_32x32_x16(tmem + ((q4 * 32) << 16) + i * c.nt + col + h, z);
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t j = 0; j < 16; j++) v[h + j] = __float_as_uint(__uint_as_float(v[h + j]) + __uint_as_float(z[j]));
                    }
                }
                const uint32_t o0 = it.tt * c.nt + col;
                if (row_ok && o0 < a.m) {
                    float *y = c.out.y[it.op] + (size_t)o0 * n + it.n0 + rr;
                    const uint32_t cnt = min(32u, a.m - o0);
                    if (some) {
#pragma unroll
                        for (uint32_t j = 0; j < 32; j++)
                            if (j < cnt) atomicAdd(y + (size_t)j * n, __uint_as_float(v[j]));
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 32; j++)
                            if (j < cnt) y[(size_t)j * n] = __uint_as_float(v[j]);
                    }
                }
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) duo::arrive_at_0(&acc_empty[buf]);   // the MMA warp may start on another item here
        return true;
    };

    if (warp == 0) {
        uint32_t s = 0, ph = 1;   // (a place's first wait passes)
        for (uint32_t pos = pos0; ok && pos < pos1;) {
            const Item it = load_item(pos);
            pos = it.next;
            // (a K tail of 64 brings a chunk of the next tile, or zeros, which is not multiplied)
            uint32_t chunk = (ROUTED ? it.tt : it.tt * 2u + rank) * c.nchunks + it.kc_lo;
            for (uint32_t st = 0; st < it.nst; st++, chunk += 2) {
                if (!mbar_wait(&done[s], ph, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, kSpin)) {
                    ok = false;
                    break;
                }
                if (duo::elect()) {
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * b_stage);
                    duo::copy_3d(smem_base + s * b_stage, &wmaps.x, 0, ROUTED ? rank * 4 : 0, chunk, duo::in_cta_0(&full[s]));
                }
                __syncwarp();
                if (++s == kDuoStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc_f16(kDuoRows, c.nt);
        const uint64_t bd0 = umma_desc_k_sw128(smem_base);
        uint32_t s = 0, ph = 0, nitem = 0;
        for (uint32_t pos = pos0; ok && pos < pos1; nitem++) {
            const Item it = load_item(pos);
            pos = it.next;
            const uint32_t buf = accs == 2 ? nitem & 1u : 0u, turn = accs == 2 ? nitem >> 1 : nitem, turns = ROUTED ? 1u : c.accs;
            // the accumulator's item before has been read back
            if (rank == 0 && !mbar_wait(&acc_empty[buf], (turn & 1u) ^ 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, kSpin)) break;
            tc_fence_after();
            for (uint32_t st = 0; st < it.nst; st++) {
                if (!mbar_wait(&full[s], ph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, kSpin)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (rank == 0) {
                    if (!mbar_wait(&peer_full[s], ph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, kSpin)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (duo::elect()) {
                        const uint32_t d = tmem + (ROUTED ? buf * 128 : (st & (turns - 1u)) * c.nt);   // (dense: accumulators take turns)
                        const uint32_t ac = tmem + kDuoCols - kDuoACols - s % RING * kDuoACols;
                        const uint64_t bd = bd0 + s * (b_stage >> 4), bd1 = bd + (b_chunk >> 4);
#pragma unroll
                        for (uint32_t q = 0; q < 4; q++) duo::mma(d, ac + 8 * q, bd + 2 * q, idesc, st >= turns || q ? 1u : 0u);
                        if (2 * st + 1 < it.nck) {
#pragma unroll
                            for (uint32_t q = 0; q < 4; q++) duo::mma(d, ac + 32 + 8 * q, bd1 + 2 * q, idesc, 1u);
                        }
                        duo::commit_both(&done[s]);
                    }
                } else {
                    tc_fence_before();
                    if (duo::elect()) duo::arrive_at_0(&peer_full[s]);
                }
                __syncwarp();
                if (++s == kDuoStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (!ok) break;
            if (rank == 0 && duo::elect()) duo::commit_both(&acc_full[buf]);
            __syncwarp();
        }
    } else if (warp == 2) {
        // (see qmm.cu: a map row is a group of 1, 2, 4 or 8 weight rows that starts on a 16-byte boundary; one copy brings a row of every group)
        const uint32_t row_bytes = (a.k / QK) * BB;
        uint32_t slot = 0, ph = 1;
        for (uint32_t pos = pos0; ok && pos < pos1;) {
            const Item it = load_item(pos);
            pos = it.next;
            const uint32_t ex = ROUTED ? __ldcg(a.tiles + 1 + 2 * it.tt) : 0u;
            for (uint32_t r = 0; r < it.nraw; r++) {
                if (!mbar_wait(&raw_empty[slot], ph, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, kSpin)) {
                    ok = false;
                    break;
                }
                if (duo::elect()) {
                    const uint32_t kb = (it.r_lo + r) * (KR / QK) * BB;
                    mbar_expect_tx(&raw_full[slot], raw_bytes);
                    for (uint32_t i = 0; i < 1u << c.row_group; i++)
                        asm volatile(
                            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                                smem_base + c.raw_off + slot * raw_bytes + i * (raw_bytes >> c.row_group)),
                            "l"(&wmaps.m[it.op]), "r"(((i * row_bytes + kb) & ~15u) >> 2), "r"(it.n0 >> c.row_group), "r"(ex), "r"(smem_u32(&raw_full[slot]))
                            : "memory");
                }
                __syncwarp();
                if (++slot == c.raw_slots) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp >= 4 && warp < 4 + kDuoDequantWarps) {
        // thread (warp w, lane l) of a set owns the weight row of lane 32 (w % 4) + l, the tensor-memory lane it may address, and the 64-element half
        // (w / 4) % 2 of the K stage: 32 packed f16 pairs = one 32-column store
        const uint32_t dw = warp - 4, q4 = dw & 3u, half = (dw >> 2) & 1u, set = dw >> 3;
        const uint32_t rr = row_of(q4 * 32 + lane);
        const uint32_t srow = ((rr & ((1u << c.row_group) - 1u)) << (7 - c.row_group)) + (rr >> c.row_group);   // the row's place in a raw stage
        const uint32_t a_dst = tmem + ((q4 * 32) << 16) + kDuoCols - kDuoACols + 32 * half;
        const uint32_t row_bytes = (a.k / QK) * BB;
        uint32_t rs = 0, rph = 0, J0 = 0, nitem = 0;
        for (uint32_t pos = pos0; ok && pos < pos1; nitem++) {
            const Item it = load_item(pos);
            pos = it.next;
            const bool row_ok = it.n0 + rr < c.out.n[it.op];
            const uint32_t row_lo4 = (it.n0 + rr) * row_bytes & 15u;   // (the weights start on a 16-byte boundary)
            for (uint32_t r = 0; r < it.nraw; r++) {
                if (!mbar_wait(&raw_full[rs], rph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, 0u)) {
                    ok = false;
                    break;
                }
                const uint32_t st = 2 * r + set;
                if (st < it.nst) {
                    const uint32_t J = J0 + st, sa = J % kDuoStages, before = J - RING;   // (J: the stage's number in the pair's whole run)
                    const uint32_t r_abs = it.r_lo + r, stage_row = smem_base + c.raw_off + rs * raw_bytes + srow * c.seg_stride;
                    uint32_t regs[32];
                    if (!RAW && c.aligned && row_ok) {
                        if constexpr (T == GT_Q4_K) {
                            dequant32_q4k_aligned(stage_row, 4 * set + 2 * half, regs);
                            dequant32_q4k_aligned(stage_row, 4 * set + 2 * half + 1, regs + 16);
                        } else if constexpr (T == GT_Q6_K) {
                            dequant64_q6k_aligned_p(r_abs & 7u, stage_row, set, half, regs);
                        } else {
                            switch (2 * set + half) {  // uniform per warp
                            case 0: dequant64_aligned<T, 0>(stage_row, regs); break;
                            case 1: dequant64_aligned<T, 1>(stage_row, regs); break;
                            case 2: dequant64_aligned<T, 2>(stage_row, regs); break;
                            default: dequant64_aligned<T, 3>(stage_row, regs); break;
                            }
                        }
                    } else if constexpr (RAW) {
                        // (With four ways to start a warp's rows start alike too, but then four of the eight versions take turns: 1024 x 2560 160 us, so 128.)
                        if (c.row_group < 2) dequant64_q6k_aligned_p((row_lo4 + r_abs * BB) >> 1 & 7u, stage_row, set, half, regs);
                        else dequant64_q6k_any(stage_row + ((row_lo4 + r_abs * BB) & 15u), set, half, regs);
                    } else {
                        const uint32_t seg = stage_row + ((row_lo4 + ((r_abs * KR) / QK) * BB) & 15u);
#pragma unroll
                        for (uint32_t hh = 0; hh < 2; hh++) {
                            uint4 v[4];
                            const uint32_t e0 = 128 * set + 64 * half + 32 * hh;
                            if (row_ok && r_abs * KR + e0 < a.k) {
                                dequant32<T>(seg, e0, v);
                            } else {
#pragma unroll
                                for (int i = 0; i < 4; i++) v[i] = make_uint4(0, 0, 0, 0);
                            }
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                regs[16 * hh + 4 * i + 0] = v[i].x;
                                regs[16 * hh + 4 * i + 1] = v[i].y;
                                regs[16 * hh + 4 * i + 2] = v[i].z;
                                regs[16 * hh + 4 * i + 3] = v[i].w;
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[rs]);   // this warp is done reading the raw stage
                    // the MMAs that read this place's previous contents have completed
                    if (J >= RING && !mbar_wait(&done[before % kDuoStages], (before / kDuoStages) & 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, 0u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    tmem_st_32x32_x32(a_dst - J % RING * kDuoACols, regs);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[sa]);
                } else {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[rs]);
                }
                if (++rs == c.raw_slots) {
                    rs = 0;
                    rph ^= 1u;
                }
            }
            if (!ok) break;
            J0 += it.nst;
            if constexpr (!ROUTED) {
                if (!read_back(it, nitem, q4, dw >> 2)) break;
            }
        }
    } else if (ROUTED && warp >= 4 + kDuoDequantWarps) {
        const uint32_t q4 = warp & 3u, g = (warp - 4 - kDuoDequantWarps) >> 2;
        uint32_t nitem = 0;
        for (uint32_t pos = pos0; pos < pos1; nitem++) {
            const Item it = load_item(pos);
            pos = it.next;
            if (!read_back(it, nitem, q4, g)) break;
        }
    }
    __syncwarp();
    if (abort_flag)   // let copies in flight land before the shared memory is released
        for (int i = 0; i < 200; i++) __nanosleep(5000);
    if (c.beside) grid_dependency_wait();   // (what comes behind waits for this kernel only)
    tc_fence_before();
    __syncthreads();
    duo::cluster_sync();   // nobody leaves while the other may still arrive here, or while the pair's MMAs read here
    if (warp == 3) {
        tc_fence_after();
        duo::dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// Pairs of SMs that hold a cluster at the same time.
static uint32_t duo_pairs() {
    static std::atomic<uint32_t> known[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t most = (uint32_t)sm_count_of_device() / 2;
    if (dev < 0 || dev >= 64) return most;
    uint32_t v = known[dev].load(std::memory_order_acquire);
    if (!v) {
        int n = 0;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(most * 2);
        cfg.blockDim = dim3(duo_threads(false));
        cfg.dynamicSmemBytes = 223 * 1024;
        if (cudaFuncSetAttribute(qmm_duo_kernel<GT_Q4_0, false, 4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 223 * 1024) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, qmm_duo_kernel<GT_Q4_0, false, 4, false>, &cfg) != cudaSuccess || n < 1 || n > (int)most) {
            (void)cudaGetLastError();
            n = (int)most;
        }
        v = (uint32_t)n;
        known[dev].store(v, std::memory_order_release);
    }
    return v;
}

struct DuoPlan {
    uint32_t pairs, shared, accs;
};
// Cost in the units of tc_plan (1.74 ns).  Measured: a K stage of 128 values takes 0.47 us where dequantising bounds it (Q6_K 0.66), else
// 0.165 us + 2.3 ns per activation row; an item 1 us beside its stages.  Tiles shared by two pairs are zeroed and added up: 3 us and more for
// wide ones (every tile in halves), 5 us where ranges are shared.
// `limit`: see qmm_chain_limit.  As few accumulators as keep it; a plan that cannot is taken where the others cost 6 % more.
static uint64_t duo_plan(int type, uint64_t m, uint64_t n, uint64_t k, uint32_t nt, uint32_t limit, DuoPlan &p) {
    const uint64_t sms = duo_pairs(), nraw = (k + 255) / 256, tiles = (n + kDuoRows - 1) / kDuoRows * ((m + nt - 1) / nt);
    const uint64_t convert = type == GT_Q6_K ? 380 : 270, multiply = 95 + nt * 13 / 10, tile = 2 * nraw * (convert > multiply ? convert : multiply);
    const uint32_t room = nt <= 64 ? 4 : nt <= 192 ? 2 : 1;
    uint64_t best = ~0ull;
    auto offer = [&](uint64_t cost, uint32_t pairs, bool shared, bool halves) {
        DuoPlan q{pairs, shared, 1};
        auto chains = [&] { return chain_mean((uint32_t)nraw, halves ? 2 : 1, q.accs, tiles, shared && !halves ? sms - 1 : 0); };
        while (chains() > limit && q.accs < room) q.accs *= 2;
        if (chains() > limit) cost = cost * 106 / 100;
        if (cost < best) {
            best = cost;
            p = q;
        }
    };
    offer((tiles + sms - 1) / sms * (tile + 400) + 600, (uint32_t)(tiles < sms ? tiles : sms), false, false);
    if (tiles * nraw >= (1ull << 31) || nraw < 2) return best;
    if (tiles > sms) offer(tiles * tile / sms + (tiles / sms + 2) * 575 + 2900 + nt * 9, (uint32_t)sms, true, false);
    else if (2 * tiles <= sms) offer(tile / 2 + 2300 + nt * 12, (uint32_t)(2 * tiles), true, true);
    return best;
}

static int duo_row_group(uint32_t row_bytes) {
    int lg = 0;
    while ((row_bytes << lg) & 15u) lg++;
    return lg;
}
bool qmm_duo_takes(int ggml_type, const QmmArgs &a) {
    if (ggml_type != GT_Q4_0 && ggml_type != GT_Q8_0 && ggml_type != GT_Q6_K) return false;
    if (a.hids || a.y_ld || a.n_peer || a.x2 || a.k % 32 != 0) return false;
    const uint32_t row_bytes = (a.k / ggml_qk(ggml_type)) * ggml_block_bytes(ggml_type);
    return ((uintptr_t)a.w & 15u) == 0 && a.n % (1u << duo_row_group(row_bytes)) == 0 && encode_tiled_fn() != nullptr;
}
uint64_t qmm_duo_cost(int ggml_type, const QmmArgs &a, uint32_t nt, uint32_t limit) {
    if (nt % 32 != 0 || nt > 256 || !qmm_duo_takes(ggml_type, a)) return ~0ull;
    DuoPlan p;
    return duo_plan(ggml_type, a.m, a.n, a.k, nt, limit, p);
}

// Whether the rows go to tensor memory in the raw stages' order (RAW).  Results are then written with a stride: that pays where it is two rows (1024 x
// 4096 x 5120, 49.0 -> 44.4 us) and in routed products, whose read-back has warps of its own (512 tokens, 128 experts, 2048 x 768 95.7 -> 88.2, 1024 x 2560
// 141 -> 128), not with four or eight (2048 x 4096 x 2560: 52.4 -> 55.1), nor where results are added to another pair's (333 x 4096 x 4352: 29 -> 34).
static bool duo_raw_order(int ggml_type, uint32_t k, bool routed, bool shared) {
    const int g = duo_row_group((k / ggml_qk(ggml_type)) * ggml_block_bytes(ggml_type));
    return ggml_type == GT_Q6_K && g != 0 && (routed || (g == 1 && !shared));
}

// Maps, rings and launch.  `c`: tiles, products and pairs are filled in.
template <int T, bool ROUTED, uint32_t RING, bool RAW> static cudaError_t duo_launch(DuoCfg &c, const QmmArgs *ops, int nops, const uint8_t *xpack, cudaStream_t st, int *launches) {
    constexpr int QK = BlockTraits<T>::QK, BB = BlockTraits<T>::BYTES;
    const QmmArgs &a = ops[0];
    const uint32_t row_bytes = (a.k / QK) * BB;
    c.nchunks = (a.k + 63) / 64;
    c.row_group = (uint32_t)duo_row_group(row_bytes);
    c.aligned = row_bytes % 16 == 0 && a.k % 256 == 0;
    constexpr uint32_t kSeg = 256 / QK * BB;
    c.seg_stride = c.row_group == 0 && kSeg % 16 == 0 ? kSeg : ((kSeg + 14 + 15) / 16 | 1u) * 16;   // (an odd multiple of 16: see launch_tc_tn)
    alignas(64) DuoMaps wmaps;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return cudaErrorNotSupported;
    for (int i = 0; i < nops; i++) {
        const uint32_t lg = c.row_group;
        const cuuint64_t gdim[3] = {((uint64_t)row_bytes << lg) / 4, ops[i].n >> lg, ROUTED ? a.n_experts : 1u};
        const cuuint64_t gstride[2] = {(uint64_t)row_bytes << lg, ROUTED ? a.expert_stride : (uint64_t)ops[i].n * row_bytes};
        const cuuint32_t box[3] = {c.seg_stride / 4, 128u >> lg, 1}, estr[3] = {1, 1, 1};
        if (enc(&wmaps.m[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t *>(ops[i].w), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    {
        const uint32_t groups = c.nt / (ROUTED ? 8 : 16), box_groups = c.nt / 16;   // of a packed chunk, of a CTA's half
        const cuuint64_t gdim[3] = {256, groups, (uint64_t)c.ntiles * (ROUTED ? 1 : 2) * c.nchunks}, gstride[2] = {1024, groups * 1024ull};
        const cuuint32_t box[3] = {256, box_groups, 2}, estr[3] = {1, 1, 1};
        if (enc(&wmaps.x, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t *>(xpack), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    const uint32_t limit = 222 * 1024, b_bytes = kDuoStages * c.nt * 128u, raw_slot = 128 * c.seg_stride;
    c.raw_off = b_bytes;
    c.raw_slots = (limit - b_bytes) / raw_slot;
    if (c.raw_slots > kDuoMaxRaw) c.raw_slots = kDuoMaxRaw;
    if (c.raw_slots < 2) return cudaErrorInvalidConfiguration;
    size_t smem = (size_t)b_bytes + c.raw_slots * raw_slot + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;   // (one CTA per SM: it takes all of tensor memory)
    static std::atomic<uint32_t> prepared[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(qmm_duo_kernel<T, ROUTED, RING, RAW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 223 * 1024);
        if (e != cudaSuccess) return e;
        prepared[dev].store(1, std::memory_order_release);
    }
    (*launches)++;
    note_mat_mat(ROUTED ? "qmm_duo_id" : "qmm_duo", c.nt);
    return launch_overlapped(qmm_duo_kernel<T, ROUTED, RING, RAW>, dim3(2 * c.pairs), dim3(duo_threads(ROUTED)), smem, st, a, c, wmaps);
}

// `ops`: products of the same activations
template <int T>
static cudaError_t launch_duo_t(const QmmArgs *ops, int nops, uint32_t nt, uint32_t limit, uint8_t *xpack, cudaStream_t st, int *launches) {
    if (nops < 1 || nops > (int)kMmOps) return cudaErrorInvalidValue;
    const QmmArgs &a = ops[0];
    const uint32_t h = nt / 2, nraw = (a.k + 255) / 256, nchunks = (a.k + 63) / 64;
    DuoCfg c{};
    for (int i = 0; i < nops; i++) {
        c.n_wt += (ops[i].n + kDuoRows - 1) / kDuoRows;
        c.out.y[i] = ops[i].y;
        c.out.n[i] = ops[i].n;
        c.out.wt_end[i] = c.n_wt;
    }
    DuoPlan p;
    duo_plan(T, a.m, (uint64_t)c.n_wt * kDuoRows, a.k, nt, limit, p);
    c.nt = nt;
    c.ntiles = (a.m + nt - 1) / nt;
    c.pairs = p.pairs;
    c.accs = p.accs;
    if (p.shared) c.share = {p.pairs, c.n_wt, nraw, c.n_wt * c.ntiles * nraw, kDuoRows, nt};
    // activations in tiles of nt / 2 rows: a CTA's half of a tile
    uint32_t lanes = nchunks;
    const uint64_t slices = (uint64_t)2 * c.ntiles * ((h + kPackRows - 1) / kPackRows);
    while (lanes > 1 && (uint64_t)lanes * slices > 2048) lanes = (lanes + 1) / 2;
    (*launches)++;
    const cudaError_t e = launch_overlapped(pack_x_kernel<false>, dim3((unsigned)slices, lanes), dim3(256), 0, st, a, xpack, nchunks, h, c.share, c.out);
    if (e != cudaSuccess) return e;
    const bool deep = kDuoCols - c.accs * nt >= 4 * kDuoACols;
    if constexpr (T == GT_Q6_K)
        if (duo_raw_order(T, a.k, false, p.shared))
            return deep ? duo_launch<T, false, 4, true>(c, ops, nops, xpack, st, launches) : duo_launch<T, false, 2, true>(c, ops, nops, xpack, st, launches);
    return deep ? duo_launch<T, false, 4, false>(c, ops, nops, xpack, st, launches) : duo_launch<T, false, 2, false>(c, ops, nops, xpack, st, launches);
}

template <int T> static cudaError_t launch_duo_routed_t(const QmmArgs &a, uint32_t tiles, const uint8_t *xpack, cudaStream_t st, int *launches) {
    DuoCfg c{};
    c.n_wt = (a.n + kDuoRows - 1) / kDuoRows;
    c.out.y[0] = a.y;
    c.out.n[0] = a.n;
    c.out.wt_end[0] = c.n_wt;
    c.nt = kRoutedTile;
    c.accs = 1;
    c.ntiles = tiles;
    const uint64_t items = (uint64_t)c.n_wt * tiles;
    c.pairs = items < duo_pairs() ? (uint32_t)items : duo_pairs();
    c.beside = (a.reuse & 4u) != 0;
    if (!c.pairs) return cudaSuccess;
    if constexpr (T == GT_Q6_K)
        if (duo_raw_order(T, a.k, true, false)) return duo_launch<T, true, 4, true>(c, &a, 1, xpack, st, launches);
    return duo_launch<T, true, 4, false>(c, &a, 1, xpack, st, launches);
}

// `tiles`: bound of the list's length; `xpack`: what the list's tiles hold
bool qmm_duo_routed_fits(int ggml_type, const QmmArgs &a) {
    if (!a.hids || a.y_ld || a.n_peer || a.k % 32 != 0 || a.n_experts < 1) return false;
    const uint64_t row_bytes = (uint64_t)(a.k / ggml_qk(ggml_type)) * ggml_block_bytes(ggml_type);
    return (((uintptr_t)a.w | a.expert_stride) & 15u) == 0 && a.n % (1u << duo_row_group((uint32_t)row_bytes)) == 0 && row_bytes * a.n <= a.expert_stride &&
           encode_tiled_fn() != nullptr;
}
cudaError_t launch_qmm_duo_routed(int ggml_type, const QmmArgs &a, uint32_t tiles, const uint8_t *xpack, cudaStream_t st, int *launches) {
    switch (ggml_type) {
    case GT_Q4_0: return launch_duo_routed_t<GT_Q4_0>(a, tiles, xpack, st, launches);
    case GT_Q8_0: return launch_duo_routed_t<GT_Q8_0>(a, tiles, xpack, st, launches);
    case GT_Q6_K: return launch_duo_routed_t<GT_Q6_K>(a, tiles, xpack, st, launches);
    case GT_Q4_K: return launch_duo_routed_t<GT_Q4_K>(a, tiles, xpack, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_qmm_duo(int ggml_type, const QmmArgs *ops, int nops, uint32_t nt, uint32_t limit, uint8_t *xpack, cudaStream_t st, int *launches) {
    switch (ggml_type) {
    case GT_Q4_0: return launch_duo_t<GT_Q4_0>(ops, nops, nt, limit, xpack, st, launches);
    case GT_Q8_0: return launch_duo_t<GT_Q8_0>(ops, nops, nt, limit, xpack, st, launches);
    case GT_Q6_K: return launch_duo_t<GT_Q6_K>(ops, nops, nt, limit, xpack, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace mlxn
