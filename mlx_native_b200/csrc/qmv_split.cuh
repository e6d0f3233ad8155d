// Mat-vec for few activation rows, dense and expert-routed: y[m, n] = x[m, k] . W[n, k]^T with W in GGML blocks.
//
// HBM bounds the operation (6.4 TB/s measured copy rate: 23 bytes per cycle and SM); what a kernel loses against that is latency
// (launch, activations, waits between stages) and instructions (integer operations issue at half rate).  Hence:
//
//  * The activations of a CTA stay in shared memory for all its weight rows, in the order of the B registers of mma.sync.  One or two
//    rows (dense) as four signed 8-bit digits, for multiplies of 8-bit integers (sp_unit_int), where a warp's share of them is alike enough for one last
//    place; other shares (sp_far), more rows, and routed ones, as f16 hi + lo halves, scaled by powers of two so that both stay in range, for
//    mma.sync.m16n8k16.  One and two rows are split by every CTA
//    itself, several by qmv_pack_kernel, and arrive by bulk copies.  The loop over the weights only unpacks codes into signed integers, bytes or
//    normal f16 numbers, so products are exact and sums are f32.
//  * In f16 the 8 columns of an MMA are (activation row, hi | lo): one multiply serves up to four rows (NS = 2 sets: eight rows).
//  * Integers against f16, one row, us a call of a dependent chain (graph replay): Q4_0 24576 x 4096 21.5 -> 15.5, 4096 x 12288 13.2 -> 11.5, Q4_K 26.2 ->
//    19.2, 15.2 -> 13.1, Q6_K 30.6 -> 25.2, 17.4 -> 15.4, Q8_0 25.7 -> 23.9 (its codes took least); 151936 x 4096 Q4_0 97 -> 70, Q6_K 151936 x 5120 172 (the
//    register-level kernel) -> 144.  What is left there: Q4_0 takes 65 instructions a tile and unit, 140 cycles of a scheduler where its bytes would take 96 at the
//    copy rate (issue slots 55 percent busy, integer operations 48; Q6_K 124 instructions; profiles/qmv_split_full.md), and at the start and between chunks latency: 0.3 us
//    for a unit of a warp's activations, 1.3 us a chunk.
//  * A warp works on up to four 16-row tiles at a time: one tile at a time leaves the pipes idle between dependent steps (Q4_0,
//    75776 x 4096: 70.7 us, 2.5 TB/s, against 44.9, 3.9 TB/s).
//  * K may be split over the CTAs of a cluster (1, 2, 4, 8): a matrix of few rows still fills the chip, and long activation rows
//    still fit into shared memory.  The ranks' partial sums travel through distributed shared memory (st.async) and are added in
//    rank order by the CTA that owns the row: no atomics, results are bit-reproducible.
//  * A producer warp fills a ring of stages (16-row tiles x SU units of 64 K values) by TMA: tensor copies where every weight row
//    starts on a 16-byte boundary (ALN) or every other one does, else one bulk copy per row of the 16-byte superset of its segment, so a K that is no
//    multiple of 256 and a weight address that is even do for Q4_0, Q8_0 and Q6_K (Q8_0 2873 x 2880, five rows: 11.7 us where the
//    kernel that reads blocks from global memory took 181).  Q4_K and Q5_K have to start on 16-byte boundaries.
//  * Expert-routed: every CTA sorts the (token, slot) pairs by expert itself (at most 256 pairs), and the rows of one expert share
//    a pass over its weights, four at a time.  K is not split here.
//
// The activations in shared memory bound K: 133120 values for one row, 65536 for two, 30720 for up to four, 14336 for more; routed
// 3840, and 16640 for a single pair (qmv_split_fits).  Beyond that the other mat-vec kernels take over.
#pragma once
#include "tensor_map.cuh"

#include <cstdio>
#include <cstdlib>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "mma_f16.cuh"
#include "ptx.cuh"

namespace mlxn {

constexpr int kSpWarps = 8;                         // consumer warps
constexpr int kSpThreads = (kSpWarps + 1) * 32;     // and one producer warp
constexpr int kSpTiles = 4;                         // 16-row tiles of a chunk, at most
__host__ __device__ constexpr int sp_tiles(int mp) { return mp > 4 ? 2 : kSpTiles; }
constexpr int kSpMaxOps = 8;                        // mat-vecs one launch carries
constexpr int kSpMaxSlots = 8;
constexpr int kSpMaxPairs = 256;                    // (token, slot) pairs of a routed launch
// Two CTAs share an SM: 228 KB less 1 KB each for the system and the kernel's static 3 KB.
constexpr size_t kSpSmem = 110 * 1024;
constexpr int kSpMaxUnits = kSpSmem / 256;          // units of activations that a CTA holds, all rows together

// SU: units (64 K values) of a stage, a multiple of the warps.  NG: sub-blocks of a unit that have an offset of their own, and
// with it the sum of their activations (Q4_K, Q5_K).
template <int T> struct SpTraits;
template <> struct SpTraits<GT_Q4_0> { static constexpr int B256 = 144, SU = 16, NG = 0; };
template <> struct SpTraits<GT_Q8_0> { static constexpr int B256 = 272, SU = 8, NG = 0; };
template <> struct SpTraits<GT_Q4_K> { static constexpr int B256 = 144, SU = 16, NG = 2; };
template <> struct SpTraits<GT_Q5_K> { static constexpr int B256 = 176, SU = 16, NG = 2; };
template <> struct SpTraits<GT_Q6_K> { static constexpr int B256 = 210, SU = 8, NG = 0; };

// Bytes of shared memory per row of a stage: an odd multiple of 16 (32-bit reads of eight rows hit distinct banks).
template <int T> __host__ __device__ constexpr uint32_t sp_pitch(bool aln) {
    const uint32_t lead = aln && T != GT_Q6_K ? 0u : 14u;
    return 16u * (((SpTraits<T>::SU / 4 * SpTraits<T>::B256 + lead + 15u) / 16u) | 1u);
}

struct SpOp {
    const uint8_t *w;
    const float *x;
    const float *x2;          // fused SwiGLU: the activations are silu(x) * x2
    float *y;
    uint32_t n, k, m;
    uint32_t step_end;        // steps (of `step` 16-row tiles) of the ops up to and including this one
    uint32_t row_bytes;
    uint32_t units;           // ceil(k / 64)
    uint32_t slice;           // units per cluster rank (a multiple of 4)
    uint32_t xkey;            // ops with equal keys have the same activations
    uint32_t x_div;           // routed: the activation row of pair p is p / x_div
    uint32_t y_ld, y_col0, n_peer;
    float *y_peer[kMaxPeers];
    uint64_t expert_stride;
    // packed activations (see qmv_pack_kernel): per row pk_units x 256 bytes of B registers, pk_units x NG sums, one scale
    const uint8_t *xp;
    const float *xsum, *xinv;
    uint32_t pk_units;
    uint32_t row_end;         // rows to pack of the ops up to and including this one
    // where the packed values of a row's super-block lie: bytes from one row and from one super-block to the next
    uint64_t xp_row, xp_super;
    uint32_t wide_rows;       // qmv_wide.cu: rows of a super-block; odd rows have lo before hi, sums are [super-block][row / 8][8][row % 8]
};
struct SpBatch {
    SpOp op[kSpMaxOps];
    const uint32_t *ids;      // routed: expert of every pair
    uint32_t nops, npairs, n_experts;
    uint32_t nent;            // dense: groups of mp activation rows; routed: counted on the device
    uint32_t mp;              // activation rows of an entry (1, 2, 4 or 8)
    uint32_t tr, step;        // tiles of a chunk, at most, and of a step of the clusters' shares
    uint32_t dealt;           // steps are dealt out to the clusters in turn; otherwise a share is contiguous
    uint32_t early_weights;
    uint32_t *status;
    uint32_t nslots;          // ring depth, and what lies behind the ring in shared memory
    uint32_t xf_off, cc_off, tab_off, red_off, recv_off;
    uint32_t xstride, cstride;   // bytes from one activation row to the next
    uint32_t packed;          // the activations have been packed by qmv_pack_kernel
    uint32_t pairs;           // every other row starts on a 16-byte boundary: the rows arrive by tensor copies all the same
};
struct SpMaps {
    CUtensorMap m[kSpMaxOps];
};

__device__ __forceinline__ void bulk_g2s_a(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
}
namespace sp {
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// a store to another CTA's shared memory that counts as 4 arrived bytes on a barrier there
__device__ __forceinline__ void st_async(uint32_t a, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a), "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
// Power of two that brings amax into [2^13, 2^14), and its inverse; 1 for an all-zero run.  (An infinite one: the factor of the
// largest numbers; both are normal numbers for every amax, the smallest come out below 2^13.)
__device__ __forceinline__ void pow2(float amax, float &s, float &inv) {
    s = inv = 1.f;
    if (amax > 0.f) {
        int e = 13 + 127 - (int)((__float_as_uint(amax) >> 23) & 0xffu);
        e = max(-114, min(126, e));
        s = __uint_as_float((uint32_t)(e + 127) << 23);
        inv = __uint_as_float((uint32_t)(127 - e) << 23);
    }
}
// a and b as f16 hi + lo: 22 bits of the largest, no error above 2^-39 of it in any other.  (An infinity is all in hi.)
__device__ __forceinline__ void split(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 w = __half22float2(h);
    const __half2 l = __floats2half2_rn(fabsf(w.x) < INFINITY ? a - w.x : 0.f, fabsf(w.y) < INFINITY ? b - w.y : 0.f);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// The largest magnitude by its bits: an infinity is above every number, a NaN above that.
__device__ __forceinline__ uint32_t peak_bits(const float (&v)[4]) {
    uint32_t b[4];
#pragma unroll
    for (int e = 0; e < 4; e++) b[e] = __float_as_uint(v[e]) & 0x7FFFFFFFu;
    return max(max(b[0], b[1]), max(b[2], b[3]));
}
// How the values of a warp's share compare with the largest: `peak` of four a lane, of 32 eight neighbouring lanes; `least`: what counts.
struct Spread {
    uint32_t held = 0, some = 0;
    bool lost = false;
    __device__ __forceinline__ void look(uint32_t peak, uint32_t least, uint32_t lane) {
        const uint32_t h = __ballot_sync(0xffffffffu, peak >= least), n = __ballot_sync(0xffffffffu, peak != 0), m = 0xFFu << (lane & 24u);
        held += __popc(h);
        some += __popc(n);
        lost = lost || ((n & m) != 0 && (h & m) == 0);
    }
    __device__ __forceinline__ bool far() const { return __any_sync(0xffffffffu, lost) || 2 * held < some; }
};
// Two powers of two whose product brings amax (its bits; a number) into [2^13, 2^14), and those of the way back from units of the last digit.
// (One factor would not be a normal number where amax is tiny.)
__device__ __forceinline__ void pow2_int(uint32_t amax, float &s0, float &s1, float &inv0, float &inv1) {
    const int e = 13 + 127 - (int)(amax >> 23), a = e >> 1, b = e - a;
    s0 = __uint_as_float((uint32_t)(127 + a) << 23);
    s1 = __uint_as_float((uint32_t)(127 + b) << 23);
    inv0 = __uint_as_float((uint32_t)(127 - 15 - a) << 23);
    inv1 = __uint_as_float((uint32_t)(127 - b) << 23);
}
// Four numbers below 2^14 as four signed digits each, in units of 2^-15: l[0] + 256 l[1] + 2^15 (l[2] + 256 l[3]); l[i] holds digit i of all
// four, a byte each.  (Adding 1.5 * 2^23 leaves the nearest integer in the low bits, here with 128 more, so that the low byte is a signed digit
// once its top bit has changed; a conversion instruction issues at an eighth of the rate.)
constexpr float kDigitWeight = 32768.f;   // of digits 2 and 3 against 0 and 1
__device__ __forceinline__ void digits(const float (&c)[4], uint32_t (&l)[4]) {
    constexpr float M = 12582912.f + 128.f;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float t = __fadd_rn(c[i], M);
        hi[i] = __float_as_uint(t);
        lo[i] = __float_as_uint(__fmaf_rn(__fsub_rn(c[i], __fsub_rn(t, M)), kDigitWeight, M));
    }
    const uint32_t a = __byte_perm(lo[0], lo[1], 0x5140), b = __byte_perm(lo[2], lo[3], 0x5140);
    const uint32_t e = __byte_perm(hi[0], hi[1], 0x5140), d = __byte_perm(hi[2], hi[3], 0x5140);
    l[0] = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
    l[1] = __byte_perm(a, b, 0x7632);
    l[2] = __byte_perm(e, d, 0x5410) ^ 0x80808080u;
    l[3] = __byte_perm(e, d, 0x7632);
}
// D = A (16 x 32, row) * B (32 x 8, col) + C in 8-bit integers.  Lane (g, t): a0 = A[g][4t .. 4t+3], a1 = A[g+8][..], a2 = A[g][16+4t ..],
// a3 = A[g+8][16+4t ..]; b0 = B[4t .. 4t+3][g], b1 = B[16+4t ..][g]; c and d as mma16816.
__device__ __forceinline__ void mma_s8(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const uint32_t (&c)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// Integers to f32 without a conversion: with C = kBias the bits of D are those of 1.5 * 2^23 + the sum, while that is below 2^22.
constexpr uint32_t kBias = 0x4B400000u;
// acc += (d0 or d1) * the sums: rows g and g + 8, two columns at a time
__device__ __forceinline__ void scaled(float (&acc)[4], const uint32_t (&d)[4], float d0, float d1) {
    const uint64_t off = pack2(-12582912.f, -12582912.f);
    uint64_t lo = ffma2(pack2(d0, d0), fadd2(pack2u(d[0], d[1]), off), pack2(acc[0], acc[1]));
    uint64_t hi = ffma2(pack2(d1, d1), fadd2(pack2u(d[2], d[3]), off), pack2(acc[2], acc[3]));
    unpack2(lo, acc[0], acc[1]);
    unpack2(hi, acc[2], acc[3]);
}
// Codes to signed integers.  A code n in the low bits of a half with exponent field 0x64 reads 1024 + n, one four bits further up
// 1024 + 16 n; the bias goes off exactly.  (Codes that stay subnormals, n 2^-24, save this operation, but the tensor core aligns
// products by their exponents before it adds them, and a subnormal's leading zeros are then bits lost: Q4_0 had errors of 5e-7 on
// normal activations and 1e-5 with outliers, against 64 bits.)
__device__ __forceinline__ uint32_t less(uint32_t v, uint32_t bias) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(bias));
    return r;
}
__device__ __forceinline__ uint32_t lo4(uint32_t v) { return less((v & 0x000F000Fu) | 0x64006400u, 0x64086408u); }   // n - 8
__device__ __forceinline__ uint32_t hi4(uint32_t v) {                                                                 // (1024 + 16 n) / 16 - 72
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"((v & 0x00F000F0u) | 0x64006400u), "r"(0x2C002C00u), "r"(0xD480D480u));
    return r;
}
// bytes 0, 2 and bytes 1, 3 of a word
__device__ __forceinline__ uint32_t bytes02(uint32_t v, uint32_t bias) { return less(__byte_perm(v, 0x64646464u, 0x4240), bias); }
__device__ __forceinline__ uint32_t bytes13(uint32_t v, uint32_t bias) { return less(__byte_perm(v, 0x64646464u, 0x4341), bias); }
}  // namespace sp

// Where in its unit the four values lie that quad lane t multiplies in MMA q, as two pairs of consecutive elements.  Q4_0 and
// Q8_0 with aligned rows work on pairs of blocks: the even block starts on a 4-byte boundary, so its codes (2 bytes in)
// straddle the words; lanes 1..3 take whole words and lane 0 the two half words at either end, which sit in the words that
// hold the pair's two scales.  (Q6_K: relative to the super-block.)
template <int T, bool ALN> __device__ __forceinline__ void sp_pairs(uint32_t u, uint32_t q, uint32_t t, uint32_t &p0, uint32_t &p1) {
    if constexpr (T == GT_Q6_K) {
        p0 = 128u * ((u >> 1) & 1u) + 32u * q + 16u * (u & 1u) + 4u * t;
        p1 = p0 + 2;
    } else if constexpr ((T == GT_Q4_0 || T == GT_Q8_0) && ALN) {
        const uint32_t h = q & 1u;
        if (q >= 2) {
            p0 = 32 + 16 * h + 4 * t;
            p1 = p0 + 2;
        } else if (T == GT_Q8_0 && h) {
            p0 = 14 + 4 * t;
            p1 = 16 + 4 * t;
        } else {
            p0 = t ? 4 * t - 2 : 0;
            p1 = t ? 4 * t : (T == GT_Q8_0 ? 30 : 14);
            if (T == GT_Q4_0) { p0 += 16 * h; p1 += 16 * h; }
        }
    } else {
        p0 = 16u * q + 4u * t;
        p1 = p0 + 2;
    }
}

// The four activations at x + p0 and x + p1, of which the pairs i0 and i1 exist; y: fused SwiGLU, silu(x) * y (as src/shaders/silu_mul.metal:17-30).
__device__ __forceinline__ void sp_act(const float *x, const float *y, uint32_t p0, uint32_t p1, bool i0, bool i1, float (&v)[4]) {
    if (i0) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(x + p0));
    if (i1) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[2]), "=f"(v[3]) : "l"(x + p1));
    if (y) {
        float w[4] = {0.f, 0.f, 0.f, 0.f};
        if (i0) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(w[0]), "=f"(w[1]) : "l"(y + p0));
        if (i1) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(w[2]), "=f"(w[3]) : "l"(y + p1));
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = v[e] / (1.0f + expf(-v[e])) * w[e];
    }
}

// One unit (64 K values) of a stage against NT tiles.  a0 / a1: shared address of rows g and g + 8 of tile 0 at the unit's
// first byte (Q4_K, Q5_K, Q6_K: of its super-block), lead-in included; tiles are 16 PITCH bytes apart.  bf: the B registers
// [set][MMA][2]; cc: per set and sub-block the sum of the activations (Q4_K, Q5_K); tab: the warp's scale table.  FACT: the activations of MMAs
// 0 and 1 and those of 2 and 3 have a power of two each, beside the one of the share; f2: its inverses for the lane's columns.
template <int T, bool ALN, int NT, bool FACT, int NS, int TM>
__device__ __forceinline__ void sp_unit(uint32_t a0, uint32_t a1, uint32_t u, uint32_t t, uint32_t g, uint32_t tab, bool half,
                                        const uint32_t (&bf)[NS][4][2], [[maybe_unused]] const float (&cc)[NS][2], [[maybe_unused]] const float (&f2)[2],
                                        float (&acc)[TM][NS][4]) {
    constexpr uint32_t TS = 16u * sp_pitch<T>(ALN);
    if constexpr (T == GT_Q4_0 || T == GT_Q8_0) {
        constexpr bool Q8 = T == GT_Q8_0;
        constexpr uint32_t BB = Q8 ? 34u : 18u;
        // row g + 8 relative to row g is a compile-time distance only with aligned rows
        const uint32_t b0[2] = {ALN ? a0 + 4 * t : (a0 & ~3u) + 4 * t, ALN ? a1 + 4 * t : (a1 & ~3u) + 4 * t};
        const uint32_t e0 = a0 + (t ? 4 * t : (Q8 ? 32u : 16u)), e1 = a1 + (t ? 4 * t : (Q8 ? 32u : 16u));
        const uint32_t sel = t ? 0x3210u : 0x5432u;
        uint32_t se[2], so[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const bool mis = !ALN && ((h ? a1 : a0) & 2u) != 0;
            se[h] = mis ? 0x7654u : 0x5432u;
            so[h] = mis ? 0x5432u : 0x3210u;
        }
        static_for<0, NT>([&](auto J) {
            constexpr uint32_t o = decltype(J)::value * TS;
            uint32_t w[4][2];   // even block, MMA 0 / 1; odd block, MMA 0 / 1 (Q4_0: one word per block)
            float d0[2], d1[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t b = b0[h];
                [[maybe_unused]] const uint32_t e = h ? e1 : e0, a = h ? a1 : a0;
                if constexpr (ALN) {
                    w[0][h] = __byte_perm(lds32i<o>(b), lds32i<o>(e), sel);
                    if constexpr (Q8) {
                        w[1][h] = lds32i<o + 16>(b);
                        w[2][h] = lds32i<o + 36>(b);
                        w[3][h] = lds32i<o + 52>(b);
                    } else {
                        w[2][h] = lds32i<o + 20>(b);
                    }
                } else {
                    w[0][h] = __byte_perm(lds32i<o>(b), lds32i<o + 4>(b), se[h]);
                    if constexpr (Q8) {
                        w[1][h] = __byte_perm(lds32i<o + 16>(b), lds32i<o + 20>(b), se[h]);
                        w[2][h] = __byte_perm(lds32i<o + 36>(b), lds32i<o + 40>(b), so[h]);
                        w[3][h] = __byte_perm(lds32i<o + 52>(b), lds32i<o + 56>(b), so[h]);
                    } else {
                        w[2][h] = __byte_perm(lds32i<o + 20>(b), lds32i<o + 24>(b), so[h]);
                    }
                }
                d0[h] = f16lo_to_float(lds_u16i<o>(a));
                d1[h] = f16lo_to_float(lds_u16i<o + BB>(a));
                if constexpr (!ALN) d1[h] = half ? 0.f : d1[h];
                if constexpr (FACT) {
                    d0[h] *= f2[0];
                    d1[h] *= f2[1];
                }
            }
            uint32_t a[4][4];
            if constexpr (Q8) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t x0 = w[q][0] ^ 0x80808080u, x1 = w[q][1] ^ 0x80808080u;
                    a[q][0] = sp::bytes02(x0, 0x64806480u); a[q][1] = sp::bytes02(x1, 0x64806480u);
                    a[q][2] = sp::bytes13(x0, 0x64806480u); a[q][3] = sp::bytes13(x1, 0x64806480u);
                }
            } else {              // low nibbles: elements 0..15; high nibbles: 16..31
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    const uint32_t x0 = w[2 * b][0], x1 = w[2 * b][1], y0 = x0 >> 8, y1 = x1 >> 8;
                    a[2 * b][0] = sp::lo4(x0); a[2 * b][1] = sp::lo4(x1);
                    a[2 * b][2] = sp::lo4(y0); a[2 * b][3] = sp::lo4(y1);
                    a[2 * b + 1][0] = sp::hi4(x0); a[2 * b + 1][1] = sp::hi4(x1);
                    a[2 * b + 1][2] = sp::hi4(y0); a[2 * b + 1][3] = sp::hi4(y1);
                }
            }
            constexpr int j = decltype(J)::value;
#pragma unroll
            for (int s = 0; s < NS; s++) {
                constexpr float zero[4] = {0.f, 0.f, 0.f, 0.f};
                float r0[4], r1[4];
                mma16816(r0, a[0][0], a[0][1], a[0][2], a[0][3], bf[s][0][0], bf[s][0][1], zero);
                mma16816(r1, a[2][0], a[2][1], a[2][2], a[2][3], bf[s][2][0], bf[s][2][1], zero);
                mma16816(r0, a[1][0], a[1][1], a[1][2], a[1][3], bf[s][1][0], bf[s][1][1], r0);
                mma16816(r1, a[3][0], a[3][1], a[3][2], a[3][3], bf[s][3][0], bf[s][3][1], r1);
                acc[j][s][0] = fmaf(d1[0], r1[0], fmaf(d0[0], r0[0], acc[j][s][0]));
                acc[j][s][1] = fmaf(d1[0], r1[1], fmaf(d0[0], r0[1], acc[j][s][1]));
                acc[j][s][2] = fmaf(d1[1], r1[2], fmaf(d0[1], r0[2], acc[j][s][2]));
                acc[j][s][3] = fmaf(d1[1], r1[3], fmaf(d0[1], r0[3], acc[j][s][3]));
            }
        });
    } else if constexpr (T == GT_Q4_K || T == GT_Q5_K) {
        constexpr bool Q5 = T == GT_Q5_K;
        const uint32_t pu = u & 3u, qo = (Q5 ? 48u : 16u) + 32 * pu + 4 * t;
        const uint32_t q0 = a0 + qo, q1 = a1 + qo, h0 = a0 + 16 + 4 * t, h1 = a1 + 16 + 4 * t, tr = tab + g * 16;
        static_for<0, NT>([&](auto J) {
            constexpr int j = decltype(J)::value;
            constexpr uint32_t o = j * TS;
            uint32_t x[2][2];   // [first / second 16 elements][row g, g + 8]
            x[0][0] = lds32i<o>(q0); x[1][0] = lds32i<o + 16>(q0);
            x[0][1] = lds32i<o>(q1); x[1][1] = lds32i<o + 16>(q1);
            uint32_t p0[4], p1[4];   // scales and offsets (sp_table_row) of rows g and g + 8
            lds128i<j * 256u>(tr, p0);
            lds128i<j * 256u + 128u>(tr, p1);
            if constexpr (FACT) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    p0[q] = __float_as_uint(__uint_as_float(p0[q]) * f2[q & 1]);
                    p1[q] = __float_as_uint(__uint_as_float(p1[q]) * f2[q & 1]);
                }
            }
            uint32_t a[4][4];
            if constexpr (Q5) {   // five-bit codes, one per byte: nibble | fifth bit << 4
                uint32_t f[2][2];
                f[0][0] = lds32i<o>(h0) >> (2 * pu); f[1][0] = lds32i<o + 16>(h0) >> (2 * pu);
                f[0][1] = lds32i<o>(h1) >> (2 * pu); f[1][1] = lds32i<o + 16>(h1) >> (2 * pu);
#pragma unroll
                for (int e = 0; e < 2; e++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t lo = (x[e][h] & 0x0F0F0F0Fu) | ((f[e][h] & 0x01010101u) << 4);
                        const uint32_t hi = ((x[e][h] >> 4) & 0x0F0F0F0Fu) | ((f[e][h] & 0x02020202u) << 3);
                        a[e][h] = sp::bytes02(lo, 0x64106410u); a[e][h + 2] = sp::bytes13(lo, 0x64106410u);
                        a[e + 2][h] = sp::bytes02(hi, 0x64106410u); a[e + 2][h + 2] = sp::bytes13(hi, 0x64106410u);
                    }
            } else {
#pragma unroll
                for (int e = 0; e < 2; e++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t y = x[e][h] >> 8;
                        a[e][h] = sp::lo4(x[e][h]); a[e][h + 2] = sp::lo4(y);
                        a[e + 2][h] = sp::hi4(x[e][h]); a[e + 2][h + 2] = sp::hi4(y);
                    }
            }
#pragma unroll
            for (int s = 0; s < NS; s++) {
                constexpr float zero[4] = {0.f, 0.f, 0.f, 0.f};
                float r0[4], r1[4];
                mma16816(r0, a[0][0], a[0][1], a[0][2], a[0][3], bf[s][0][0], bf[s][0][1], zero);
                mma16816(r1, a[2][0], a[2][1], a[2][2], a[2][3], bf[s][2][0], bf[s][2][1], zero);
                mma16816(r0, a[1][0], a[1][1], a[1][2], a[1][3], bf[s][1][0], bf[s][1][1], r0);
                mma16816(r1, a[3][0], a[3][1], a[3][2], a[3][3], bf[s][3][0], bf[s][3][1], r1);
                const float c0 = cc[s][0], c1 = cc[s][1];
                auto f = [](uint32_t v) { return __uint_as_float(v); };
                acc[j][s][0] = fmaf(f(p0[1]), r1[0], fmaf(f(p0[0]), r0[0], fmaf(f(p0[3]), c1, fmaf(f(p0[2]), c0, acc[j][s][0]))));
                acc[j][s][1] = fmaf(f(p0[1]), r1[1], fmaf(f(p0[0]), r0[1], acc[j][s][1]));
                acc[j][s][2] = fmaf(f(p1[1]), r1[2], fmaf(f(p1[0]), r0[2], fmaf(f(p1[3]), c1, fmaf(f(p1[2]), c0, acc[j][s][2]))));
                acc[j][s][3] = fmaf(f(p1[1]), r1[3], fmaf(f(p1[0]), r0[3], acc[j][s][3]));
            }
        });
    } else {
        const uint32_t nh = (u >> 1) & 1u, js = u & 1u, tr = tab + g * 16;
        const uint32_t lo = 64 * nh + 16 * js + 4 * t, ho = 128 + 32 * nh + 16 * js + 4 * t;
        // super-blocks are 210 bytes: where one starts 2 bytes past a word boundary, words are joined from two.  With aligned
        // rows that is the same for all rows (SHIFT known per call), else a matter of the row.
        auto body = [&](auto SHIFT) {
            constexpr int shift = decltype(SHIFT)::value;   // 0: word-aligned, 1: joined, 2: per row
            const uint32_t b0 = a0 & ~3u, b1 = a1 & ~3u;
            const uint32_t L[2] = {b0 + lo, b1 + lo}, H[2] = {b0 + ho, b1 + ho};
            const uint32_t sl[2] = {(a0 & 2u) ? 0x5432u : 0x3210u, (a1 & 2u) ? 0x5432u : 0x3210u};
            static_for<0, NT>([&](auto J) {
                constexpr int j = decltype(J)::value;
                constexpr uint32_t o = j * TS;
                uint32_t qv[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t A = lds32i<o>(L[h]), B = lds32i<o + 32>(L[h]), X = lds32i<o>(H[h]);
                    if constexpr (shift != 0) {
                        const uint32_t s = shift == 1 ? 0x5432u : sl[h];
                        A = __byte_perm(A, lds32i<o + 4>(L[h]), s);
                        B = __byte_perm(B, lds32i<o + 36>(L[h]), s);
                        X = __byte_perm(X, lds32i<o + 4>(H[h]), s);
                    }
                    qv[h][0] = (A & 0x0F0F0F0Fu) | ((X & 0x03030303u) << 4);
                    qv[h][1] = (B & 0x0F0F0F0Fu) | ((X & 0x0C0C0C0Cu) << 2);
                    qv[h][2] = ((A >> 4) & 0x0F0F0F0Fu) | (X & 0x30303030u);
                    qv[h][3] = ((B >> 4) & 0x0F0F0F0Fu) | ((X & 0xC0C0C0C0u) >> 2);
                }
                uint32_t p0[4], p1[4];
                lds128i<j * 256u>(tr, p0);
                lds128i<j * 256u + 128u>(tr, p1);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t x0 = sp::bytes02(qv[0][q], 0x64206420u), x2 = sp::bytes13(qv[0][q], 0x64206420u);
                    const uint32_t x1 = sp::bytes02(qv[1][q], 0x64206420u), x3 = sp::bytes13(qv[1][q], 0x64206420u);
                    float pa = __uint_as_float(p0[q]), pb = __uint_as_float(p1[q]);
                    if constexpr (FACT) {
                        pa *= f2[q >> 1];
                        pb *= f2[q >> 1];
                    }
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        constexpr float zero[4] = {0.f, 0.f, 0.f, 0.f};
                        float r[4];
                        mma16816(r, x0, x1, x2, x3, bf[s][q][0], bf[s][q][1], zero);
                        acc[j][s][0] = fmaf(pa, r[0], acc[j][s][0]);
                        acc[j][s][1] = fmaf(pa, r[1], acc[j][s][1]);
                        acc[j][s][2] = fmaf(pb, r[2], acc[j][s][2]);
                        acc[j][s][3] = fmaf(pb, r[3], acc[j][s][3]);
                    }
                }
            });
        };
        if constexpr (ALN) {
            if (a0 & 2u) body(std::integral_constant<int, 1>{});
            else body(std::integral_constant<int, 0>{});
        } else {
            body(std::integral_constant<int, 2>{});
        }
    }
}

// One unit of a stage against NT tiles, for one or two activation rows: codes as signed bytes, activations as four signed digits
// (sp::digits), 8-bit integer multiplies.  A multiply takes 32 K values where the f16 form takes 16, Q8_0 codes go in as they lie, 4-bit codes
// take three operations for eight (with f16 they take twelve), sums of a block are exact, and the digits hold 28 bits of the largest activation.
// The columns of a multiply are (first | second scale group, digit) of one activation row; a column's B registers are zero outside its group, so
// one accumulator serves both blocks of a unit (Q6_K, whose scales change every 16 values: both halves of one multiply), and a lane scales its
// columns with the one scale of their group.  Codes are taken 16 times (Q4_0, Q4_K) or 4 times (Q6_K) as large:
// that centres them without an addition (the top bit of the byte changes sign), and sp_code_scale takes it back.  bf: B registers [set][word].
template <int T> constexpr float sp_code_scale = T == GT_Q8_0 ? 1.f : T == GT_Q6_K ? 0.25f : 0.0625f;
// alike: all rows start at the same half of a word.  OFF: the unit's bytes within a stage from the warp's first unit on.  c: kBias four times, in registers (as an immediate every multiply would
// copy it into four of them).
template <int T, bool ALN, uint32_t OFF, int NT, int NS, int TM>
__device__ __forceinline__ void sp_unit_int(uint32_t a0, uint32_t a1, uint32_t u, uint32_t t, uint32_t tab, bool half, [[maybe_unused]] bool alike, const uint32_t (&bf)[NS][4],
                                            [[maybe_unused]] const float (&cc)[NS], const uint32_t (&c)[4], float (&acc)[TM][NS][4]) {
    constexpr uint32_t TS = 16u * sp_pitch<T>(ALN), R8 = ALN ? 8u * sp_pitch<T>(true) : 0u;
    auto f = [](uint32_t v) { return __uint_as_float(v); };
    if constexpr (T == GT_Q4_0 || T == GT_Q8_0) {
        constexpr bool Q8 = T == GT_Q8_0;
        constexpr uint32_t BB = Q8 ? 34u : 18u;
        // row g + 8 relative to row g is a compile-time distance only with aligned rows
        const uint32_t b[2] = {ALN ? a0 + 4 * t : (a0 & ~3u) + 4 * t, ALN ? a0 + 4 * t : (a1 & ~3u) + 4 * t}, a[2] = {a0 + (t >> 1) * BB, (ALN ? a0 : a1) + (t >> 1) * BB};
        const uint32_t e = a0 + (t ? 4 * t : (Q8 ? 32u : 16u));
        const uint32_t sel = t ? 0x3210u : 0x5432u;
        uint32_t se[2], so[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const bool mis = !ALN && ((h ? a1 : a0) & 2u) != 0;
            se[h] = mis ? 0x7654u : 0x5432u;
            so[h] = mis ? 0x5432u : 0x3210u;
        }
        static_for<0, NT>([&](auto J) {
            constexpr int j = decltype(J)::value;
            uint32_t w[4][2];   // as in sp_unit
            float d[2];
            static_for<0, 2>([&](auto H) {
                constexpr int h = decltype(H)::value;
                constexpr uint32_t o = OFF + j * TS + h * R8;
                if constexpr (ALN) {
                    w[0][h] = __byte_perm(lds32i<o>(b[h]), lds32i<o>(e), sel);
                    if constexpr (Q8) {
                        w[1][h] = lds32i<o + 16>(b[h]);
                        w[2][h] = lds32i<o + 36>(b[h]);
                        w[3][h] = lds32i<o + 52>(b[h]);
                    } else {
                        w[2][h] = lds32i<o + 20>(b[h]);
                    }
                } else {
                    w[0][h] = __byte_perm(lds32i<o>(b[h]), lds32i<o + 4>(b[h]), se[h]);
                    if constexpr (Q8) {
                        w[1][h] = __byte_perm(lds32i<o + 16>(b[h]), lds32i<o + 20>(b[h]), se[h]);
                        w[2][h] = __byte_perm(lds32i<o + 36>(b[h]), lds32i<o + 40>(b[h]), so[h]);
                        w[3][h] = __byte_perm(lds32i<o + 52>(b[h]), lds32i<o + 56>(b[h]), so[h]);
                    } else {
                        w[2][h] = __byte_perm(lds32i<o + 20>(b[h]), lds32i<o + 24>(b[h]), so[h]);
                    }
                }
                d[h] = f16lo_to_float(lds_u16i<o>(a[h]));
                if constexpr (!ALN) d[h] = half ? 0.f : d[h];
            });
            if constexpr (!Q8) {   // low nibbles: elements 0..15; high nibbles: 16..31
#pragma unroll
                for (int q = 0; q < 4; q += 2)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t x = w[q][h];
                        w[q][h] = ((x << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
                        w[q + 1][h] = (x & 0xF0F0F0F0u) ^ 0x80808080u;
                    }
            }
#pragma unroll
            for (int s = 0; s < NS; s++) {
                uint32_t r[4];
                sp::mma_s8(r, w[0][0], w[0][1], w[1][0], w[1][1], bf[s][0], bf[s][1], c);
                sp::mma_s8(r, w[2][0], w[2][1], w[3][0], w[3][1], bf[s][2], bf[s][3], r);
                sp::scaled(acc[j][s], r, d[0], d[1]);
            }
        });
    } else if constexpr (T == GT_Q4_K) {
        const uint32_t q0 = a0 + 32 * (u & 3u) + 4 * t;
        static_for<0, NT>([&](auto J) {
            constexpr int j = decltype(J)::value;
            uint32_t a[2][4], p[2][2];   // codes (first sub-block: low nibbles, second: high ones); scale and offset (sp_table_row) of rows g, g + 8
            static_for<0, 2>([&](auto H) {
                constexpr int h = decltype(H)::value;
                constexpr uint32_t q = OFF + j * TS + h * R8 + 16u;
                lds64i<j * 256u + h * 128u>(tab, p[h][0], p[h][1]);
                static_for<0, 2>([&](auto E) {   // first, second 16 elements
                    constexpr int e = decltype(E)::value;
                    const uint32_t x = lds32i<q + 16 * e>(q0);
                    a[0][2 * e + h] = ((x << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
                    a[1][2 * e + h] = (x & 0xF0F0F0F0u) ^ 0x80808080u;
                });
            });
#pragma unroll
            for (int s = 0; s < NS; s++) {
                uint32_t r[4];
                sp::mma_s8(r, a[0][0], a[0][1], a[0][2], a[0][3], bf[s][0], bf[s][1], c);
                sp::mma_s8(r, a[1][0], a[1][1], a[1][2], a[1][3], bf[s][2], bf[s][3], r);
                // the offset joins the top digit (cc is zero in lanes without it)
                acc[j][s][1] = fmaf(f(p[0][1]), cc[s], acc[j][s][1]);
                acc[j][s][3] = fmaf(f(p[1][1]), cc[s], acc[j][s][3]);
                sp::scaled(acc[j][s], r, f(p[0][0]), f(p[1][0]));
            }
        });
    } else {
        const uint32_t nh = (u >> 1) & 1u, js = u & 1u;
        const uint32_t lo = 64 * nh + 16 * js + 4 * t, ho = 128 + 32 * nh + 16 * js + 4 * t;
        auto body = [&](auto SHIFT) {   // as in sp_unit
            constexpr int shift = decltype(SHIFT)::value;
            const uint32_t b0 = a0 & ~3u, b1 = ALN ? b0 : a1 & ~3u;
            const uint32_t L[2] = {b0 + lo, b1 + lo}, X[2] = {b0 + ho, b1 + ho};
            const uint32_t sl[2] = {(a0 & 2u) ? 0x5432u : 0x3210u, (a1 & 2u) ? 0x5432u : 0x3210u};
            static_for<0, NT>([&](auto J) {
                constexpr int j = decltype(J)::value;
                uint32_t q[4][2];
                static_for<0, 2>([&](auto H) {
                    constexpr int h = decltype(H)::value;
                    constexpr uint32_t o = OFF + j * TS + h * R8;
                    uint32_t A = lds32i<o>(L[h]), B = lds32i<o + 32>(L[h]), F = lds32i<o>(X[h]);
                    if constexpr (shift != 0) {
                        const uint32_t s = shift == 1 ? 0x5432u : sl[h];
                        A = __byte_perm(A, lds32i<o + 4>(L[h]), s);
                        B = __byte_perm(B, lds32i<o + 36>(L[h]), s);
                        F = __byte_perm(F, lds32i<o + 4>(X[h]), s);
                    }
                    auto join = [](uint32_t n, uint32_t x) { return (((n & 0x3C3C3C3Cu) | (x & 0xC3C3C3C3u)) & 0xFCFCFCFCu) ^ 0x80808080u; };
                    q[0][h] = join(A << 2, F << 6);
                    q[1][h] = join(B << 2, F << 4);
                    q[2][h] = join(A >> 2, F << 2);
                    q[3][h] = join(B >> 2, F);
                });
                uint32_t pa[2], pb[2];   // scales of the lane's group, first and second multiply, rows g and g + 8
                lds64i<j * 256u>(tab, pa[0], pa[1]);
                lds64i<j * 256u + 128u>(tab, pb[0], pb[1]);
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        uint32_t r[4];
                        sp::mma_s8(r, q[2 * i][0], q[2 * i][1], q[2 * i + 1][0], q[2 * i + 1][1], bf[s][2 * i], bf[s][2 * i + 1], c);
                        sp::scaled(acc[j][s], r, f(pa[i]), f(pb[i]));
                    }
            });
        };
        if (ALN || alike) {   // (even and odd rows are 8 bytes apart: the same half word)
            if (a0 & 2u) body(std::integral_constant<int, 1>{});
            else body(std::integral_constant<int, 0>{});
        } else {
            body(std::integral_constant<int, 2>{});
        }
    }
}

// Scale table of one unit for one row: d * scale of the unit's groups (Q6_K: four), or the scales d sc and the offsets C d sc - dmin m
// of its two sub-blocks (Q4_K, Q5_K: the codes are taken less C = 8 or 16, the middle of their range, so that the offset is small
// where scale and minimum belong together; 6-bit fields as in src/gguf/mod.rs:440-452).  rb: shared address of the row's super-block.
template <int T, bool INT> __device__ __forceinline__ void sp_table_row(uint32_t dst, uint32_t rb, uint32_t u) {
    auto put = [&](float a, float b, float c, float d) { sts128(dst, __float_as_uint(a), __float_as_uint(b), __float_as_uint(c), __float_as_uint(d)); };
    if constexpr (T == GT_Q6_K) {
        const uint32_t s = rb + 192 + 8 * ((u >> 1) & 1u) + (u & 1u);
        const float d = f16lo_to_float(lds_u16i<208>(rb));
        constexpr uint32_t s1 = INT ? 4 : 2, s2 = INT ? 2 : 4;   // (integers: even groups before odd ones)
        put(d * (float)lds_s8(s), d * (float)lds_s8(s + s1), d * (float)lds_s8(s + s2), d * (float)lds_s8(s + 6));
    } else {
        const uint32_t pu = u & 3u, dd = lds32(rb), s0 = lds32i<4>(rb), s1 = lds32i<8>(rb);
        const float d = f16lo_to_float(dd), dmin = f16hi_to_float(dd);
        uint32_t c0, c1, m0, m1;
        if (pu < 2) {
            const uint32_t a = s0 >> (16 * pu), b = s1 >> (16 * pu);
            c0 = a & 63u; c1 = (a >> 8) & 63u;
            m0 = b & 63u; m1 = (b >> 8) & 63u;
        } else {
            const uint32_t sh = 16 * (pu - 2);
            const uint32_t a = lds32i<12>(rb) >> sh, lo = s0 >> sh, hi = s1 >> sh;
            c0 = (a & 15u) | (((lo >> 6) & 3u) << 4);
            c1 = ((a >> 8) & 15u) | (((lo >> 14) & 3u) << 4);
            m0 = ((a >> 4) & 15u) | (((hi >> 6) & 3u) << 4);
            m1 = ((a >> 12) & 15u) | (((hi >> 14) & 3u) << 4);
        }
        constexpr float C = T == GT_Q5_K ? 16.f : 8.f;
        const float e0 = d * (float)c0, e1 = d * (float)c1;   // (17 bits: exact, as the products with the minima)
        const float o0 = fmaf(C, e0, -(dmin * (float)m0)), o1 = fmaf(C, e1, -(dmin * (float)m1));
        if constexpr (INT) put(e0, o0, e1, o1);
        else put(e0, e1, o0, o1);
    }
}

// One product of a Q4_K or Q5_K row in f32, value by value: for results that are no numbers.  Lane `part` of `parts` adds up every parts-th super-block.
// (One loop over a super-block's values: with the scales formed once for 32 of them the kernel of qmv_wide.cu has fewer registers, 1652 x 8042 x 1024 247 -> 255 us.)
template <int T> __device__ __noinline__ float sp_again(const uint8_t *w, const float *x, uint32_t k, uint32_t part, uint32_t parts) {
    float acc = 0.f;
    w += (size_t)part * BlockTraits<T>::BYTES;
    for (uint32_t b = part; b < k / 256; b += parts, w += (size_t)parts * BlockTraits<T>::BYTES)
        for (uint32_t e = 0; e < 256; e++) {
            const uint32_t j = e >> 5, l = e & 31u;
            uint32_t sc, mn;
            q4k_scale_min(j, w + 4, sc, mn);
            const float d = __fmul_rn(half_bits_to_float(ld_u16(w)), (float)sc), m = __fmul_rn(half_bits_to_float(ld_u16(w + 2)), (float)mn);
            uint32_t q = (w[(T == GT_Q5_K ? 48 : 16) + 32 * (j >> 1) + l] >> (4 * (j & 1u))) & 15u;
            if (T == GT_Q5_K) q |= ((w[16 + l] >> j) & 1u) << 4;
            acc = fmaf(__fsub_rn(__fmul_rn(d, (float)q), m), x[256 * b + e], acc);
        }
    return acc;
}

// The tiles of all entries and ops form one line, of which every cluster takes a share, in steps.  A chunk: the next tiles of
// the share, `nt` of op `op` for entry `ent` from the op's tile `tile` on.  Dense, one and two rows:
// steps of one tile, shares contiguous and equal; what is left of an op is cut into chunks of equal length (shares of whole chunks of four leave a last round part
// empty: Q4_0 24576 x 4096 has 384 such chunks for 296 CTAs, or 1536 tiles).  Otherwise steps of a chunk.  Three and four rows: dealt out in turn (in f16 a
// chunk's sums and descriptions cost more than an uneven last round: steps of a tile took 12.8 us where 11.6 do for 6144 x 4096 Q4_0, 14.0 / 12.3 Q8_0, Q4_0
// 49152 x 2048 27.1 / 23.4, 151936 x 1024 40.5 / 38.0).  Routed: contiguous (a share that crosses into another entry has its activations to split, 16 pairs of
// 768 x 2048 12.9 us, 15.7 in steps of a tile).  Eight rows: of activations that are better loaded by fewer CTAs.
struct __align__(16) SpChunk {
    uint32_t ent, op, tile, nt;
    uint32_t un, key, e0, cnt;   // this rank's units; the same key: the same activations; the entry's first row or pair and their number
    uint32_t steps;              // to the next one
};
__device__ __forceinline__ SpChunk sp_chunk(const SpBatch &b, uint32_t pos, uint32_t last) {
    SpChunk c;
    const uint32_t all = b.op[b.nops - 1].step_end;
    c.ent = pos < all ? 0u : pos / all;
    const uint32_t r = pos - c.ent * all;
    c.op = 0;
    uint32_t from = 0, to = b.op[0].step_end;
    while (r >= to) {
        from = to;
        to = b.op[++c.op].step_end;
    }
    c.tile = (r - from) * b.step;
    const uint32_t left = min((b.op[c.op].n + 15u) / 16u - c.tile, (last - pos) * b.step);
    c.nt = min(b.tr, left);
    if (b.step == 1 && left > b.tr && left < 8 * b.tr) {   // (from eight chunks on: whole ones)
        uint32_t parts = 2;
        while (parts * b.tr < left) parts++;
        c.nt = (left + parts - 1) / parts;
    }
    return c;
}

// The row of a tile that lies at place p of its 16 in a stage (pairs: the even rows come first).
__device__ __forceinline__ uint32_t sp_row(uint32_t pairs, uint32_t p) { return pairs ? ((p & 7u) << 1) + (p >> 3) : p; }

// Packs activation rows into B register order for the kernel below: f16 hi + lo halves under one power of two per row, the sums of the
// sub-blocks that have offsets, and the inverse scale.  One block per row.  Several rows (or row groups: Q4_K has no other form
// for many rows) are packed once instead of by every CTA, where eight rows cost more time than the weights of a 12288 x 4096 matrix.
template <int T, bool ALN>
__global__ void __launch_bounds__(256) qmv_pack_kernel(const __grid_constant__ SpBatch bt) {
    constexpr int NG = SpTraits<T>::NG;
    __shared__ float s_am[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, q = (tid >> 2) & 3u, tt = tid & 3u;
    uint32_t op = 0;   // (ops that share another's activations have no rows of their own here)
    while (blockIdx.x >= bt.op[op].row_end) op++;
    const SpOp &P = bt.op[op];
    const size_t row = blockIdx.x - (op ? bt.op[op - 1].row_end : 0u);
    const uint32_t k = P.k, units = P.units, pk_units = P.pk_units;
    const float *x = P.x;
    uint8_t *xp = const_cast<uint8_t *>(P.xp);
    float *xsum = const_cast<float *>(P.xsum), *xinv = const_cast<float *>(P.xinv);
    grid_dependency_wait();
    allow_dependents();   // (not earlier: the kernel behind may overwrite what this one's predecessors still read)
    const float *xr = x + row * k;
    auto load = [&](uint32_t u, float (&v)[4]) {
        uint32_t p0, p1;
        sp_pairs<T, ALN>(u, q, tt, p0, p1);
        const uint32_t kb = T == GT_Q6_K ? 256u * (u >> 2) : 64u * u;
        v[0] = v[1] = v[2] = v[3] = 0.f;
        if (u >= units) return;
        if (kb + p0 < k) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(xr + kb + p0));
        if (kb + p1 < k) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[2]), "=f"(v[3]) : "l"(xr + kb + p1));
    };
    constexpr int HELD = 8;   // a pass of the block takes 16 units; K = 8192 stays in registers
    float v[HELD][4], am = 0.f;
#pragma unroll
    for (int p = 0; p < HELD; p++) {
        if (16u * p >= pk_units) break;
        load(16u * p + (tid >> 4), v[p]);
    }
#pragma unroll
    for (int p = 0; p < HELD; p++) {
        if (16u * p >= pk_units) break;
#pragma unroll
        for (int e = 0; e < 4; e++) am = fmaxf(am, fabsf(v[p][e]));
    }
    for (uint32_t u = 16u * HELD + (tid >> 4); u < pk_units; u += 16) {
        float z[4];
        load(u, z);
#pragma unroll
        for (int e = 0; e < 4; e++) am = fmaxf(am, fabsf(z[e]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (lane == 0) s_am[warp] = am;
    __syncthreads();
    am = s_am[lane & 7u];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    float s, inv;
    sp::pow2(am, s, inv);
    if (tid == 0) xinv[row] = inv;
    auto put = [&](uint32_t u, const float (&z)[4]) {
        const float c[4] = {z[0] * s, z[1] * s, z[2] * s, z[3] * s};
        float sum = 0.f;
        if constexpr (NG != 0) {
            sum = (c[0] + c[1]) + (c[2] + c[3]);
#pragma unroll
            for (int o = 1; o <= 4; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        uint2 hi, lo;
        sp::split(c[0], c[2], hi.x, lo.x);
        sp::split(c[1], c[3], hi.y, lo.y);
        if (u >= pk_units) return;
        uint2 *d = reinterpret_cast<uint2 *>(xp + row * P.xp_row + (u >> 2) * P.xp_super + (u & 3u) * 256u + (q >> 1) * 128u + tt * 32u + (q & 1u) * 8u);
        const uint32_t odd = P.wide_rows ? row & 1u : 0u;
        d[2 * odd] = hi;
        d[2 - 2 * odd] = lo;
        if (NG != 0 && (tid & 7u) == 0) {
            const size_t at = P.wide_rows ? ((size_t)(u >> 2) * P.wide_rows + (row & ~7u)) * 8 + ((u & 3u) * 2 + (q >> 1)) * 8 + (row & 7u)
                                          : (row * pk_units + u) * NG + (q >> 1);
            xsum[at] = sum;
        }
    };
#pragma unroll
    for (int p = 0; p < HELD; p++) {
        if (16u * p >= pk_units) break;
        put(16u * p + (tid >> 4), v[p]);
    }
    for (uint32_t u0 = 16u * HELD; u0 < pk_units; u0 += 16) {
        float z[4];
        load(u0 + (tid >> 4), z);
        put(u0 + (tid >> 4), z);
    }
}

// A warp's share of up to two activation rows in halves, where digits would lose its small values (see `far` in the kernel): a power of two for
// every 32 values (lanes 8 j .. 8 j + 7 hold them), as one for the share (inv: its inverse) and one beside it for the 32, whose inverse's exponent goes to
// rel[unit][row][32 values].  x: the entry's first row, from the rank's slice on; left: values from there to the end of the row.
template <int T, bool ALN, int MPC>
__device__ __forceinline__ void sp_far(const float *x, uint32_t k, uint32_t left, uint32_t cnt, uint32_t un, uint32_t warp, uint32_t lane,
                                       uint32_t xf, uint32_t xs, [[maybe_unused]] uint32_t ccb, [[maybe_unused]] uint32_t cs, float *inv, uint8_t *rel) {
    constexpr int NG = SpTraits<T>::NG;
    const uint32_t q = (lane >> 2) & 3u, tt = lane & 3u, hf = lane >> 4;
    uint32_t p0, p1;
    sp_pairs<T, ALN>(warp, q, tt, p0, p1);
    auto load = [&](uint32_t row, uint32_t u, float (&v)[4]) {
        v[0] = v[1] = v[2] = v[3] = 0.f;
        if (u >= un) return;
        const uint32_t o = T == GT_Q6_K ? 256u * (u >> 2) : 64u * u;
        const size_t at = (size_t)row * k + o;
        sp_act(x + at, nullptr, p0, p1, o + p0 < left, o + p1 < left, v);
    };
    for (uint32_t row = 0; row < cnt; row++) {
        uint32_t am = 0;
        for (uint32_t u = warp; u < un; u += 16) {
            float z[4];
            load(row, u + 8 * hf, z);
            am = max(am, sp::peak_bits(z));
        }
        am = __reduce_max_sync(0xffffffffu, am);
        float s, i;
        sp::pow2(__uint_as_float(am), s, i);
        if (lane == 0) inv[row] = i;
        for (uint32_t u = warp; u < un; u += 16) {
            const uint32_t mine = u + 8 * hf;
            float z[4];
            load(row, mine, z);
            uint32_t b = sp::peak_bits(z);
#pragma unroll
            for (int o = 1; o <= 4; o *= 2) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
            const uint32_t beside = min((am >> 23) - (b >> 23), 96u);   // (scales times 2^-96 are still normal numbers)
            const float s1 = __uint_as_float((127u + beside) << 23);
#pragma unroll
            for (int e = 0; e < 4; e++) z[e] = z[e] * s * s1;
            [[maybe_unused]] float sum = (z[0] + z[1]) + (z[2] + z[3]);
            if constexpr (NG != 0) {
#pragma unroll
                for (int o = 1; o <= 4; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            }
            uint32_t hi[2], lo[2];
            sp::split(z[0], z[2], hi[0], lo[0]);
            sp::split(z[1], z[3], hi[1], lo[1]);
            if (mine >= un) continue;
            const uint32_t d = xf + row * xs + mine * 256u + (q >> 1) * 128u + tt * 32u + (q & 1u) * 8u;
            sts64(d, hi[0], hi[1]);
            sts64(d + 16, lo[0], lo[1]);
            if ((lane & 7u) == 0) {
                rel[(mine * MPC + row) * 2 + (q >> 1)] = (uint8_t)(127u - beside);
                if constexpr (NG != 0) sts32(ccb + row * cs + (mine * NG + (q >> 1)) * 4u, __float_as_uint(sum));
            }
        }
    }
    __syncwarp();
}

// The stages of a chunk against such a share; the sums go to `part`.  Returns whether all copies came.
struct SpRing {
    uint64_t *full, *empty;
    volatile uint32_t *abort_flag;
    uint32_t base, slot, ph;
};
template <int T, bool ALN, int MPC>
__device__ __forceinline__ bool sp_far_stages(const SpBatch &bt, uint32_t op, uint32_t u0, uint32_t un, uint32_t nt, SpRing &ring, uint32_t warp, uint32_t lane, uint32_t xf,
                                               uint32_t ccb, uint32_t tab, uint32_t part, const float *inv, const uint8_t *rel) {
    using K = SpTraits<T>;
    constexpr int NG = K::NG, SU = K::SU, TM = sp_tiles(MPC);
    constexpr bool TABLE = T == GT_Q4_K || T == GT_Q5_K || T == GT_Q6_K;
    constexpr uint32_t PITCH = sp_pitch<T>(ALN), UB = T == GT_Q8_0 ? 68u : 36u;
    const SpOp &P = bt.op[op];
    const uint32_t g = lane >> 2, t = lane & 3u, row = MPC == 1 ? 0u : t & 1u, stage_bytes = bt.tr * 16u * PITCH, rb15 = P.row_bytes & 15u;
    const uint32_t xlane = xf + (MPC == 1 ? 0u : (g >> 1 & 1u) * bt.xstride) + (t * 2 + (g & 1u)) * 16u;
    float acc[TM][1][4];
#pragma unroll
    for (int j = 0; j < TM; j++) acc[j][0][0] = acc[j][0][1] = acc[j][0][2] = acc[j][0][3] = 0.f;
    bool ok = true;
    for (uint32_t us = 0; us == 0 || us < un; us += SU) {
        const uint32_t off = (u0 + us) / 4 * (uint32_t)K::B256, wl = ALN ? 0u : ((uint32_t)(uintptr_t)P.w + off) & 15u;
        auto lead = [&](uint32_t r) { return ALN ? (T == GT_Q6_K ? off & 15u : 0u) : (wl + sp_row(bt.pairs, r & 15u) * rb15) & 15u; };
        if (!mbar_wait(&ring.full[ring.slot], ring.ph, ring.abort_flag, bt.status, ST_WAIT_FULL_TIMEOUT, 0u)) {
            ok = false;
            break;
        }
        const uint32_t stage = ring.base + ring.slot * stage_bytes;
        for (uint32_t ul = warp; ul < (uint32_t)SU && us + ul < un; ul += kSpWarps) {
            const uint32_t uu = us + ul, ub = TABLE ? (ul >> 2) * (uint32_t)K::B256 : ul * UB;
            uint32_t bf[1][4][2], v[4];
            float cc[1][2];
            lds128i<0>(xlane + uu * 256u, v);
            bf[0][0][0] = v[0]; bf[0][0][1] = v[1]; bf[0][1][0] = v[2]; bf[0][1][1] = v[3];
            lds128i<128>(xlane + uu * 256u, v);
            bf[0][2][0] = v[0]; bf[0][2][1] = v[1]; bf[0][3][0] = v[2]; bf[0][3][1] = v[3];
#pragma unroll
            for (int q = 0; q < NG; q++) cc[0][q] = __uint_as_float(lds32(ccb + row * bt.cstride + (uu * NG + q) * 4u));
            const uint8_t *e = rel + (uu * MPC + row) * 2;
            const float f2[2] = {__uint_as_float((uint32_t)e[0] << 23), __uint_as_float((uint32_t)e[1] << 23)};
            if constexpr (TABLE) {
                __syncwarp();   // the table of the unit before has been read
                for (uint32_t r = lane; r < 16u * nt; r += 32) sp_table_row<T, false>(tab + r * 16, stage + r * PITCH + lead(r) + ub, ul);
                __syncwarp();
            }
            const bool half = (u0 + uu) * 64 + 32 >= P.k;   // (the second block of the last unit lies past the row)
            auto tiles = [&](auto NT) {
                sp_unit<T, ALN, decltype(NT)::value, true>(stage + g * PITCH + lead(g) + ub, stage + (g + 8) * PITCH + lead(g + 8) + ub, ul, t, g, tab, half, bf, cc, f2, acc);
            };
            if (nt == 1) tiles(std::integral_constant<int, 1>{});
            else if (nt == 2) tiles(std::integral_constant<int, 2>{});
            else if (nt == 3) tiles(std::integral_constant<int, 3>{});
            else tiles(std::integral_constant<int, TM>{});
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ring.empty[ring.slot]);
        if (++ring.slot == bt.nslots) {
            ring.slot = 0;
            ring.ph ^= 1u;
        }
    }
    if (t < (uint32_t)MPC)
#pragma unroll
        for (int j = 0; j < TM; j++)
            if (j < (int)nt) {
                const uint32_t a = part + (t * 16u * bt.tr + 16 * j + g) * 4;
                sts32(a, __float_as_uint((acc[j][0][0] + acc[j][0][1]) * inv[t]));
                sts32(a + 32, __float_as_uint((acc[j][0][2] + acc[j][0][3]) * inv[t]));
            }
    return ok;
}

// INT: one or two activation rows (MPC), in 8-bit integers (sp_unit_int), a set of columns each.  Otherwise f16: up to four in one set, up to eight in two; MPC 1: a
// single routed pair (its activations loaded as one row's: 768 x 2048 Q4_0 7.1 us, 7.8 with four rows' loads and reductions).
template <int T, bool ALN, int MPC, bool INT>
__global__ void __launch_bounds__(kSpThreads, 2) qmv_split_kernel(const __grid_constant__ SpBatch bt, const __grid_constant__ SpMaps maps) {
    using K = SpTraits<T>;
    constexpr int NS = INT ? MPC : MPC > 4 ? 2 : 1, NG = K::NG, SU = K::SU, TM = sp_tiles(MPC);
    constexpr bool TABLE = T == GT_Q4_K || T == GT_Q5_K || T == GT_Q6_K;
    constexpr uint32_t PITCH = sp_pitch<T>(ALN), TILE = 16 * PITCH;
    constexpr uint32_t UB = T == GT_Q8_0 ? 68u : 36u;               // bytes of a unit (Q4_0, Q8_0)

    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;      // (the same in every CTA of a cluster)
    __shared__ __align__(8) uint64_t full[kSpMaxSlots], empty[kSpMaxSlots], sync_bar[3], recv_bar[4], x_bar, c_bar;
    __shared__ float s_inv[kSpWarps][8];                            // inverse activation scales of a warp's share of K
    // integers, shares in halves (sp_far): exponents of the inverse scales of [unit][row][32 values], beside the share's
    __shared__ __align__(2) uint8_t s_rel[INT ? kSpMaxUnits * 2 : 2];
    __shared__ volatile uint32_t abort_flag, s_again;
    __shared__ uint32_t s_nent;
    __shared__ SpChunk s_chunk[16];                                 // the chunks in work
    constexpr int PAIRS = INT ? 1 : kSpMaxPairs;
    __shared__ uint16_t s_id[PAIRS];                                // routed: expert of every pair (there are at most 65535)
    __shared__ uint16_t s_ord[PAIRS], s_ent[PAIRS + 1];             // pairs by expert; entry e = pairs s_ord[s_ent[e] ..]
    __shared__ uint32_t s_wcnt[kSpWarps];
    const bool routed = !INT && bt.ids;                             // (routed products never leave in integers)

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t ranks, rank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    rank = sp::cluster_rank();
    const uint32_t mp = bt.mp, tr = bt.tr, R = 16u * tr, STAGE = tr * TILE;
    auto place = [&](uint32_t p) { return MPC > 4 ? p : sp_row(bt.pairs, p); };   // (eight rows: registers are short, rows off boundaries come one by one)

    if (tid == 0) {
        abort_flag = s_again = 0;
        for (uint32_t s = 0; s < bt.nslots; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kSpWarps);
        }
        for (int s = 0; s < 3; s++) mbar_init(&sync_bar[s], kSpWarps);
        for (int s = 0; s < 4; s++) mbar_init(&recv_bar[s], 1);
        mbar_init(&x_bar, 1);
        mbar_init(&c_bar, kSpWarps);
        mbar_init_fence();
    }
    if (routed) {
        grid_dependency_wait();   // the expert ids belong to the kernels ahead
        for (uint32_t p = tid; p < kSpMaxPairs; p += kSpThreads) s_id[p] = p < bt.npairs ? (uint16_t)min(__ldcg(bt.ids + p), bt.n_experts) : (uint16_t)0xFFFFu;
    }
    __syncwarp();
    if (ranks > 1) sp::cluster_sync();   // the others' barriers exist before anything is sent there
    else __syncthreads();
    allow_dependents();
    if (routed) {
        // rank of every pair by (expert, pair); an entry starts at every mp-th pair of an expert
        uint32_t pos = 0, before = 0, me = 0;
        if (tid < bt.npairs) {
            me = s_id[tid];
            for (uint32_t q = 0; q < bt.npairs; q++) {
                const uint32_t o = s_id[q];
                const bool eq = o == me && q < tid;
                before += eq ? 1u : 0u;
                pos += (o < me || eq) ? 1u : 0u;
            }
            s_ord[pos] = (uint16_t)(tid | (before % mp == 0 ? 0x8000u : 0u));
        }
        __syncthreads();
        bool start = false;
        if (tid < bt.npairs) {
            const uint32_t v = s_ord[tid];
            start = (v & 0x8000u) != 0;
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, start);
        if (warp < kSpWarps && lane == 0) s_wcnt[warp] = __popc(bal);
        __syncthreads();
        uint32_t at = 0, total = 0;
        for (uint32_t w = 0; w < kSpWarps; w++) {
            if (w < warp) at += s_wcnt[w];
            total += s_wcnt[w];
        }
        if (start) s_ent[at + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)tid;
        if (tid == 0) {
            s_ent[total] = (uint16_t)bt.npairs;
            s_nent = total;
        }
        if (tid < bt.npairs) s_ord[tid] &= 0x7FFFu;
        __syncthreads();
    }
    const uint32_t nent = routed ? s_nent : bt.nent;
    // this cluster's share of the tiles
    const uint32_t ncl = gridDim.x / ranks, cl = blockIdx.x / ranks;
    const uint64_t steps = (uint64_t)nent * bt.op[bt.nops - 1].step_end;
    // (whole chunks: as many for every cluster as the fullest one has, so that fewer shares cross into another entry: gate and up, 20 pairs of 16
    // experts, 768 x 2560 Q4_K, the layer 61 us, 66 with equal shares)
    const uint64_t most = (steps + ncl - 1) / ncl;
    const uint32_t first = bt.step == 1 ? (uint32_t)(steps * cl / ncl) : bt.dealt ? cl : (uint32_t)min(steps, most * cl);
    const uint32_t last = bt.step == 1 ? (uint32_t)(steps * (cl + 1) / ncl) : bt.dealt ? (uint32_t)steps : (uint32_t)min(steps, most * (cl + 1));
    auto stages_of = [&](uint32_t at) {   // (what the copies need to know)
        SpChunk c = sp_chunk(bt, at, last);
        const SpOp &P = bt.op[c.op];
        const uint32_t u0 = rank * P.slice;
        c.un = u0 < P.units ? min(P.slice, P.units - u0) : 0u;
        c.steps = bt.step == 1 ? c.nt : bt.dealt ? ncl : 1u;
        c.e0 = routed ? s_ent[c.ent] : 0u;
        return c;
    };
    auto chunk = [&](uint32_t at) {
        SpChunk c = stages_of(at);
        const SpOp &P = bt.op[c.op];
        if (routed) {
            c.cnt = s_ent[c.ent + 1] - c.e0;
        } else {
            c.e0 = c.ent * mp;
            c.cnt = min(mp, P.m - c.e0);
        }
        c.key = c.ent * kSpMaxOps + P.xkey;
        return c;
    };

    if (warp == kSpWarps) {
        // ======================= producer =======================
        if (!bt.early_weights) grid_dependency_wait();
        uint64_t pol;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
        uint32_t slot = 0, ph = 1;   // (a slot's first wait passes)
        bool ok = true;
        for (uint32_t at = first, i = 0; ok && at < last; i++) {
            const SpChunk c = INT ? chunk(at) : stages_of(at);
            at += c.steps;
            const SpOp &P = bt.op[c.op];
            const uint32_t u0 = rank * P.slice;
            const uint32_t ex = routed ? s_id[s_ord[c.e0]] : 0u;
            // (integers, a rank without units for the chunk: a stage without data, so that the consumers get the chunk's description with it)
            for (uint32_t u = 0; (INT && u == 0) || u < c.un; u += SU) {
                if (!mbar_wait(&empty[slot], ph, &abort_flag, bt.status, ST_WAIT_EMPTY_TIMEOUT, 0u)) {
                    ok = false;
                    break;
                }
                const uint32_t dst = base + slot * STAGE;
                const uint32_t off = (u0 + u) / 4 * (uint32_t)K::B256;
                // Sixteen descriptions are enough: the one written here was last read for a chunk 16 before, and the slot that the wait above
                // found empty was left by warps that have arrived for chunk i - 2 - kSpMaxSlots at least.
                if (INT && u == 0 && lane == 0) s_chunk[i & 15u] = c;
                if (INT && c.un == 0) {
                    if (lane == 0) mbar_arrive(&full[slot]);
                } else if constexpr (ALN) {
                    if (lane == 0) {
                        mbar_expect_tx(&full[slot], c.nt * TILE);
                        for (uint32_t j = 0; j < c.nt; j++)
                            asm volatile(
                                "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
                                ::"r"(dst + j * TILE), "l"(&maps.m[c.op]), "r"((off & ~15u) >> 3), "r"((c.tile + j) * 16u), "r"(ex),
                                  "r"(smem_u32(&full[slot])), "l"(pol)
                                : "memory");
                    }
                } else if (MPC <= 4 && bt.pairs) {
                    // A row of the tensor map is two weight rows, a copy the even or the odd rows of a tile (see sp_row).  (Four or eight weight
                    // rows a map row would do for any address, but copies have to start on 128 bytes, where their rows would meet in the
                    // same banks.)
                    if (lane == 0) {
                        mbar_expect_tx(&full[slot], c.nt * TILE);
                        for (uint32_t j = 0; j < c.nt; j++)
#pragma unroll
                            for (uint32_t r = 0; r < 2; r++)
                                asm volatile(
                                    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
                                    ::"r"(dst + j * TILE + r * 8 * PITCH), "l"(&maps.m[c.op]), "r"(((r * P.row_bytes + off) & ~15u) >> 3),
                                      "r"((c.tile + j) * 8u), "r"(ex), "r"(smem_u32(&full[slot])), "l"(pol)
                                    : "memory");
                    }
                } else {
                    // one bulk copy per row: the 16-byte superset of the row's segment (an expert that does not exist: expert 0,
                    // whose products are not stored)
                    const uint32_t len = min((uint32_t)(SU / 4 * K::B256), P.row_bytes - off);
                    const uint8_t *w = P.w + (ex < bt.n_experts ? (uint64_t)ex * P.expert_stride : 0ull) + off;
                    uint32_t tx = 0;
                    for (uint32_t r = lane; r < c.nt * 16u; r += 32) {
                        const uint32_t row = c.tile * 16u + r;
                        if (row < P.n) tx += (((uint32_t)(uintptr_t)(w + (uint64_t)row * P.row_bytes) & 15u) + len + 15u) & ~15u;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) tx += __shfl_xor_sync(0xffffffffu, tx, o);
                    if (lane == 0) mbar_expect_tx(&full[slot], tx);
                    __syncwarp();
                    for (uint32_t r = lane; r < c.nt * 16u; r += 32) {
                        const uint32_t row = c.tile * 16u + r;
                        if (row >= P.n) continue;
                        const uintptr_t src = (uintptr_t)(w + (uint64_t)row * P.row_bytes);
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                                         dst + r * PITCH),
                                     "l"(src & ~(uintptr_t)15), "r"((((uint32_t)src & 15u) + len + 15u) & ~15u), "r"(smem_u32(&full[slot])), "l"(pol)
                                     : "memory");
                    }
                }
                if (++slot == bt.nslots) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        }
    } else {
        // ======================= consumers =======================
        const uint32_t g = lane >> 2, t = lane & 3u;
        const uint32_t xf = base + bt.xf_off, ccb = base + bt.cc_off, tab = base + bt.tab_off + warp * (R * 16u), red = base + bt.red_off;
        const uint32_t xs = bt.xstride, cs = bt.cstride;
        // integers: column g is digit g % 4 of the set's row in group g / 4; a lane scales columns 2 t and 2 t + 1, which are of group t / 2
        const uint32_t xlane = INT ? xf + (g & 3u) * 64u + t * 16u : xf + ((g >> 1) & (mp - 1)) * xs + (t * 2 + (g & 1u)) * 16u;
        const uint32_t clane = ccb + (INT ? (t >> 1) * 4u : (t & (mp - 1)) * cs);
        uint32_t slot = 0, ph = 0, cur = 0xFFFFFFFFu;
        bool ok = true;
        [[maybe_unused]] uint32_t bias[4];
        if constexpr (INT) {
#pragma unroll
            for (int q = 0; q < 4; q++) asm volatile("mov.u32 %0, %1;" : "=r"(bias[q]) : "n"(sp::kBias));
        }
        auto wait = [&](uint64_t &bar, uint32_t parity, uint32_t code) {
            ok = mbar_wait(&bar, parity, &abort_flag, bt.status, code, 0u) && ok;
            return ok;
        };
        auto store = [&](const SpChunk &d, uint32_t col, uint32_t row, float v) {
            const SpOp &P = bt.op[d.op];
            const uint32_t grow = d.tile * 16u + (ALN ? row : (row & ~15u) + place(row & 15u));
            if (col >= d.cnt || row >= d.nt * 16u || grow >= P.n) return;
            const uint32_t pair = routed ? (uint32_t)s_ord[d.e0 + col] : d.e0 + col;
            const size_t o = (size_t)pair * P.y_ld + P.y_col0 + grow;
            if (routed && s_id[pair] >= bt.n_experts) v = 0.f;   // an id that names no expert
            if (NG != 0 && v != v) s_again = 1;
            P.y[o] = v;
            for (uint32_t pr = 0; pr < P.n_peer; pr++) P.y_peer[pr][o] = v;
        };
        [[maybe_unused]] auto again = [&](const SpChunk &d, uint32_t col, uint32_t row, uint32_t parts) {
            const SpOp &P = bt.op[d.op];
            const uint32_t grow = d.tile * 16u + (ALN ? row : (row & ~15u) + place(row & 15u));
            if (col >= d.cnt || row >= d.nt * 16u || grow >= P.n) return;
            const uint32_t pair = routed ? (uint32_t)s_ord[d.e0 + col] : d.e0 + col;
            const size_t o = (size_t)pair * P.y_ld + P.y_col0 + grow;
            if (P.y[o] == P.y[o]) return;
            float v = sp_again<T>(P.w + (routed ? s_id[pair] * P.expert_stride : 0ull) + (uint64_t)grow * P.row_bytes,
                                  P.x + (size_t)(routed ? pair / P.x_div : pair) * P.k, P.k, tid % parts, parts);
            if (parts == 4) {
                const uint32_t four = 0xFu << (lane & 28u);
                v += __shfl_xor_sync(four, v, 1);
                v += __shfl_xor_sync(four, v, 2);
                if (tid & 3u) return;
            }
            P.y[o] = v;
            for (uint32_t pr = 0; pr < P.n_peer; pr++) P.y_peer[pr][o] = v;
        };
        const uint32_t share = R / ranks;   // rows of a chunk that a rank finishes
        const uint32_t RS = mp * R + (INT ? 8 : 0);   // floats from one warp's sums to the next (integers: what four lanes read is in distinct banks)
        // the CTA's sums of chunk j, in warp order: results, or for the rank that finishes the row
        auto add = [&](uint32_t j, uint32_t at) {
            if (!wait(sync_bar[j & 1u], (j >> 1) & 1u, ST_WAIT_EMPTY_TIMEOUT)) return false;
            const SpChunk d = s_chunk[at];
            const uint32_t part = red + (INT ? j & 3u : j & 1u) * (kSpWarps * RS * 4u), buf = j & 3u;
            if (INT && ranks == 1) {   // four lanes a result, two warps' sums each
                for (uint32_t q = tid >> 2; q < (MPC == 1 ? 16u * d.nt : mp * R); q += kSpWarps * 8) {
                    const uint32_t a = part + ((tid & 3u) * RS + q) * 4;
                    float v = __uint_as_float(lds32(a)) + __uint_as_float(lds32(a + 16 * RS));
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    const uint32_t col = MPC == 1 || q < R ? 0u : 1u;
                    if ((tid & 3u) == 0) store(d, col, q - col * R, v);
                }
            } else
            for (uint32_t q = tid; q < mp * R; q += 256) {
                const uint32_t col = q / R, row = q - col * R;
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < kSpWarps; w++) v += __uint_as_float(lds32(part + (w * RS + q) * 4));
                if (ranks == 1) {
                    store(d, col, row, v);
                } else {
                    const uint32_t to = row / share;
                    const uint32_t a = base + bt.recv_off + (((buf * ranks + rank) * mp + col) * share + row - to * share) * 4;
                    sp::st_async(sp::map_rank(a, to), v, sp::map_rank(smem_u32(&recv_bar[buf]), to));
                }
            }
            __syncwarp();
            if (!INT && lane == 0) mbar_arrive(&sync_bar[2]);
            if (ranks > 1 && tid == 0) mbar_expect_tx(&recv_bar[buf], mp * R * 4u);
            return true;
        };
        // The ranks' sums of chunk j, in rank order.  Four buffers are enough although other warps of this rank send and read on:
        // chunk j + 4 comes here from a rank all of whose warps have finished j + 2; that takes rows of j + 2 sent by this rank,
        // which its warps send only once every one of them has arrived on sync_bar for j + 2; and a warp does that after it has read
        // chunk j here.
        auto finish = [&](uint32_t j, uint32_t at) {
            const uint32_t buf = j & 3u;
            const SpChunk d = s_chunk[at];
            if (!wait(recv_bar[buf], (j >> 2) & 1u, ST_WAIT_FULL_TIMEOUT)) return false;
            for (uint32_t q = tid; q < mp * share; q += 256) {
                const uint32_t col = q / share, row = q - col * share;
                float v = 0.f;
                for (uint32_t r = 0; r < ranks; r++) v += __uint_as_float(lds32(base + bt.recv_off + (((buf * ranks + r) * mp + col) * share + row) * 4));
                store(d, col, rank * share + row, v);
            }
            return true;
        };
        uint32_t x_ph = 0, c_ph = 0;
        auto csync = [&]() {   // all warps
            __syncwarp();
            if (lane == 0) mbar_arrive(&c_bar);
            const bool r = wait(c_bar, c_ph, ST_WAIT_EMPTY_TIMEOUT);
            c_ph ^= 1u;
            return r;
        };
        uint32_t d1 = 0, d2 = 0;   // where the descriptions of the last two chunks are
        uint32_t i = 0;   // the CTA's chunks so far
        // (Integers: what the first chunk needs of the launch's parameters is fetched before the wait.)
        [[maybe_unused]] SpChunk c0{};
        if constexpr (INT) {
            c0 = chunk(first < last ? first : 0);
            const SpOp &P = bt.op[c0.op];
            asm volatile("" ::"l"(P.x), "r"(P.k), "r"(P.slice));
        }
        if (!routed) grid_dependency_wait();   // the activations belong to the kernels ahead until those are done
        uint32_t at = first;
        for (; ok && at < last; i++) {
            SpChunk c;
            if (!INT) {
                c = chunk(at);
            } else if (i == 0) {
                c = c0;
            } else {   // the producer's description comes with the first stage
                if (!wait(full[slot], ph, ST_WAIT_FULL_TIMEOUT)) break;
                c = s_chunk[i & 15u];
            }
            // (f16: the copies start without it.  Who comes here for chunk i + 16 has found every warp's arrival for chunk i + 14, and a warp arrives
            // there after it has read what belongs to chunk i.)
            if (!INT && tid == 0) s_chunk[i & 15u] = c;
            at += c.steps;
            const SpOp &P = bt.op[c.op];
            const uint32_t u0 = rank * P.slice, un = c.un, e0 = c.e0, cnt = c.cnt, key = c.key;
            [[maybe_unused]] const uint32_t ex = routed && !ALN ? s_id[s_ord[e0]] : 0u;
            if (!INT && key != cur && bt.packed) {
                // the rows' slices come ready from the pack kernel's scratch area
                if (cur != 0xFFFFFFFFu && !csync()) break;   // nobody reads the entry before any more
                cur = key;
                const uint32_t un4 = (un + 3) & ~3u, xb = un4 * 256u, cb = un4 * NG * 4u;
                if (warp == 0) {
                    if (lane == 0) mbar_expect_tx(&x_bar, cnt * (xb + cb));
                    __syncwarp();
                    if (lane < cnt && un) {
                        const uint8_t *px = P.xp + ((size_t)(e0 + lane) * P.pk_units + u0) * 256u;
                        bulk_g2s_a(xf + lane * xs, px, xb, &x_bar);
                        if constexpr (NG != 0)
                            bulk_g2s_a(ccb + lane * cs, reinterpret_cast<const uint8_t *>(P.xsum) + ((size_t)(e0 + lane) * P.pk_units + u0) * (NG * 4u), cb, &x_bar);
                    }
                }
                if (lane < cnt) s_inv[warp][lane] = __ldcg(P.xinv + e0 + lane);
                if (!wait(x_bar, x_ph, ST_WAIT_FULL_TIMEOUT)) break;
                x_ph ^= 1u;
                __syncwarp();
            }
            if (key != cur) {
                [[maybe_unused]] bool far = false;   // digits do not do for the share
                // ---- the entry's activations of this warp's units: f16 hi + lo in B register order.  A pass takes two units
                // (lane = (unit of the pass, MMA q, quad lane tt), four values each) ----
                cur = key;
                const uint32_t q = (lane >> 2) & 3u, tt = lane & 3u, hf = lane >> 4;
                uint32_t p0, p1;
                sp_pairs<T, ALN>(warp, q, tt, p0, p1);
                const uint32_t kb = (T == GT_Q6_K ? 256u * ((u0 + warp) >> 2) : 64u * (u0 + warp)) + 512u * hf;
                const uint32_t mine = un > warp ? (un - warp + 7) / 8 : 0u;          // the warp's units
                // a pass's values: the sums of the sub-blocks, and the halves or digits
                const uint32_t d0 = xf + (INT ? (warp + 8 * hf) * 256u + tt * 16u + q * 4u : ((warp + 8 * hf) * 2 + (q >> 1)) * 128u + tt * 32u + (q & 1u) * 8u);
                auto write = [&](const float (&z)[4], float s, float s1, uint32_t p, uint32_t row, bool mine_too) {
                    float c[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) c[e] = INT ? z[e] * s * s1 : z[e] * s;
                    [[maybe_unused]] float sum = 0.f;
                    if constexpr (NG != 0) {
                        sum = (c[0] + c[1]) + (c[2] + c[3]);
#pragma unroll
                        for (int o = 1; o <= 4; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                        if constexpr (INT) sum *= 1.f / (256.f * sp_code_scale<T>);   // (in units of the top digit and of the codes)
                    }
                    uint32_t l[4];
                    if constexpr (INT) {
                        sp::digits(c, l);
                    } else {
                        sp::split(c[0], c[2], l[0], l[2]);
                        sp::split(c[1], c[3], l[1], l[3]);
                    }
                    if (2 * p + hf >= mine || !mine_too) return;
                    const uint32_t d = d0 + p * 4096u + row * xs;
                    if constexpr (INT) {
#pragma unroll
                        for (int i = 0; i < 4; i++) sts32(d + 64 * i, l[i]);
                    } else {
                        sts64(d, l[0], l[1]);
                        sts64(d + 16, l[2], l[3]);
                    }
                    if (NG != 0 && (lane & 7u) == 0) sts32(ccb + ((warp + 8 * hf) * NG + (q >> 1)) * 4u + p * (64u * NG) + row * cs, __float_as_uint(sum));
                };
                __syncwarp();
                if constexpr (INT) {
                    uint32_t from[MPC];   // (below 2^31 for a product: qmv_split_fits)
#pragma unroll
                    for (int r = 0; r < MPC; r++) from[r] = (e0 + min((uint32_t)r, cnt - 1)) * P.k + kb;
                    auto load = [&](int r, uint32_t p, float (&v)[4]) {
                        v[0] = v[1] = v[2] = v[3] = 0.f;
                        const uint32_t o = 1024u * p, at = from[r] + o;
                        if (2 * p + hf >= mine) return;
                        sp_act(P.x + at, nullptr, p0, p1, kb + o + p0 < P.k, kb + o + p1 < P.k, v);
                    };
                    auto peak = [](const float (&v)[4]) { return sp::peak_bits(v); };
                    // Passes whose values stay in registers; those beyond are loaded again.  (Two rows have no registers for four: Q4_K 24576 x 4096 28.0 us, so
                    // 26.6; Q4_0 21.4, 20.8.)
                    constexpr int HELD = MPC == 2 ? 2 : 4;
                    float v[MPC][HELD][4], s[MPC], s1[MPC];
                    uint32_t am[MPC];
#pragma unroll
                    for (int r = 0; r < MPC; r++)
#pragma unroll
                        for (int p = 0; p < HELD; p++) load(r, p, v[r][p]);
#pragma unroll
                    for (int r = 0; r < MPC; r++) {
                        am[r] = 0;
#pragma unroll
                        for (int p = 0; p < HELD; p++) am[r] = max(am[r], peak(v[r][p]));
                        for (uint32_t p = HELD; 2 * p < mine; p++) {
                            float z[4];
                            load(r, p, z);
                            am[r] = max(am[r], peak(z));
                        }
                        am[r] = __reduce_max_sync(0xffffffffu, am[r]);
                        float inv0, inv1;
                        sp::pow2_int(am[r], s[r], s1[r], inv0, inv1);
                        if (lane == 0) {
                            s_inv[warp][2 * r] = inv0 * sp_code_scale<T>;
                            s_inv[warp][2 * r + 1] = inv1;
                        }
                    }
                    // Digits have one last place for all of the share, 2^-28 of its largest value or less, and small values beside a large one would lose to
                    // it what halves keep.  So the share goes in halves (sp_far) unless every 32 values that are not all zero, and half of all fours that are
                    // not, hold one of 2^-6 of the largest or more.  (Normal activations and their products, as after SwiGLU, are so; one of 90 deviations or
                    // more beside normal ones is not.)  Error of a result whose weight for the large ones is zero, of the 2-norm of its terms, Q4_0, one of R
                    // deviations in every 512 values, digits / halves under one power of two a share / what leaves here: R = 60 8.6e-8 / 9.8e-8 / 8.6e-8,
                    // 300 1.6e-7 / 9.8e-8 / 8.6e-8, 1e4 4.4e-6 / 9.8e-8 / 8.6e-8, 1e6 2.8e-4 / 3.9e-7 / 2.8e-7.  It costs 7 us of 17.5 (24576 x 4096), 60 of
                    // 145 (Q6_K, 151936 x 5120), also where it is one warp's share alone.
#pragma unroll
                    for (int r = 0; r < MPC; r++) {
                        const uint32_t least = am[r] > (7u << 23) ? am[r] - (6u << 23) : 1u;
                        sp::Spread spread;
#pragma unroll
                        for (int p = 0; p < HELD; p++)
                            if (2u * p < mine) {
                                spread.look(peak(v[r][p]), least, lane);
                                write(v[r][p], s[r], s1[r], p, r, r < (int)cnt);
                            }
                        for (uint32_t p = HELD; 2 * p < mine; p++) {
                            float z[4];
                            load(r, p, z);
                            spread.look(peak(z), least, lane);
                            write(z, s[r], s1[r], p, r, r < (int)cnt);
                        }
                        far = far || spread.far() || am[r] >= 0x7F800000u;   // (halves hold infinities)
                    }
                } else if constexpr (MPC == 1) {
                    const size_t o = (size_t)((uint32_t)s_ord[e0] / P.x_div) * P.k + kb;
                    const float *x = P.x + o, *y = P.x2 ? P.x2 + o : nullptr;
                    auto load = [&](uint32_t p, float (&v)[4]) {
                        v[0] = v[1] = v[2] = v[3] = 0.f;
                        const uint32_t o = 1024u * p;
                        if (2 * p + hf >= mine) return;
                        sp_act(x + o, y ? y + o : nullptr, p0, p1, kb + o + p0 < P.k, kb + o + p1 < P.k, v);
                    };
                    auto peak = [](const float (&v)[4]) { return fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))); };
                    constexpr int HELD = 4;
                    float v[HELD][4], am = 0.f, s, inv;
#pragma unroll
                    for (int p = 0; p < HELD; p++) load(p, v[p]);
#pragma unroll
                    for (int p = 0; p < HELD; p++) am = fmaxf(am, peak(v[p]));
                    for (uint32_t p = HELD; 2 * p < mine; p++) {
                        float z[4];
                        load(p, z);
                        am = fmaxf(am, peak(z));
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
                    sp::pow2(am, s, inv);
                    if (lane == 0) s_inv[warp][0] = inv;
#pragma unroll
                    for (int p = 0; p < HELD; p++)
                        if (2u * p < mine) write(v[p], s, 1.f, p, 0, true);
                    for (uint32_t p = HELD; 2 * p < mine; p++) {
                        float z[4];
                        load(p, z);
                        write(z, s, 1.f, p, 0, true);
                    }
                } else {
                // Four passes are in flight at a time: of one row, or of two or four rows where a row has fewer.
                const uint32_t passes = (mine + 1) / 2, sh = passes <= 1 ? 0u : passes == 2 ? 1u : 2u, rows = 4u >> sh;
                for (uint32_t rb = 0; rb < cnt; rb += rows) {
                    const float *x[4], *y[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t r = min(rb + (j >> sh), cnt - 1);
                        const size_t o = (size_t)(routed ? (uint32_t)s_ord[e0 + r] / P.x_div : e0 + r) * P.k + kb;
                        x[j] = P.x + o;
                        y[j] = P.x2 ? P.x2 + o : nullptr;
                    }
                    auto load = [&](const float *xr, const float *yr, uint32_t p, float (&v)[4]) {
                        v[0] = v[1] = v[2] = v[3] = 0.f;
                        const uint32_t o = 1024u * p;
                        if (2 * p + hf >= mine) return;
                        const bool i0 = kb + o + p0 < P.k, i1 = kb + o + p1 < P.k;
                        if (i0) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(xr + o + p0));
                        if (i1) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v[2]), "=f"(v[3]) : "l"(xr + o + p1));
                        if (yr) {   // silu(gate) * up, as src/shaders/silu_mul.metal:17-30
                            float w[4] = {0.f, 0.f, 0.f, 0.f};
                            if (i0) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(w[0]), "=f"(w[1]) : "l"(yr + o + p0));
                            if (i1) asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(w[2]), "=f"(w[3]) : "l"(yr + o + p1));
#pragma unroll
                            for (int e = 0; e < 4; e++) v[e] = v[e] / (1.0f + expf(-v[e])) * w[e];
                        }
                    };
                    auto peak = [](const float (&v)[4]) { return fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))); };
                    float v[4][4], am[4], s[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) load(x[j], y[j], j & ((1u << sh) - 1u), v[j]);
#pragma unroll
                    for (int j = 0; j < 4; j++) am[j] = peak(v[j]);
                    for (uint32_t p = 4; p < passes; p++) {   // a long row: its other passes are loaded twice
                        float z[4];
                        load(x[0], y[0], p, z);
                        am[0] = fmaxf(am[0], peak(z));
                    }
                    if (sh == 1) {
                        am[0] = fmaxf(am[0], am[1]);
                        am[2] = fmaxf(am[2], am[3]);
                    } else if (sh == 2) {
                        am[0] = fmaxf(fmaxf(am[0], am[1]), fmaxf(am[2], am[3]));
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                        for (int j = 0; j < 4; j++) am[j] = fmaxf(am[j], __shfl_xor_sync(0xffffffffu, am[j], o));
                    if (sh == 1) {
                        am[1] = am[0];
                        am[3] = am[2];
                    } else if (sh == 2) {
                        am[1] = am[2] = am[3] = am[0];
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {   // one power of two brings the row's largest value into [2^13, 2^14)
                        float inv;
                        sp::pow2(am[j], s[j], inv);
                        if (lane == 0 && rb + (j >> sh) < cnt) s_inv[warp][rb + (j >> sh)] = inv;
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) write(v[j], s[j], 1.f, j & ((1u << sh) - 1u), rb + (j >> sh), rb + (j >> sh) < cnt);
                    for (uint32_t p = 4; p < passes; p++) {
                        float z[4];
                        load(x[0], y[0], p, z);
                        write(z, s[0], 1.f, p, rb, true);
                    }
                }
                }
                __syncwarp();
                if (INT && far) {
                    at -= c.steps;
                    break;
                }
            }

            float acc[TM][NS][4];
#pragma unroll
            for (int j = 0; j < TM; j++)
#pragma unroll
                for (int s = 0; s < NS; s++) acc[j][s][0] = acc[j][s][1] = acc[j][s][2] = acc[j][s][3] = 0.f;

            if constexpr (INT) {
                // (the tiles are a compile-time number for all of the chunk: addresses are then offsets of the loads)
                auto stages = [&](auto N) {
                    constexpr int NT = decltype(N)::value;
                    for (uint32_t us = 0; us == 0 || us < un; us += SU) {
                        const uint32_t off = (u0 + us) / 4 * (uint32_t)K::B256;
                        const uint32_t wl = ALN ? 0u : ((uint32_t)(uintptr_t)P.w + off) & 15u;
                        const uint32_t rb15 = P.row_bytes & 15u;
                        auto lead = [&](uint32_t row) { return ALN ? (T == GT_Q6_K ? off & 15u : 0u) : (wl + place(row & 15u) * rb15) & 15u; };
                        const uint32_t stage = base + slot * STAGE + (TABLE ? (warp >> 2) * (uint32_t)K::B256 : warp * UB);
                        const uint32_t xa = xlane + (us + warp) * 256u;
                        [[maybe_unused]] const uint32_t ca = clane + (us + warp) * (NG * 4u);
                        if ((us != 0 || i == 0) && !mbar_wait(&full[slot], ph, &abort_flag, bt.status, ST_WAIT_FULL_TIMEOUT, 0u)) {
                            ok = false;
                            break;
                        }
                        static_for<0, SU / kSpWarps>([&](auto I) {
                            constexpr uint32_t i = decltype(I)::value, OFF = i * (kSpWarps / 4) * K::B256;
                            const uint32_t uu = us + warp + kSpWarps * i;
                            if (uu >= un) return;
                            uint32_t b[NS][4];
                            float cc[NS];
#pragma unroll
                            for (int s = 0; s < NS; s++) {
                                lds128i<i * kSpWarps * 256u>(xa + s * xs, b[s]);
                                constexpr int own = T == GT_Q6_K ? 5 : 3;   // words of the first group (Q6_K: the even groups)
#pragma unroll
                                for (int q = 0; q < 4; q++) b[s][q] = ((g & 4u) != 0) != ((own >> q & 1) != 0) ? b[s][q] : 0u;
                                cc[s] = 0.f;
                                if constexpr (NG != 0)
                                    if (t & 1u) cc[s] = __uint_as_float(lds32i<i * kSpWarps * NG * 4u>(ca + s * cs));
                            }
                            if constexpr (TABLE) {
                                __syncwarp();   // the table of the unit before has been read
#pragma unroll
                                for (int rr = 0; rr < (NT + 1) / 2; rr++) {
                                    const uint32_t r = lane + 32u * rr;
                                    if (r < 16u * NT) sp_table_row<T, true>(tab + r * 16, stage + OFF + r * PITCH + lead(r), warp);
                                }
                                __syncwarp();
                            }
                            // (an odd number of blocks: the second block of the last unit lies past the row)
                            const bool half = !ALN && t >= 2 && (u0 + uu) * 64 + 32 >= P.k;
                            sp_unit_int<T, ALN, OFF, NT>(stage + g * PITCH + lead(g), stage + (g + 8) * PITCH + lead(g + 8), warp, t,
                                                         tab + g * 16 + (t >> 1) * 8, half, !ALN && bt.pairs, b, cc, bias, acc);
                        });
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&empty[slot]);
                        if (++slot == bt.nslots) {
                            slot = 0;
                            ph ^= 1u;
                        }
                    }
                };
                if (c.nt == 1) stages(std::integral_constant<int, 1>{});
                else if (c.nt == 2) stages(std::integral_constant<int, 2>{});
                else if (c.nt == 3) stages(std::integral_constant<int, 3>{});
                else stages(std::integral_constant<int, TM>{});
            } else {
                for (uint32_t us = 0; us < un; us += SU) {
                    const uint32_t off = (u0 + us) / 4 * (uint32_t)K::B256;
                    // where a row's data starts in its 16-byte superset (tiles are 16 rows: the same for every tile)
                    const uint32_t wl = ALN ? 0u : ((uint32_t)(uintptr_t)P.w + (ex < bt.n_experts ? ex : 0u) * (uint32_t)P.expert_stride + off) & 15u;
                    const uint32_t rb15 = P.row_bytes & 15u;
                    auto lead = [&](uint32_t row) { return ALN ? (T == GT_Q6_K ? off & 15u : 0u) : (wl + place(row & 15u) * rb15) & 15u; };
                    if (!mbar_wait(&full[slot], ph, &abort_flag, bt.status, ST_WAIT_FULL_TIMEOUT, 0u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t stage = base + slot * STAGE;
                    const uint32_t r0 = stage + g * PITCH + lead(g), r1 = stage + (g + 8) * PITCH + lead(g + 8);
#pragma unroll
                    for (int i = 0; i < SU / kSpWarps; i++) {
                        const uint32_t ul = warp + 8u * i, uu = us + ul;
                        if (uu >= un) break;
                        uint32_t bf[NS][4][2];
                        float cc[NS][2];
#pragma unroll
                        for (int s = 0; s < NS; s++) {
                            uint32_t v[4];
                            const uint32_t xa = xlane + uu * 256u + s * 4u * xs;
                            [[maybe_unused]] const uint32_t ca = clane + uu * NG * 4u + s * 4u * cs;
                            lds128i<0>(xa, v);
                            bf[s][0][0] = v[0]; bf[s][0][1] = v[1]; bf[s][1][0] = v[2]; bf[s][1][1] = v[3];
                            lds128i<128>(xa, v);
                            bf[s][2][0] = v[0]; bf[s][2][1] = v[1]; bf[s][3][0] = v[2]; bf[s][3][1] = v[3];
#pragma unroll
                            for (int q = 0; q < NG; q++) cc[s][q] = __uint_as_float(lds32(ca + q * 4u));
                        }
                        const uint32_t ub = TABLE ? (ul >> 2) * (uint32_t)K::B256 : ul * UB;
                        if constexpr (TABLE) {
                            __syncwarp();   // the table of the unit before has been read
#pragma unroll
                            for (int rr = 0; rr < TM / 2; rr++) {
                                const uint32_t r = lane + 32u * rr;
                                if (r < 16u * c.nt) sp_table_row<T, false>(tab + r * 16, stage + r * PITCH + lead(r) + ub, ul);
                            }
                            __syncwarp();
                        }
                        // (an odd number of blocks: the second block of the last unit lies past the row)
                        const bool half = (u0 + uu) * 64 + 32 >= P.k;
                        auto tiles = [&](auto NT) { sp_unit<T, ALN, decltype(NT)::value, false>(r0 + ub, r1 + ub, ul, t, g, tab, half, bf, cc, {1.f, 1.f}, acc); };
                        if (c.nt == 1) tiles(std::integral_constant<int, 1>{});
                        else if (TM == 2 || c.nt == 2) tiles(std::integral_constant<int, 2>{});
                        else if (c.nt == 3) tiles(std::integral_constant<int, TM == 2 ? 2 : 3>{});
                        else tiles(std::integral_constant<int, TM>{});
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[slot]);
                    if (++slot == bt.nslots) {
                        slot = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok) break;

            // ---- the warps' partial sums go to shared memory; they are added one chunk later, and what the other ranks send is
            // waited for two chunks later, so that nobody stands still for the slowest warp or for the way between SMs ----
            // (finish comes before this warp's arrivals for chunk i: four receive buffers rest on that, see there)
            if (i >= 2 && ranks > 1 && !finish(i - 2, d2)) break;
            // Chunk i - 2 has been read out of the area.  (Integers: four areas.  Who comes here has found every warp's arrival for chunk i - 2, and
            // a warp arrives there after it has read chunk i - 4.)
            if (!INT && i >= 2 && !wait(sync_bar[2], i & 1u, ST_WAIT_EMPTY_TIMEOUT)) break;
            const uint32_t part = red + (INT ? i & 3u : i & 1u) * (kSpWarps * RS * 4u);
            if constexpr (INT) {
                // A result is the sum of its row's columns over the four lanes: digits 0 and 1 or 2 and 3 of the first or second groups.  The
                // lanes exchange halves of what they have, so that each ends up with the sums of one tile (or of half a tile).
                const bool odd = t & 1u, up = t & 2u;
                const float w0 = odd ? sp::kDigitWeight : 1.f, w1 = 256.f * w0;
                auto swap = [](float keep, float give, int o) { return keep + __shfl_xor_sync(0xffffffffu, give, o); };
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    const float i0 = s_inv[warp][2 * s], i1 = s_inv[warp][2 * s + 1];
                    const uint32_t a = part + (warp * RS + s * R + g) * 4;
                    float v[TM][2];
#pragma unroll
                    for (int j = 0; j < TM; j++)
#pragma unroll
                        for (int h = 0; h < 2; h++) v[j][h] = fmaf(acc[j][s][2 * h + 1], w1, acc[j][s][2 * h] * w0);
                    if (TM > 2 && c.nt > 2) {
                        float k[2][2];
#pragma unroll
                        for (int j = 0; j < 2; j++)
#pragma unroll
                            for (int h = 0; h < 2; h++) k[j][h] = swap(odd ? v[TM - 2 + j][h] : v[j][h], odd ? v[j][h] : v[TM - 2 + j][h], 1);
                        const float r0 = swap(up ? k[1][0] : k[0][0], up ? k[0][0] : k[1][0], 2), r1 = swap(up ? k[1][1] : k[0][1], up ? k[0][1] : k[1][1], 2);
                        const uint32_t j = 2 * (t & 1u) + (t >> 1);
                        if (j < c.nt) {
                            sts32(a + 64 * j, __float_as_uint(r0 * i0 * i1));
                            sts32(a + 64 * j + 32, __float_as_uint(r1 * i0 * i1));
                        }
                    } else if (c.nt == 2) {
                        float k[2];
#pragma unroll
                        for (int h = 0; h < 2; h++) k[h] = swap(odd ? v[1][h] : v[0][h], odd ? v[0][h] : v[1][h], 1);
                        const float r = swap(up ? k[1] : k[0], up ? k[0] : k[1], 2);
                        sts32(a + 64 * (t & 1u) + 32 * (t >> 1), __float_as_uint(r * i0 * i1));
                    } else {
                        float r = swap(odd ? v[0][1] : v[0][0], odd ? v[0][0] : v[0][1], 1);
                        r += __shfl_xor_sync(0xffffffffu, r, 2);
                        if (t < 2) sts32(a + 32 * t, __float_as_uint(r * i0 * i1));
                    }
                }
            } else {
#pragma unroll
            for (int j = 0; j < TM; j++)
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    const uint32_t col = t + 4 * s;
                    if (col < mp && j < (int)c.nt) {
                        const float inv = s_inv[warp][col];
                        const uint32_t a = part + (warp * RS + col * R + 16 * j + g) * 4;
                        sts32(a, __float_as_uint((acc[j][s][0] + acc[j][s][1]) * inv));
                        sts32(a + 32, __float_as_uint((acc[j][s][2] + acc[j][s][3]) * inv));
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sync_bar[i & 1u]);
            if (i >= 1 && !add(i - 1, d1)) break;
            d2 = d1;
            d1 = i & 15u;
        }
        // The chunks from a share on that digits do not do for, in halves.  (A loop of its own: in the other one it cost one row of Q4_K 1.4 us of 20 and two
        // rows 2 us of 21.)
        if constexpr (INT)
            if (ok && at < last) {
                cur = 0xFFFFFFFFu;
                SpRing ring{full, empty, &abort_flag, base, slot, ph};
                for (; ok && at < last; i++) {
                    if (!wait(full[ring.slot], ring.ph, ST_WAIT_FULL_TIMEOUT)) break;
                    __syncwarp();
                    const SpChunk c = s_chunk[i & 15u];
                    const SpOp &P = bt.op[c.op];
                    const uint32_t u0 = rank * P.slice, k0 = 64u * u0;
                    at += c.steps;
                    if (c.key != cur) {
                        cur = c.key;
                        const size_t o = (size_t)c.e0 * P.k + k0;
                        sp_far<T, ALN, MPC>(P.x + o, P.k, P.k > k0 ? P.k - k0 : 0u, c.cnt, c.un, warp, lane, xf, xs, ccb, cs, s_inv[warp], s_rel);
                    }
                    ok = sp_far_stages<T, ALN, MPC>(bt, c.op, u0, c.un, c.nt, ring, warp, lane, xf, ccb, tab, red + ((i & 3u) * kSpWarps + warp) * RS * 4u, s_inv[warp], s_rel) && ok;
                    if (!ok) break;
                    if (i >= 2 && ranks > 1 && !finish(i - 2, d2)) break;   // (the order of the steps is that of the loop above)
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sync_bar[i & 1u]);
                    if (i >= 1 && !add(i - 1, d1)) break;
                    d2 = d1;
                    d1 = i & 15u;
                }
            }
        if (ok && i >= 1) ok = add(i - 1, d1);
        if (ok && ranks > 1 && i >= 2) ok = finish(i - 2, d2);
        if (ok && ranks > 1 && i >= 1) ok = finish(i - 1, d1);
        // An infinite activation's products with codes and offset may cancel where the weight has a sign: results that are no numbers are formed again,
        // weight by weight, each by the threads that stored it (integers: by the four lanes that added it up).  (Not on the way: the call costs the loop registers.)
        if constexpr (NG != 0) {
            __syncwarp();
            if (__any_sync(0xffffffffu, ok && s_again)) {
                const uint32_t rows = ranks == 1 ? R : share, parts = INT && ranks == 1 ? 4u : 1u;
                for (uint32_t at = first; at < last;) {
                    const SpChunk c = chunk(at);
                    at += c.steps;
                    for (uint32_t q = tid / parts; q < mp * rows; q += 256 / parts) again(c, q / rows, (ranks == 1 ? 0u : rank * share) + q % rows, parts);
                }
            }
        }
    }
    if (abort_flag)   // let copies in flight land before the CTA's shared memory is released
        for (int i = 0; i < 200; i++) __nanosleep(5000);
    __syncwarp();
    // nobody leaves while a peer may still send here
    if (ranks > 1) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
struct SpShape {          // geometry of a launch
    uint32_t ranks, tr, nslots, grid;
    size_t smem;
};

template <int T> inline size_t sp_tail(uint32_t ranks, uint32_t tr, uint32_t mp, uint32_t xunits, SpBatch *b) {
    const size_t r = 16u * tr;
    const size_t xf = (size_t)xunits * mp * 256, cc = SpTraits<T>::NG ? (((size_t)xunits * SpTraits<T>::NG * 4 + 16) * mp + 127) / 128 * 128 : 0;
    const size_t tab = SpTraits<T>::B256 == 272 || T == GT_Q4_0 ? 0 : (size_t)kSpWarps * r * 16;
    const size_t red = (size_t)(mp <= 2 ? 4 * kSpWarps * (mp * r + 8) : 2 * kSpWarps * mp * r) * 4, recv = ranks > 1 ? (size_t)4 * mp * r * 4 : 0;
    if (b) {
        b->cc_off = b->xf_off + (uint32_t)xf;
        b->tab_off = b->cc_off + (uint32_t)cc;
        b->red_off = b->tab_off + (uint32_t)tab;
        b->recv_off = b->red_off + (uint32_t)red;
        b->xstride = xunits * 256;
        b->cstride = xunits * SpTraits<T>::NG * 4 + 16;   // (+ 16: four rows in distinct banks)
    }
    return xf + cc + tab + red + recv;
}

template <int T, bool ALN, int MPC, bool INT>
static cudaError_t sp_launch(SpBatch &bt, const SpMaps &maps, uint32_t ranks, uint32_t tr, uint64_t entries, uint32_t xunits, int sm_count, cudaStream_t st) {
    const uint32_t STAGE = tr * 16 * sp_pitch<T>(ALN);
    bt.tr = tr;
    bt.step = bt.ids || bt.mp > 2 ? tr : 1u;   // (see SpChunk)
    bt.dealt = bt.step != 1 && entries == 1;
    uint32_t per = 0;   // steps of an entry
    for (uint32_t i = 0; i < bt.nops; i++) bt.op[i].step_end = per += ((bt.op[i].n + 15) / 16 + bt.step - 1) / bt.step;
    const uint64_t steps = per * entries;
    const size_t tail = sp_tail<T>(ranks, tr, bt.mp, xunits, nullptr);
    uint32_t nslots = (uint32_t)((kSpSmem - 128 - tail) / STAGE);
    if (nslots > (uint32_t)kSpMaxSlots) nslots = kSpMaxSlots;
    if (tail + STAGE + 128 > kSpSmem || nslots < 1) return cudaErrorInvalidConfiguration;
    bt.nslots = nslots;
    bt.xf_off = nslots * STAGE;
    sp_tail<T>(ranks, tr, bt.mp, xunits, &bt);
    const size_t smem = (size_t)nslots * STAGE + tail + 128;
    auto kernel = qmv_split_kernel<T, ALN, MPC, INT>;
    static std::atomic<uint32_t> prepared[64] = {};   // per device: the attribute has been set
    static std::atomic<uint32_t> fit[64][4] = {};     // ... and the clusters of 2, 4 and 8 CTAs that are resident together
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpSmem);
        if (e != cudaSuccess) return e;
        prepared[dev].store(1, std::memory_order_release);
    }
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ranks;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kSpThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    // clusters that are resident at the same time (a cluster lives in one GPC, so not every SM may be covered)
    uint32_t ncl = (uint32_t)(2 * sm_count) / ranks;
    if (ranks > 1) {
        const int l = ranks == 2 ? 1 : ranks == 4 ? 2 : 3;
        uint32_t f = fit[dev][l].load(std::memory_order_relaxed);
        if (!f) {
            int n = 0;
            cfg.gridDim = dim3(ncl * ranks);
            cfg.dynamicSmemBytes = kSpSmem;   // (the largest the kernel is launched with)
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                (void)cudaGetLastError();
                n = (int)ncl;
            }
            cfg.dynamicSmemBytes = smem;
            f = (uint32_t)n;
            fit[dev][l].store(f, std::memory_order_relaxed);
        }
        ncl = f < ncl ? f : ncl;
    }
    if (steps < ncl) ncl = (uint32_t)steps;
    // Clusters of four and eight: no more than the longest share needs.  They have to find their places in one GPC while the kernel ahead still has CTAs there; where every place is
    // wanted and the first come lie badly, the last cluster waits for another's end.  (Behind silu_mul 4096 x 14336 Q6_K took 25.5 us on 71 clusters, 17.6 on the 64 that
    // are as fast alone; a decode layer of 4096 / 14336 in Q4_K and Q6_K 66 us, 61.)
    if (ranks > 2 && bt.step == 1) {
        const uint64_t longest = (steps + ncl - 1) / ncl;
        ncl = (uint32_t)((steps + longest - 1) / longest);
    }
    cfg.gridDim = dim3(ncl * ranks);
    return cudaLaunchKernelEx(&cfg, kernel, bt, maps);
}

// Chooses the cluster size and the tiles of a chunk; ranks == 0: no geometry fits.  qmv_split_supported asks the same function, so that
// no call is promised this kernel and then refused.
struct SpPick {
    uint32_t ranks, tr;
};
template <int T> inline SpPick sp_pick(bool aln, uint32_t mp, bool packed, bool routed, uint64_t tiles, uint32_t max_units, int sm_count) {
    SpPick pick{0, 0};
    double best = 1e30;
    int force_c = 0, force_tr = 0;
    if (const char *e = exp_env("MLXN_SP_C")) force_c = atoi(e);
    if (const char *e = exp_env("MLXN_SP_TR")) force_tr = atoi(e);
    for (uint32_t c = 1; c <= (routed ? 1u : 8u); c *= 2) {
        const uint32_t slice = ((max_units + c - 1) / c + 3) / 4 * 4;
        // a rank without work: only where nothing smaller fits (K = 10304 with eight rows: seven slices of 24 units do, four of 44 do not)
        if (c > 1 && slice * (c - 1) >= max_units && pick.ranks) continue;
        // (there are fewer clusters than CTAs would do for: 71 of four and 33 of eight on 148 SMs; whole numbers, since this runs for every product that is encoded)
        const uint32_t places = 2u * (uint32_t)sm_count / c, fit = c == 4 ? places * 24 / 25 : c == 8 ? places * 9 / 10 : places, ncl = fit ? fit : 1, units = (slice + 7) / 8;
        const uint32_t share = (uint32_t)((tiles + ncl - 1) / ncl), whole = (uint32_t)tiles;   // (below 2^31 for a product: qmv_split_fits)
        for (uint32_t tr = 1; tr <= (uint32_t)sp_tiles((int)mp); tr++) {
            if ((force_c && !routed && (int)c != force_c) || (force_tr && (int)tr != force_tr)) continue;
            const size_t stage = (size_t)tr * 16 * sp_pitch<T>(aln), tail = sp_tail<T>(c, tr, mp, (slice + 1) & ~1u, nullptr);
            if (tail + 2 * stage + 128 > kSpSmem) continue;
            double cost;
            if (mp <= 2 && !routed) {   // in integers
                // Every CTA splits the activations; a chunk costs waits and sums, a unit of a warp a share per tile; ranks wait for one another.  Fitted to 192 products (four types,
                // one and two rows, 1024 to 49152 rows of 1024 to 12288 values) timed at every geometry: what is taken is within 5 percent of the fastest for 177 of
                // them, 1.2 percent slower on average, 17 at most (Q8_0, two rows, three of 4096 x 4096; profiles/qmv_split_geometry.md).
                const double chunks = (share + tr - 1) / tr, tile = (T == GT_Q4_0 ? 0.2 : T == GT_Q8_0 ? 0.28 : T == GT_Q6_K ? 0.29 : 0.32) * (mp == 2 ? 1.3 : 1.0);
                cost = units * (mp == 2 ? 0.71 : 0.31) + chunks * (1.3 + 0.03 * units) + (double)units * share * tile + (c == 1 ? 0.0 : (c == 2 ? 1.2 : c == 4 ? 2.7 : 3.5) + 0.05 * chunks);
            } else if (mp <= 4 && !routed) {   // the same for whole chunks, fitted to 92 products of four rows: 1 percent slower on average, 12 at most
                const size_t slots = (kSpSmem - 128 - tail) / stage;
                const double chunks = ((whole + tr - 1) / tr + ncl - 1) / ncl, tile = T == GT_Q4_0 ? 0.1 : T == GT_Q8_0 ? 0.28 : T == GT_Q6_K ? 0.29 : 0.22;
                cost = chunks * (1.05 + 0.41 * units + tr * units * tile + (slots == 2 ? 0.18 : slots == 3 ? 0.07 : 0.0)) + (c == 1 ? 0.0 : (c == 2 ? 0.66 : c == 4 ? 1.4 : 1.7) + 0.86 * chunks);
            } else {
                // Fitted to 12288 x 4096 and 4096 x 4096, all types: a chunk costs waits and sums, with eight rows and four ranks 4.5 us.
                const double chunks = ((whole + tr - 1) / tr + places - 1) / (places ? places : 1), tile = (T == GT_Q6_K ? 0.3 : 0.23) * (mp > 4 ? 1.5 : 1.0);
                cost = (packed ? 1.0 : 0.3 + 0.27 * units) + chunks * ((mp > 4 && c == 4 ? 4.5 : 1.9) + tr * tile * units) + (c > 1 ? 0.3 : 0.0) +
                       ((kSpSmem - 128 - tail) / stage < 3 ? 0.3 : 0.0);
            }
            if (cost < best) {
                best = cost;
                pick = {c, tr};
            }
        }
    }
    return pick;
}

template <int T, bool ALN, int MPC, bool INT>
static cudaError_t sp_choose(SpBatch &bt, const SpMaps &maps, uint64_t tiles, uint64_t entries, uint32_t max_units, bool routed, int sm_count, cudaStream_t st) {
    const SpPick pick = sp_pick<T>(ALN, bt.mp, bt.packed != 0, routed, tiles, max_units, sm_count);
    if (!pick.ranks) return cudaErrorInvalidConfiguration;
    for (uint32_t i = 0; i < bt.nops; i++) bt.op[i].slice = ((bt.op[i].units + pick.ranks - 1) / pick.ranks + 3) / 4 * 4;
    const uint32_t xunits = (((max_units + pick.ranks - 1) / pick.ranks + 3) / 4 * 4 + 1) & ~1u;
    return sp_launch<T, ALN, MPC, INT>(bt, maps, pick.ranks, pick.tr, entries, xunits, sm_count, st);
}

// Scratch bytes of a mat-vec's packed activations.
template <int T> inline size_t sp_pack_bytes(uint32_t m, uint32_t k) {
    return ((size_t)m * (((k + 63) / 64 + 3) & ~3u) * (256 + 4 * SpTraits<T>::NG) + (size_t)m * 4 + 255) / 256 * 256;
}

// Instantiated once per block type (qmv_split_*.cu).  `ops`: dense, or all routed over the same pairs.
template <int T> cudaError_t sp_run(const QmvArgs *ops, int nops, int sm_count, uint8_t *scratch, int *launches, cudaStream_t st) {
    if (nops < 1 || nops > kSpMaxOps) return cudaErrorInvalidValue;
    const bool routed = ops[0].ids != nullptr;
    if (T == GT_Q5_K && !routed) return cudaErrorNotSupported;
    bool aln = true, pairs = true;
    for (int i = 0; i < nops; i++) {
        const uint64_t rb = (uint64_t)(ops[i].k / BlockTraits<T>::QK) * BlockTraits<T>::BYTES;
        const bool base = ((uintptr_t)ops[i].w & 15u) == 0 && (!routed || ops[i].expert_stride % 16 == 0);
        aln = aln && rb % 16 == 0 && base;
        pairs = pairs && rb % 16 == 8 && base && ops[i].n % 2 == 0 && (routed || ops[i].m <= 4);
    }
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return cudaErrorNotSupported;
    static thread_local SpBatch bt;
    alignas(64) static thread_local SpMaps maps;
    bt.nops = (uint32_t)nops;
    bt.pairs = pairs;
    bt.ids = ops[0].ids;
    bt.npairs = routed ? ops[0].nprob : 0;
    bt.n_experts = routed ? ops[0].n_experts : 1;
    bt.status = ops[0].status;
    bt.early_weights = routed ? 0u : 1u;
    uint32_t rows = 1, tiles = 0, max_units = 0;
    for (int i = 0; i < nops; i++) {
        const QmvArgs &a = ops[i];
        SpOp &P = bt.op[i];
        P.w = a.w;
        P.x = a.x;
        P.x2 = a.x2;
        P.y = a.y;
        P.n = a.n;
        P.k = a.k;
        P.m = a.m;
        tiles += (a.n + 15) / 16;
        P.row_bytes = (a.k / BlockTraits<T>::QK) * BlockTraits<T>::BYTES;
        P.units = (a.k + 63) / 64;
        P.x_div = a.top_k ? a.top_k : 1;
        P.y_ld = qmv_ld(a);
        P.y_col0 = a.y_col0;
        P.n_peer = a.n_peer;
        for (int q = 0; q < kMaxPeers; q++) P.y_peer[q] = q < (int)a.n_peer ? a.y_peer[q] : nullptr;
        P.expert_stride = routed ? a.expert_stride : 0;
        P.xkey = (uint32_t)i;
        P.pk_units = (P.units + 3) & ~3u;
        P.xp_row = P.pk_units * 256u;
        P.xp_super = 1024;
        P.wide_rows = 0;
        for (int q = 0; q < i; q++)
            if (ops[q].x == a.x && ops[q].x2 == a.x2 && ops[q].m == a.m && ops[q].k == a.k && ops[q].top_k == a.top_k) {
                P.xkey = bt.op[q].xkey;
                P.xp = bt.op[q].xp;
                P.xsum = bt.op[q].xsum;
                P.xinv = bt.op[q].xinv;
                break;
            }
        if (!routed && P.xkey == (uint32_t)i) {
            const size_t u = (size_t)a.m * P.pk_units;
            P.xp = scratch;
            P.xsum = reinterpret_cast<float *>(scratch + u * 256);
            P.xinv = P.xsum + u * SpTraits<T>::NG;
            scratch += sp_pack_bytes<T>(a.m, a.k);
        }
        if (!a.early_weights) bt.early_weights = 0;
        rows = a.m > rows ? a.m : rows;
        max_units = P.units > max_units ? P.units : max_units;
        if (aln || pairs) {
            const uint64_t rb = (uint64_t)P.row_bytes * (pairs ? 2 : 1);
            const cuuint64_t dim[3] = {rb / 8, pairs ? a.n / 2 : a.n, routed ? a.n_experts : 1}, stride[2] = {rb, routed ? a.expert_stride : (uint64_t)P.row_bytes * a.n};
            const cuuint32_t box[3] = {sp_pitch<T>(aln) / 8, pairs ? 8u : 16u, 1}, one[3] = {1, 1, 1};
            if (enc(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<uint8_t *>(a.w), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return cudaErrorInvalidValue;
        }
    }
    // rows of an entry: dense, as many as fit two sets of columns; routed, one set (most experts have few rows)
    bt.mp = routed ? ((ops[0].nprob <= 1 ? 1u : 4u)) : rows <= 1 ? 1u : rows <= 2 ? 2u : rows <= 4 ? 4u : 8u;
    bt.nent = routed ? 0u : (rows + bt.mp - 1) / bt.mp;
    const uint64_t entries = routed ? ops[0].nprob : bt.nent, all = tiles * entries;
    bt.packed = !routed && bt.mp > 2;
    *launches = 1;
    auto go = [&](auto ALN) {
        constexpr bool A = decltype(ALN)::value;
        if constexpr (T != GT_Q5_K) {   // (expert-routed only: never packed, one set of columns)
            if (bt.packed) {
                uint32_t end = 0;
                for (int i = 0; i < nops; i++) bt.op[i].row_end = end += bt.op[i].xkey == (uint32_t)i ? bt.op[i].m : 0u;
                const cudaError_t e = launch_overlapped(qmv_pack_kernel<T, A>, dim3(end), dim3(256), 0, st, bt);
                if (e != cudaSuccess) return e;
                ++*launches;
            }
            if (bt.mp > 4) return sp_choose<T, A, 8, false>(bt, maps, all, entries, max_units, routed, sm_count, st);
        }
        // (Routed rows are always summed in f16: one form has to serve a call whatever its pairs, so that a pair's sum does not depend on those that travel with
        // it, and rows that share an expert gain more from one pass over its codes than from integers, where every row is a multiply of its own.  Q4_0,
        // 768 x 2048, 256 pairs of 16 experts 35.6 us, with two rows a pass in integers 47.6; 8 pairs of 128 experts 11.0, in integers 8.7.  A row's sum in integers
        // would be the same bits with one set of columns or several, so a choice by the number of experts could take them.)
        if constexpr (T != GT_Q5_K) {
            if (!routed && bt.mp == 2) return sp_choose<T, A, 2, true>(bt, maps, all, entries, max_units, false, sm_count, st);
            if (!routed && bt.mp == 1) return sp_choose<T, A, 1, true>(bt, maps, all, entries, max_units, false, sm_count, st);
        }
        if (bt.mp == 1) return sp_choose<T, A, 1, false>(bt, maps, all, entries, max_units, routed, sm_count, st);
        return sp_choose<T, A, 4, false>(bt, maps, all, entries, max_units, routed, sm_count, st);
    };
    if (aln) return go(std::true_type{});
    if constexpr (T == GT_Q4_K || T == GT_Q5_K) return cudaErrorNotSupported;   // (144- and 176-byte blocks: only a misaligned base)
    else return go(std::false_type{});
}

}  // namespace mlxn
