// Raw GGML blocks in shared memory to f16: the exact value of a weight, rounded once.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace mlxn {

__device__ __forceinline__ uint32_t lds32s(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16s(uint32_t addr) {
    uint32_t v;
    asm volatile("{ .reg .u16 t; ld.shared.u16 t, [%1]; cvt.u32.u16 %0, t; }" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ int lds_s8s(uint32_t addr) {
    int v;
    asm volatile("{ .reg .s16 t; ld.shared.s8 t, [%1]; cvt.s32.s16 %0, t; }" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }

// NWORDS logical 32-bit words at a 2-byte-aligned shared address
template <int NWORDS> __device__ __forceinline__ void lds_words_n(uint32_t addr, uint32_t (&out)[NWORDS]) {
    const uint32_t al = addr & ~3u, sh = (addr & 2u) * 8u;
    uint32_t prev = lds32s(al);
#pragma unroll
    for (int j = 0; j < NWORDS; j++) {
        const uint32_t nxt = lds32s(al + 4 * (j + 1));
        out[j] = __funnelshift_rc(prev, nxt, sh);
        prev = nxt;
    }
}
// four bytes (each < 128 after the caller's masking) -> two half2 of (1024 + byte)
__device__ __forceinline__ void bytes_to_h2(uint32_t w, __half2 &lo, __half2 &hi) {
    lo = u32_as_h2(__byte_perm(w, 0x64646464u, 0x4140));
    hi = u32_as_h2(__byte_perm(w, 0x64646464u, 0x4342));
}

// Thirty-two consecutive elements [e, e+32) (e a multiple of 32) of one weight row segment in shared
// memory -> four 16-byte groups of eight f16 values, each the exact product rounded once (RNE).
template <int T> __device__ __forceinline__ void dequant32(uint32_t seg, uint32_t e, uint4 (&out)[4]) {
    if constexpr (T == GT_Q4_0) {
        const uint32_t o = seg + 18u * (e >> 5);
        const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)lds16s(o)));
        const __half2 off = __float2half2_rn(1032.0f);  // 1024 + 8
        uint32_t q[4];
        lds_words_n<4>(o + 2, q);
#pragma unroll
        for (int j = 0; j < 4; j++) {  // j = 0,1: low nibbles of bytes 0-7, 8-15; j = 2,3: high nibbles
            const uint32_t w0 = ((j & 2) ? (q[2 * (j & 1)] >> 4) : q[2 * (j & 1)]) & 0x0F0F0F0Fu;
            const uint32_t w1 = ((j & 2) ? (q[2 * (j & 1) + 1] >> 4) : q[2 * (j & 1) + 1]) & 0x0F0F0F0Fu;
            __half2 a, b, cc, dd;
            bytes_to_h2(w0, a, b);
            bytes_to_h2(w1, cc, dd);
            out[j].x = h2_as_u32(__hmul2(__hsub2(a, off), d2));
            out[j].y = h2_as_u32(__hmul2(__hsub2(b, off), d2));
            out[j].z = h2_as_u32(__hmul2(__hsub2(cc, off), d2));
            out[j].w = h2_as_u32(__hmul2(__hsub2(dd, off), d2));
        }
    } else if constexpr (T == GT_Q8_0) {
        const uint32_t o = seg + 34u * (e >> 5);
        const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)lds16s(o)));
        const __half2 off = __float2half2_rn(1152.0f);  // 1024 + 128
        uint32_t q[8];
        lds_words_n<8>(o + 2, q);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            __half2 a, b, cc, dd;
            bytes_to_h2(q[2 * j] ^ 0x80808080u, a, b);
            bytes_to_h2(q[2 * j + 1] ^ 0x80808080u, cc, dd);
            out[j].x = h2_as_u32(__hmul2(__hsub2(a, off), d2));
            out[j].y = h2_as_u32(__hmul2(__hsub2(b, off), d2));
            out[j].z = h2_as_u32(__hmul2(__hsub2(cc, off), d2));
            out[j].w = h2_as_u32(__hmul2(__hsub2(dd, off), d2));
        }
    } else if constexpr (T == GT_Q4_K) {
        // sub-block j of the 144-byte super-block: 32 nibbles of the bytes 16 + 32 (j / 2) ..., low for even j;
        // value = (d sc) q - (dmin m) (src/gguf/mod.rs:582-644), formed in f32 and rounded to f16 once
        const uint32_t o = seg + 144u * (e >> 8);
        const uint32_t j = (e & 255u) >> 5;
        const uint32_t dd = lds16s(o) | (lds16s(o + 2) << 16);
        uint32_t sw[3];
        lds_words_n<3>(o + 4, sw);                      // scales[0..11]
        uint32_t sc, mn;
        if (j < 4) {
            sc = (sw[0] >> (8 * j)) & 63u;
            mn = (sw[1] >> (8 * j)) & 63u;
        } else {
            const uint32_t sh = 8 * (j - 4);
            sc = ((sw[2] >> sh) & 15u) | ((((sw[0] >> sh) >> 6) & 3u) << 4);
            mn = (((sw[2] >> sh) >> 4) & 15u) | ((((sw[1] >> sh) >> 6) & 3u) << 4);
        }
        const float ds = half_bits_to_float(dd & 0xFFFFu) * (float)sc;
        const float dm = half_bits_to_float(dd >> 16) * (float)mn;
        const float c = fmaf(-128.0f, ds, -dm);
        uint32_t Q[8];
        lds_words_n<8>(o + 16 + 32 * (j >> 1), Q);
        const uint32_t ash = (j & 1u) ? 4u : 0u;
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
            uint32_t res[4];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t u = (Q[2 * jj + i] >> ash) & 0x0F0F0F0Fu;
                // 128 + u spliced into an f32 mantissa; fma(128 + u, ds, -128 ds - dm) = ds u - dm
                const float f0 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7044)), ds, c);
                const float f1 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7144)), ds, c);
                const float f2 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7244)), ds, c);
                const float f3 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7344)), ds, c);
                res[2 * i] = h2_as_u32(__floats2half2_rn(f0, f1));
                res[2 * i + 1] = h2_as_u32(__floats2half2_rn(f2, f3));
            }
            out[jj] = make_uint4(res[0], res[1], res[2], res[3]);
        }
    } else {
        const uint32_t o = seg + 210u * (e >> 8);
        const uint32_t r = e & 255u, h = r >> 7, g = (r & 127u) >> 5;
        uint32_t A[8], H[8];
        lds_words_n<8>(o + 64 * h + 32 * (g & 1u), A);
        lds_words_n<8>(o + 128 + 32 * h, H);
        const float d = half_bits_to_float(lds16s(o + 208));
        const float ds0 = d * (float)lds_s8s(o + 192 + 8 * h + 2 * g);
        const float ds1 = d * (float)lds_s8s(o + 192 + 8 * h + 2 * g + 1);
        const uint32_t hsh = 2 * g, ash = (g & 2u) ? 4u : 0u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float ds = j < 2 ? ds0 : ds1;
            const float c = -160.0f * ds;  // exact: ds has <= 18 significant bits
            uint32_t res[4];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t u = ((A[2 * j + i] >> ash) & 0x0F0F0F0Fu) | (((H[2 * j + i] >> hsh) & 0x03030303u) << 4);
                // 128 + u spliced into an f32 mantissa; fma(128+u, ds, -160 ds) = ds*(u-32) exactly
                const float f0 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7044)), ds, c);
                const float f1 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7144)), ds, c);
                const float f2 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7244)), ds, c);
                const float f3 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7344)), ds, c);
                res[2 * i] = h2_as_u32(__floats2half2_rn(f0, f1));
                res[2 * i + 1] = h2_as_u32(__floats2half2_rn(f2, f3));
            }
            out[j] = make_uint4(res[0], res[1], res[2], res[3]);
        }
    }
}

// ---- rows that start on 16-byte boundaries: 16-byte shared loads at compile-time offsets ----------------------
// The generic routines above read the raw rows with 32-bit loads at 2-byte granular addresses; with rows an odd
// multiple of 16 bytes apart those are 4-way bank-conflicted (two thirds of the kernel's shared-memory wavefronts).
// When every weight row starts on a 16-byte boundary and the raw stage is a whole number of 16-byte units per row
// (k % 256 == 0), each thread's 64 elements sit at a compile-time byte offset of the row's stage, so they can
// be fetched with conflict-free 16-byte loads and static funnel shifts.
__device__ __forceinline__ void q4_0_block_to_h(uint32_t dbits, const uint32_t (&q)[4], uint32_t *out /*16 words*/) {
    const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)dbits));
    const __half2 off = __float2half2_rn(1032.0f);  // 1024 + 8
#pragma unroll
    for (int j = 0; j < 4; j++) {  // j = 0,1: low nibbles of bytes 0-7, 8-15; j = 2,3: high nibbles
        const uint32_t w0 = ((j & 2) ? (q[2 * (j & 1)] >> 4) : q[2 * (j & 1)]) & 0x0F0F0F0Fu;
        const uint32_t w1 = ((j & 2) ? (q[2 * (j & 1) + 1] >> 4) : q[2 * (j & 1) + 1]) & 0x0F0F0F0Fu;
        __half2 a, b, cc, dd;
        bytes_to_h2(w0, a, b);
        bytes_to_h2(w1, cc, dd);
        out[4 * j + 0] = h2_as_u32(__hmul2(__hsub2(a, off), d2));
        out[4 * j + 1] = h2_as_u32(__hmul2(__hsub2(b, off), d2));
        out[4 * j + 2] = h2_as_u32(__hmul2(__hsub2(cc, off), d2));
        out[4 * j + 3] = h2_as_u32(__hmul2(__hsub2(dd, off), d2));
    }
}
__device__ __forceinline__ void q8_0_block_to_h(uint32_t dbits, const uint32_t (&q)[8], uint32_t *out /*16 words*/) {
    const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)dbits));
    const __half2 off = __float2half2_rn(1152.0f);  // 1024 + 128
#pragma unroll
    for (int j = 0; j < 8; j++) {
        __half2 a, b;
        bytes_to_h2(q[j] ^ 0x80808080u, a, b);
        out[2 * j + 0] = h2_as_u32(__hmul2(__hsub2(a, off), d2));
        out[2 * j + 1] = h2_as_u32(__hmul2(__hsub2(b, off), d2));
    }
}
// Quarter S4 (64 elements = 2 blocks) of a row's 256-wide raw stage at the 16-byte aligned shared address `unit`.
template <int T, int S4> __device__ __forceinline__ void dequant64_aligned(uint32_t unit, uint32_t (&r)[32]) {
    constexpr int SUB = 2 * BlockTraits<T>::BYTES;   // bytes of two blocks
    constexpr int c0 = (SUB * S4) >> 4;              // first 16-byte chunk touched
    constexpr int wo = ((SUB * S4) & 15) >> 2;       // word offset inside it (SUB * S4 is a multiple of 4)
    if constexpr (T == GT_Q4_0) {
        uint32_t W[12];
#pragma unroll
        for (int i = 0; i < 3; i++) lds128(unit + 16 * (c0 + i), W[4 * i], W[4 * i + 1], W[4 * i + 2], W[4 * i + 3]);
        uint32_t q0[4], q1[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            q0[i] = __funnelshift_r(W[wo + i], W[wo + i + 1], 16);  // block 0's codes start 2 bytes into a word
            q1[i] = W[wo + 5 + i];                                  // block 1's are word aligned
        }
        q4_0_block_to_h(W[wo] & 0xFFFFu, q0, r);
        q4_0_block_to_h(W[wo + 4] >> 16, q1, r + 16);
    } else {
        uint32_t W[20];
#pragma unroll
        for (int i = 0; i < 5; i++) lds128(unit + 16 * (c0 + i), W[4 * i], W[4 * i + 1], W[4 * i + 2], W[4 * i + 3]);
        uint32_t q0[8], q1[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            q0[i] = __funnelshift_r(W[wo + i], W[wo + i + 1], 16);
            q1[i] = W[wo + 9 + i];
        }
        q8_0_block_to_h(W[wo] & 0xFFFFu, q0, r);
        q8_0_block_to_h(W[wo + 8] >> 16, q1, r + 16);
    }
}
// Q6_K: 64 elements (half h's runs 2 q and 2 q + 1) of the super-block that starts PRE bytes into the row's aligned stage.  The two runs
// have the same 32 bytes of high bits, and their 64 bytes of low bits follow one another.  A code is put beside 1024 in f16, widened, and scaled
// two at a time: fma(1024 + u, ds, -1056 ds) = ds (u - 32), exact in f32 (ds has at most 18 significant bits), then rounded once to f16.
// field(o, w): the 32 bytes at byte o of the super-block; rest: shared address of the super-block (its last 18 bytes are scales and d).
template <class F> __device__ __forceinline__ void dequant64_q6k(F &&field, uint32_t rest, uint32_t h, uint32_t q, uint32_t (&out)[32]) {
    uint32_t H[8];
    field(128 + 32 * h, H);
    const float d = half_bits_to_float(lds_u16(rest + 208));
    const uint32_t sc[2] = {lds_u16(rest + 192 + 8 * h + 4 * q), lds_u16(rest + 194 + 8 * h + 4 * q)};
    const uint32_t ash = 4 * q;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        uint32_t A[8];
        field(64 * h + 32 * g, A);
        const uint32_t rot = (4u - 4 * q - 2 * g) & 31u;   // brings a byte's two bits to bits 4 and 5
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float ds = d * (float)(int)(int8_t)(j < 4 ? sc[g] & 0xFFu : sc[g] >> 8);
            const float c = -1056.0f * ds;
            const uint32_t u = ((A[j] >> ash) & 0x0F0F0F0Fu) | (__funnelshift_l(H[j], H[j], rot) & 0x30303030u);
            __half2 lo, hi;
            bytes_to_h2(u, lo, hi);
            const uint64_t ds2 = pack2(ds, ds), c2 = pack2(c, c);
            float f0, f1, f2, f3;
            unpack2(ffma2(pack2(__low2float(lo), __high2float(lo)), ds2, c2), f0, f1);
            unpack2(ffma2(pack2(__low2float(hi), __high2float(hi)), ds2, c2), f2, f3);
            out[16 * g + 2 * j] = h2_as_u32(__floats2half2_rn(f0, f1));
            out[16 * g + 2 * j + 1] = h2_as_u32(__floats2half2_rn(f2, f3));
        }
    }
}
template <int PRE> __device__ __forceinline__ void dequant64_q6k_aligned(uint32_t stage_row, uint32_t h, uint32_t q, uint32_t (&out)[32]) {
    dequant64_q6k([&](uint32_t o, uint32_t (&w)[8]) { lds_field<PRE, 8>(stage_row + o, w); }, stage_row + PRE, h, q, out);
}
// The same for a super-block at any even address, which may differ from lane to lane: 8-byte loads, of which a select takes the words and a
// shift the halves.  (For rows that are neighbours in shared memory, an odd multiple of 16 bytes apart: there a load of 4 bytes a lane takes as many
// passes as one of 8.)
__device__ __forceinline__ void dequant64_q6k_any(uint32_t seg, uint32_t h, uint32_t q, uint32_t (&out)[32]) {
    const bool odd = (seg & 4u) != 0;
    const uint32_t sh = (seg & 2u) * 8u, base = seg & ~7u;
    dequant64_q6k([&](uint32_t o, uint32_t (&w)[8]) {   // (o is a multiple of 32)
        uint32_t W[10];
#pragma unroll
        for (int i = 0; i < 5; i++) lds64(base + o + 8 * i, W[2 * i], W[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < 9; i++) W[i] = odd ? W[i + 1] : W[i];
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = __funnelshift_r(W[i], W[i + 1], sh);
    }, seg, h, q, out);
}
__device__ __forceinline__ void dequant64_q6k_aligned_p(uint32_t p8, uint32_t stage_row, uint32_t h, uint32_t q, uint32_t (&out)[32]) {
    switch (p8) {  // uniform over the CTA
    case 0: dequant64_q6k_aligned<0>(stage_row, h, q, out); break;
    case 1: dequant64_q6k_aligned<2>(stage_row, h, q, out); break;
    case 2: dequant64_q6k_aligned<4>(stage_row, h, q, out); break;
    case 3: dequant64_q6k_aligned<6>(stage_row, h, q, out); break;
    case 4: dequant64_q6k_aligned<8>(stage_row, h, q, out); break;
    case 5: dequant64_q6k_aligned<10>(stage_row, h, q, out); break;
    case 6: dequant64_q6k_aligned<12>(stage_row, h, q, out); break;
    default: dequant64_q6k_aligned<14>(stage_row, h, q, out); break;
    }
}

// Q4_K: sub-block j (32 elements) of the super-block at a 16-byte boundary, as dequant32 forms it, by 16-byte loads.
__device__ __forceinline__ void dequant32_q4k_aligned(uint32_t o, uint32_t j, uint32_t *out /*16 words*/) {
    uint32_t dd, s0, s1, s2, Q[8];
    lds128(o, dd, s0, s1, s2);
    lds128(o + 16 + 32 * (j >> 1), Q[0], Q[1], Q[2], Q[3]);
    lds128(o + 32 + 32 * (j >> 1), Q[4], Q[5], Q[6], Q[7]);
    uint32_t sc, mn;
    if (j < 4) {
        sc = (s0 >> (8 * j)) & 63u;
        mn = (s1 >> (8 * j)) & 63u;
    } else {
        const uint32_t sh = 8 * (j - 4);
        sc = ((s2 >> sh) & 15u) | ((((s0 >> sh) >> 6) & 3u) << 4);
        mn = (((s2 >> sh) >> 4) & 15u) | ((((s1 >> sh) >> 6) & 3u) << 4);
    }
    const float ds = half_bits_to_float(dd & 0xFFFFu) * (float)sc, dm = half_bits_to_float(dd >> 16) * (float)mn;
    const float c = fmaf(-128.0f, ds, -dm);
    const uint32_t ash = (j & 1u) ? 4u : 0u;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t u = (Q[i] >> ash) & 0x0F0F0F0Fu;
        const float f0 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7044)), ds, c);
        const float f1 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7144)), ds, c);
        const float f2 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7244)), ds, c);
        const float f3 = fmaf(__uint_as_float(__byte_perm(u, 0x43000000u, 0x7344)), ds, c);
        out[2 * i] = h2_as_u32(__floats2half2_rn(f0, f1));
        out[2 * i + 1] = h2_as_u32(__floats2half2_rn(f2, f3));
    }
}

}  // namespace mlxn
