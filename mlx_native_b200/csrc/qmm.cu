// Mat-mat kernels for GGML Q4_0 / Q8_0 / Q6_K weights (prefill path, m > 8), dense and grouped by expert.
//
// Replaces upstream kernel_mul_mm_*_tensor_f32 (src/shaders/quantized_matmul_mm_tensor.metal:170-343),
// kernel_mul_mm_id_*_tensor_f32 (src/shaders/quantized_matmul_id_mm_tensor.metal:165-341) and the
// simdgroup variants beside them.  Operand semantics are those of the upstream tensor path: weights
// are dequantised in f32 and rounded once to f16, activations are rounded f32 -> f16, products are
// accumulated in f32.
//
//   qmm_tc    tcgen05 kernel.  Per CTA one output tile of 128 weight rows x NT activation rows.
//             Activations are packed once per call into f16 tiles already in the tensor core's
//             K-major 128-byte-swizzled shared-memory layout (pack_x), so the GEMM fetches them with
//             one bulk async copy per 64-wide K chunk.  Raw weight blocks are bulk-copied into a
//             staging ring, eight warps dequantise them into the swizzled f16 A tile, one thread
//             issues tcgen05.mma (M=128, N=NT, K=16) accumulating in tensor memory, and the same
//             eight warps read the accumulator back with tcgen05.ld and store y.
//             Calls whose weights allow it go to pairs of SMs (qmm_duo.cu); the row-sharded form and the rest run here.
//   qmm_simt  plain CUDA-core tile kernel with the same operand rounding; used for shapes the
//             tcgen05 kernel does not take and as an on-device cross-check.
#include <cuda_fp16.h>

#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "dequant.cuh"
#include "ptx.cuh"
#include "qmm.cuh"
#include "tensor_map.cuh"

namespace mlxn {

// =================================================================================================
// element-wise dequantisation helpers
// =================================================================================================
// Exact value of element `e` of a weight row stored as raw GGML blocks (global memory).
template <int T> __device__ __forceinline__ float dequant_elem(const uint8_t *row, uint32_t e) {
    if constexpr (T == GT_Q4_0) {
        const uint8_t *blk = row + 18u * (e >> 5);
        const uint32_t i = e & 31u;
        const uint32_t byte = blk[2 + (i & 15u)];
        const int nib = (i < 16) ? (int)(byte & 15u) : (int)(byte >> 4);
        return half_bits_to_float(ld_u16(blk)) * (float)(nib - 8);
    } else if constexpr (T == GT_Q8_0) {
        const uint8_t *blk = row + 34u * (e >> 5);
        return half_bits_to_float(ld_u16(blk)) * (float)(int)(int8_t)blk[2 + (e & 31u)];
    } else if constexpr (T == GT_Q4_K) {
        // f16 d, f16 dmin, scales[12], qs[128]; sub-block j = e / 32 of the super-block, byte (j / 2) * 32 + l,
        // low nibble for even j (src/gguf/mod.rs:582-644).  (d sc) q - (dmin m), each step rounded in f32.
        const uint8_t *blk = row + 144u * (e >> 8);
        const uint32_t r = e & 255u, j = r >> 5, l = r & 31u;
        uint32_t sc, mn;
        q4k_scale_min(j, blk + 4, sc, mn);
        const uint32_t byte = blk[16 + 32 * (j >> 1) + l];
        const uint32_t q = (j & 1u) ? (byte >> 4) : (byte & 15u);
        const float dj = __fmul_rn(half_bits_to_float(ld_u16(blk)), (float)sc);
        const float mj = __fmul_rn(half_bits_to_float(ld_u16(blk + 2)), (float)mn);
        return __fsub_rn(__fmul_rn(dj, (float)q), mj);
    } else {
        const uint8_t *blk = row + 210u * (e >> 8);
        const uint32_t r = e & 255u, h = r >> 7, g = (r & 127u) >> 5, l = r & 31u;
        const uint32_t qlb = blk[64 * h + 32 * (g & 1u) + l];
        const uint32_t nib = (g < 2) ? (qlb & 15u) : (qlb >> 4);
        const uint32_t hb = (blk[128 + 32 * h + l] >> (2 * g)) & 3u;
        const int q = (int)(nib | (hb << 4)) - 32;
        const float sc = (float)(int)(int8_t)blk[192 + 8 * h + (l >> 4) + 2 * g];
        return half_bits_to_float(ld_u16(blk + 208)) * sc * (float)q;
    }
}

__device__ __forceinline__ float round_f16(float v) { return __half2float(__float2half_rn(v)); }

// =================================================================================================
// qmm_simt: 64 x 64 output tile, K step 32, 256 threads, 4 x 4 outputs per thread
// =================================================================================================
// grid (ceil(rows/64), ceil(n/64), n_experts or 1)
template <int T>
__global__ void __launch_bounds__(256) qmm_simt_kernel(const QmmArgs a) {
    __shared__ float Ws[32][64 + 1];
    __shared__ float Xs[32][64 + 1];
    __shared__ int32_t orow[64];  // output row of each tile row, -1 if none
    __shared__ int32_t xrow[64];  // activation row of each tile row
    const uint32_t tid = threadIdx.x;
    const uint32_t r1 = blockIdx.x * 64, r0 = blockIdx.y * 64, e = blockIdx.z;
    const uint8_t *w = a.w;
    uint32_t nrows = a.m;
    if (a.hids) {
        nrows = a.htpe[e];
        if (r1 >= nrows) return;
        w += (size_t)e * a.expert_stride;
    }
    if (tid < 64) {
        int32_t o = -1, xr = 0;
        if (r1 + tid < nrows) {
            if (a.hids) {
                const int32_t id = a.hids[(size_t)e * a.hids_stride + r1 + tid];
                if (id >= 0 && (uint32_t)id < a.total_rows) {
                    o = id;
                    xr = id / (int32_t)a.top_k;
                }
            } else {
                o = (int32_t)(r1 + tid);
                xr = o;
            }
        }
        orow[tid] = o;
        xrow[tid] = xr;
    }
    __syncthreads();
    const size_t row_bytes = (size_t)(a.k / BlockTraits<T>::QK) * BlockTraits<T>::BYTES;
    const uint32_t tx = tid & 15, ty = tid >> 4;  // tx: weight-row quad, ty: activation-row quad
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
    for (uint32_t k0 = 0; k0 < a.k; k0 += 32) {
        for (uint32_t idx = tid; idx < 64 * 32; idx += 256) {
            const uint32_t rr = idx >> 5, kk = idx & 31u;
            float wv = 0.0f, xv = 0.0f;
            if (k0 + kk < a.k) {
                if (r0 + rr < a.n) wv = round_f16(dequant_elem<T>(w + (size_t)(r0 + rr) * row_bytes, k0 + kk));
                if (orow[rr] >= 0) xv = round_f16(a.x[(size_t)xrow[rr] * a.k + k0 + kk]);
            }
            Ws[kk][rr] = wv;
            Xs[kk][rr] = xv;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < 32; kk++) {
            float wv[4], xv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                wv[i] = Ws[kk][tx * 4 + i];
                xv[i] = Xs[kk][ty * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int32_t o = orow[ty * 4 + i];
        if (o < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t col = r0 + tx * 4 + j;
            if (col < a.n) a.y[(size_t)o * a.n + col] = acc[i][j];
        }
    }
}

// =================================================================================================
// routed tile list + activation packing for qmm_tc
// =================================================================================================
// Scratch header written by build_tiles: [0] = number of tiles, [1..] = (expert, row-tile) pairs.
// One CTA of 256 threads: thread i takes expert base + i, a block-wide exclusive prefix sum of the experts' tile
// counts gives each expert its place in the list (experts ascending, row tiles ascending inside an expert).
__global__ void __launch_bounds__(256) build_tiles_kernel(const uint32_t *htpe, uint32_t n_experts, uint32_t nt,
                                                          uint32_t max_tiles, uint32_t *tiles) {
    __shared__ uint32_t warp_tot[8];
    __shared__ uint32_t carry_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    grid_dependency_wait();
    allow_dependents();
    if (tid == 0) carry_s = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n_experts; base += 256) {
        const uint32_t e = base + tid;
        const uint32_t cnt = e < n_experts ? (__ldcg(htpe + e) + nt - 1) / nt : 0u;
        uint32_t incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        uint32_t before = carry_s;
        for (uint32_t w = 0; w < warp; w++) before += warp_tot[w];
        uint32_t pos = before + incl - cnt;
        for (uint32_t mt = 0; mt < cnt && pos < max_tiles; mt++, pos++) {
            tiles[1 + 2 * pos] = e;
            tiles[2 + 2 * pos] = mt;
        }
        __syncthreads();
        if (tid == 255) carry_s = before + incl;
        __syncthreads();
    }
    if (tid == 0) tiles[0] = carry_s < max_tiles ? carry_s : max_tiles;
}

// Packs activation rows into f16 tiles of nt rows (a multiple of 16) x 64 columns laid out exactly as the tensor core
// reads a K-major 128-byte-swizzled operand: row r, 16-byte chunk j (8 halves) of a tile lives at
// (r/8)*1024 + (r%8)*128 + ((j ^ (r%8)) * 16).  Tile (t, kc) starts at ((t*nchunks + kc) * nt*128) bytes.
// A CTA packs a slice of 64 rows, which is two 16-byte columns per thread and chunk: with whole tiles of 256 rows per CTA,
// 512 x 4096 activations took 10 us, most of it one load after another; with slices 6.
// grid (tiles x slices, K-chunk lanes), 256 threads.
// Eight floats (`left` of them and zeros), by one load where they are a whole 32-byte sector: from L2, two loads fetch every sector twice.
__device__ __forceinline__ void load8(const float *p, uint32_t left, float (&v)[8]) {
    if (left >= 8 && ((uintptr_t)p & 31u) == 0) {
        asm volatile("ld.global.cg.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "l"(p));
    } else if (left >= 8 && ((uintptr_t)p & 15u) == 0) {
        const float4 lo = __ldcg(reinterpret_cast<const float4 *>(p)), hi = __ldcg(reinterpret_cast<const float4 *>(p) + 1);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
        v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
        for (uint32_t u = 0; u < 8; u++) v[u] = u < left ? __ldcg(p + u) : 0.0f;
    }
}
template <bool SWIGLU>
__global__ void __launch_bounds__(256, SWIGLU ? 4 : 5) pack_x_kernel(const QmmArgs a, uint8_t *xpack, uint32_t nchunks, uint32_t nt, const TcShare sh, const __grid_constant__ TcOut res) {
    // CTA (t, c) packs the chunks c, c + gridDim.y, ... of its slice, so that the slice's routing lookups (a chain of
    // dependent loads) are paid once per CTA, not once per chunk.
    const uint32_t slices = (nt + kPackRows - 1) / kPackRows, t = blockIdx.x / slices, r0 = (blockIdx.x - t * slices) * kPackRows;
    grid_dependency_wait();   // (what the kernel ahead has written is read from L2: this SM's L1 may hold lines from before)
    allow_dependents();   // the mat-mat kernel behind may set itself up; it waits for this grid before it reads anything
    if (sh.ctas) {  // output tiles that two CTAs of the mat-mat share are added up in y (dense form only): zero them, 64 rows at a time
        const uint32_t pieces = (sh.nt + kPackRows - 1) / kPackRows, halves = sh.rows / 128u, jobs = (sh.ctas - 1) * pieces * halves;
        for (uint32_t j = blockIdx.y * gridDim.x + blockIdx.x; j < jobs; j += gridDim.x * gridDim.y) {
            const uint32_t q = j / halves, b = q / pieces, pos = sh.begin(b + 1), tile = pos / sh.nraw;
            if (tile * sh.nraw == pos) continue;   // the boundary between two CTAs is one between tiles
            const uint32_t tt = tile / sh.n_wt, lo = (q - b * pieces) * kPackRows, end = min(a.m, tt * sh.nt + min(sh.nt, lo + kPackRows));
            uint32_t wt = tile - tt * sh.n_wt;
            const uint32_t o = res.find(wt), col = wt * sh.rows + (j - q * halves) * 128u + (threadIdx.x & 127u);
            if (col < res.n[o])
                for (uint32_t row = tt * sh.nt + lo + (threadIdx.x >> 7); row < end; row += 2) res.y[o][(size_t)row * res.n[o] + col] = 0.f;
        }
    }
    uint32_t e = 0, mt = t, nrows = a.m;
    if (a.hids) {
        if (t >= __ldcg(a.tiles)) return;
        e = __ldcg(a.tiles + 1 + 2 * t);
        mt = __ldcg(a.tiles + 2 + 2 * t);
        nrows = __ldcg(a.htpe + e);
    }
    constexpr int kPer = 2;   // (row, 16-byte column) pairs per thread: the same ones in every chunk
    const float *src_row[kPer];
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        const uint32_t r = r0 + ((threadIdx.x + i * 256) >> 3), row = mt * nt + r;
        src_row[i] = nullptr;
        if (r < nt && row < nrows) {
            int64_t src = row;
            if (a.hids) {
                const int32_t id = __ldcg(a.hids + (size_t)e * a.hids_stride + row);
                src = (id >= 0 && (uint32_t)id < a.total_rows) ? id / (int32_t)a.top_k : -1;
            }
            // (perm021 form: the pointer only marks the row as present; the element addresses are formed per chunk)
            if (src >= 0) src_row[i] = a.x_bf16 ? reinterpret_cast<const float *>(a.x_bf16) : a.x + (size_t)src * a.k;
        }
    }
    for (uint32_t kc = blockIdx.y; kc < nchunks; kc += gridDim.y) {
        uint8_t *tile = xpack + ((size_t)t * nchunks + kc) * (size_t)(nt * 128);
        const uint32_t k0 = kc * 64 + 8 * (threadIdx.x & 7u);   // (the same columns in both rows)
        float v[kPer][8];
        [[maybe_unused]] float z[SWIGLU ? kPer : 1][8];
        // all loads first
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            if (!src_row[i] || k0 >= a.k) continue;
            if (a.x_bf16) {
                // eight consecutive K values lie inside one head (head_dim is a multiple of 32): 16 bytes of bf16
                const uint32_t h = k0 / a.head_dim, d0 = k0 - h * a.head_dim, row = mt * nt + r0 + ((threadIdx.x + i * 256) >> 3);
                const uint4 raw = __ldcg(reinterpret_cast<const uint4 *>(a.x_bf16 + ((size_t)h * a.m + row) * a.head_dim + d0));
                const uint32_t w4[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int u = 0; u < 4; u++) {   // bf16 -> f32 is exact; f32 -> f16 rounds to nearest even below
                    v[i][2 * u] = __uint_as_float(w4[u] << 16);
                    v[i][2 * u + 1] = __uint_as_float(w4[u] & 0xFFFF0000u);
                }
            } else {
                load8(src_row[i] + k0, a.k - k0, v[i]);
                if constexpr (SWIGLU) load8(a.x2 + (src_row[i] + k0 - a.x), a.k - k0, z[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            const uint32_t q = threadIdx.x + i * 256, r = r0 + (q >> 3), j = q & 7u;
            if (r >= nt) break;
            uint4 out = make_uint4(0, 0, 0, 0);
            if (src_row[i] && k0 < a.k) {
                if constexpr (SWIGLU) {   // fused SwiGLU: the same expression as the stand-alone kernel, so the same f32 values
#pragma unroll
                    for (int u = 0; u < 8; u++) v[i][u] = v[i][u] / (1.0f + expf(-v[i][u])) * z[i][u];
                }
                const __half2 h0 = __floats2half2_rn(v[i][0], v[i][1]), h1 = __floats2half2_rn(v[i][2], v[i][3]);
                const __half2 h2 = __floats2half2_rn(v[i][4], v[i][5]), h3 = __floats2half2_rn(v[i][6], v[i][7]);
                out = make_uint4(h2_as_u32(h0), h2_as_u32(h1), h2_as_u32(h2), h2_as_u32(h3));
            }
            *reinterpret_cast<uint4 *>(tile + (r >> 3) * 1024 + (r & 7u) * 128 + ((j ^ (r & 7u)) << 4)) = out;
        }
    }
}

template __global__ void pack_x_kernel<false>(const QmmArgs, uint8_t *, uint32_t, uint32_t, const TcShare, const __grid_constant__ TcOut);

// =================================================================================================
// qmm_tc
// =================================================================================================
// Dequantising warps: 16 in two sets of 8, set s dequantises the K stages with st % 2 == s.  Beside them the activation producer, MMA,
// weight producer and second MMA warp.
constexpr int kTcDequantWarps = 16, kTcThreads = (kTcDequantWarps + 4) * 32;
constexpr int kTcRowsW = 128;                           // weight rows per tile (UMMA M)

template <int T> struct TcTraits;
template <> struct TcTraits<GT_Q4_0> { static constexpr int KR = 256; };  // raw-stage K extent
template <> struct TcTraits<GT_Q8_0> { static constexpr int KR = 256; };
template <> struct TcTraits<GT_Q6_K> { static constexpr int KR = 256; };
template <> struct TcTraits<GT_Q4_K> { static constexpr int KR = 256; };

// position in a ring of `stages` slots plus the phase bit of the slot's current use (no divisions)
struct RingPos {
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void adv(uint32_t n, uint32_t stages) {
        s += n;
        while (s >= stages) {
            s -= stages;
            ph ^= 1u;
        }
    }
};

struct TcCfg {
    uint32_t nchunks;     // ceil(k / 64)
    uint32_t b_stages;    // depth of the activation ring, in 64-wide K chunks
    uint32_t seg_stride;  // bytes reserved per raw row segment
    uint32_t b_off, raw_off;
    uint32_t raw_slots;   // depth of the raw weight ring (2..6)
    uint32_t aligned;     // every weight row starts on a 16-byte boundary and k % 256 == 0: static-offset 16-byte raw reads
    uint32_t debug;       // experiment switches: 1 = skip dequantisation, 2 = skip raw copies, 4 = skip MMA, 8 = skip B copies
    uint32_t n_wt;        // weight-row tiles, ceil(n / 128)
    uint32_t ntiles;      // activation tiles: the count (dense) or its bound (routed: the list's length is read on the device)
    uint32_t nt;          // activation rows of a tile (a multiple of 16, at most NT)
    TcShare share;        // the CTAs' ranges where tiles are shared
    uint32_t stage_off;   // byte offset of the two staged output tiles (narrow tiles only), 0 = write y straight from registers
    uint32_t raw_tma;     // raw weight stages arrive as tensor copies; otherwise 16-byte cp.async
    uint32_t row_group;   // log2 of the copies of a stage: the map's rows are groups of 1, 2, 4 or 8 weight rows (see launch_tc_tn)
};

// ring of dequantised weight stages held in tensor memory: the columns the accumulators leave free.  Tiles of 64
// activation rows (two 64-column accumulators) keep six stages in columns [128, 512), wider ones four in [256, 512):
// the ring's depth over the latency of the loop dequantise -> MMA -> commit -> reuse is what bounds a narrow tile.
template <int NT> struct TcRing {
    static constexpr int kStages = NT <= 64 ? 6 : 4;
    static constexpr int kColBase = NT <= 64 ? 128 : 256;
};
constexpr int kTcACols = 64;       // one stage: 128 K values as f16 pairs = 64 32-bit columns
constexpr int kTcTmemCols = 512;

// grid = min(work items, SMs) persistent CTAs, one per SM; kTcThreads threads.
//
// Data flow per work item (one 128-row weight tile x one NT-row activation tile, all of K or, where tiles are shared, a part of it):
//   raw GGML blocks  --cp.async-->  shared-memory ring  --dequantise (16 warps)-->  f16 pairs in registers
//   --tcgen05.st-->  tensor-memory ring (A operand)  --tcgen05.mma, B = packed activations from the bulk-copy
//   ring in shared memory-->  f32 accumulator in tensor memory  --tcgen05.ld-->  y.
// The dequantised weights never touch shared memory: its bandwidth is the scarce resource here (the tensor
// core already reads the whole activation tile from it for every MMA).
template <int T, int NT, bool SH>
__global__ void __launch_bounds__(kTcThreads, 1) qmm_tc_kernel(const QmmArgs a, const TcCfg c, const uint8_t *xpack,
                                                               const __grid_constant__ CUtensorMap wmap) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // tensor-core operand tiles need 1024-byte alignment (128-byte swizzle atoms): align by hand
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int QK = BlockTraits<T>::QK, BB = BlockTraits<T>::BYTES, KR = TcTraits<T>::KR;
    constexpr int kMaxB = 8, kMaxRaw = 6;
    constexpr int kTcAStages = TcRing<NT>::kStages, kTcAColBase = TcRing<NT>::kColBase;
    static_assert(kMaxB / 2 <= kTcAStages, "an activation chunk's place is freed by a stage_done phase the producer can still see");
    constexpr int kNumMma = NT > 128 ? 1 : 2;   // issuing threads, each with its own accumulator
    __shared__ __align__(8) uint64_t a_full[kTcAStages], stage_done[kTcAStages], b_full[kMaxB];
    __shared__ __align__(8) uint64_t raw_full[kMaxRaw], raw_empty[kMaxRaw], acc_full, acc_empty, orow_ready[2], stage_ready[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile uint32_t abort_flag;
    __shared__ int32_t orow[2][NT];
    // SH (row-sharded result): the peers' result buffers, copied out of the parameter block once.  The plain form is a
    // separate instantiation: the peer stores' presence alone cost it 15 % (indexed reads of the parameter block).
    __shared__ float *peer_y[SH ? 7 : 1];

    // Warps 0-3 are the four single-thread roles (one per scheduler partition, and the lowest warp numbers, so that
    // they are served before the dequantising warps whenever both have an instruction ready: these threads are the
    // critical path and lose hundreds of cycles per K stage otherwise); warps 4-19 dequantise.
    constexpr uint32_t kWarpActs = 0, kWarpMma0 = 1, kWarpWeights = 2, kWarpMma1 = 3, kCtrlWarps = 4;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tid = threadIdx.x - kCtrlWarps * 32;   // index among the dequantising threads (wraps for warps 0-3)
    const uint32_t row_bytes = (a.k / QK) * BB;
    const bool raw_tma = c.raw_tma != 0;

    // ---- set-up that needs nothing from the kernels ahead in the stream (it overlaps their tail: the kernel is
    // ---- launched with programmatic stream serialisation), then the wait for them
    if (threadIdx.x == 0) {
        abort_flag = 0;
        if constexpr (SH) {
            peer_y[0] = a.y_peer[0]; peer_y[1] = a.y_peer[1]; peer_y[2] = a.y_peer[2]; peer_y[3] = a.y_peer[3];
            peer_y[4] = a.y_peer[4]; peer_y[5] = a.y_peer[5]; peer_y[6] = a.y_peer[6];
        }
        for (uint32_t s = 0; s < kTcAStages; s++) {
            mbar_init(&a_full[s], 8);  // the eight warps of one set
            mbar_init(&stage_done[s], 1);
        }
        for (uint32_t s = 0; s < c.b_stages; s++) mbar_init(&b_full[s], 1);
        for (uint32_t s = 0; s < c.raw_slots; s++) {
            // one asynchronous arrival per copying thread, or the weight producer's single arrival with the byte count
            mbar_init(&raw_full[s], raw_tma ? 1u : kTcDequantWarps * 32);
            mbar_init(&raw_empty[s], kTcDequantWarps);
        }
        mbar_init(&acc_full, kNumMma);
        mbar_init(&acc_empty, kTcDequantWarps);
        for (int s = 0; s < 2; s++) {
            mbar_init(&orow_ready[s], kTcDequantWarps);
            mbar_init(&stage_ready[s], kTcDequantWarps);
        }
        mbar_init_fence();
    }
    if (warp == kWarpMma0) {  // the first MMA warp owns tensor memory
        tmem_alloc(&tmem_base_s, kTcTmemCols);
        tmem_relinquish();
    }
    grid_dependency_wait();   // the packed activations, the tile list and the zeros of shared tiles are complete
    allow_dependents();

    // ---- work items: (weight-row tile, token tile), weight tile fastest; CTA b takes items b, b + grid, ... or, where
    // tiles are shared (TcShare), the parts of tiles that lie in its range.  Every role walks the same item sequence; ring slots and barrier phases run on across items, so the next
    // item's weights are already on their way while this item's accumulator is read back.
    const uint32_t n_tt = a.hids ? min(a.tiles[0], c.ntiles) : c.ntiles;   // uniform for the whole CTA
    const uint32_t total_items = c.n_wt * n_tt;
    const uint32_t nraw_all = (a.k + KR - 1) / KR;
    const bool shared = c.share.ctas != 0;
    const uint32_t nt = c.nt;
    const uint32_t pos0 = shared ? c.share.begin(blockIdx.x) : blockIdx.x, pos1 = shared ? c.share.begin(blockIdx.x + 1) : total_items;
    struct Item {
        uint32_t tt, e, mt, n0, r_lo, nraw, nst, nck, kc_lo, next;
        const uint8_t *wbase;
    };
    // routed: the (expert, row tile) pairs of the CTA's first items, fetched once (a lookup per item would put a
    // global-memory round trip in front of every role's start on the item)
    constexpr uint32_t kMetaItems = 32;
    __shared__ uint32_t meta[kMetaItems][2];
    if (a.hids && threadIdx.x < kMetaItems) {
        const uint32_t item = blockIdx.x + threadIdx.x * gridDim.x;
        if (item < total_items) {
            const uint32_t tt = item / c.n_wt;
            meta[threadIdx.x][0] = a.tiles[1 + 2 * tt];
            meta[threadIdx.x][1] = a.tiles[2 + 2 * tt];
        }
    }
    auto load_item = [&](uint32_t pos) -> Item {
        Item it;
        const uint32_t item = shared ? pos / nraw_all : pos;
        it.r_lo = shared ? pos - item * nraw_all : 0u;
        const uint32_t r_hi = shared ? min(nraw_all, it.r_lo + (pos1 - pos)) : nraw_all;
        it.next = shared ? pos + (r_hi - it.r_lo) : pos + gridDim.x;
        it.tt = item / c.n_wt;
        const uint32_t wt = item - it.tt * c.n_wt;
        it.e = 0;
        it.mt = it.tt;
        if (a.hids) {
            const uint32_t li = (item - blockIdx.x) / gridDim.x;   // the CTA's li-th item
            if (li < kMetaItems) {
                it.e = meta[li][0];
                it.mt = meta[li][1];
            } else {
                it.e = a.tiles[1 + 2 * it.tt];
                it.mt = a.tiles[2 + 2 * it.tt];
            }
        }
        it.wbase = a.w + (size_t)it.e * a.expert_stride;
        it.n0 = wt * kTcRowsW;
        it.nraw = r_hi - it.r_lo;
        it.kc_lo = it.r_lo * (KR / 64);
        it.nst = min((a.k + 127) / 128, r_hi * (KR / 128)) - it.r_lo * (KR / 128);   // tensor-memory stages
        it.nck = min(c.nchunks, r_hi * (KR / 64)) - it.kc_lo;                         // 64-wide activation chunks
        return it;
    };

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = tmem_base_s;
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t b_bytes = nt * 128;                 // one 64-wide K chunk of the activation tile
    const uint32_t raw_stage_bytes = kTcRowsW * c.seg_stride;
    // wait styles: the single producer / MMA warps spin (they are the critical path and cost one warp's issue
    // slots); the dequantising warps space their polls out
    const uint32_t wmode_cr = (MLXN_DBG(c) & 32u) ? 0u : 0xFFFFFFFFu;
    const uint32_t wmode_dq = (MLXN_DBG(c) & 16u) ? 0xFFFFFFFFu : 0u;
#ifdef MLXN_TC_TRACE
    // experiment: CTA 0 logs (event, clock) pairs into y (use with debug 256, which keeps the epilogue from writing y)
    uint32_t trace_n = 0;
    auto TRACE = [&](uint32_t role, uint32_t code, uint32_t x) {
        if ((MLXN_DBG(c) & 512u) && blockIdx.x == 0 && lane == 0 && trace_n < 500) {
            uint32_t *t = reinterpret_cast<uint32_t *>(a.y) + role * 1024 + 2 * trace_n;
            t[0] = (code << 16) | (x & 0xFFFFu);
            t[1] = (uint32_t)clock64();
            trace_n++;
        }
    };
#else
#define TRACE(role, code, x) ((void)0)
#endif

    if (warp == kWarpActs) {
        // ======================= producer warp: bulk copies of the packed activation tiles =======================
        // Every K stage owns two consecutive chunk slots of the ring (a K tail of 64 leaves its second one empty;
        // the producer still arrives on it so that the slot's phase moves on).  Chunk slot G reuses the place of
        // chunk slot G - b_stages, which belonged to K stage (G - b_stages) / 2: free once that stage's MMAs have
        // completed (stage_done, the same barrier the dequantising warps wait on before they overwrite the stage's
        // weights in tensor memory).  G and the stage numbers count on across items.
        if (lane == 0) {
            uint32_t s = 0, G = 0;
            bool ok = true;
            for (uint32_t pos = pos0; ok && pos < pos1;) {
                const Item it = load_item(pos);
                pos = it.next;
                for (uint32_t kc = 0; kc < 2 * it.nst; kc++, G++) {
                    if (G >= c.b_stages) {
                        const uint32_t j = (G - c.b_stages) >> 1;
                        if (!mbar_wait(&stage_done[j % kTcAStages], (j / kTcAStages) & 1u, &abort_flag, a.status,
                                       ST_WAIT_EMPTY_TIMEOUT, wmode_cr)) {
                            ok = false;
                            break;
                        }
                    }
                    if (kc >= it.nck || (MLXN_DBG(c) & 8u)) {
                        mbar_arrive(&b_full[s]);
                    } else {
                        mbar_expect_tx(&b_full[s], b_bytes);
                        bulk_g2s(smem + c.b_off + s * b_bytes,
                                 xpack + ((size_t)it.tt * c.nchunks + it.kc_lo + kc) * (size_t)b_bytes, b_bytes, &b_full[s]);
                    }
                    if (++s == c.b_stages) s = 0;
                }
            }
        }
    } else if (warp == kWarpWeights) {
        // ======================= weight producer warp: tensor copies of raw stages =======================
        // The weights as a 3-D tensor of 32-bit words [expert][row group][words]; a raw stage is 128 rows' bytes of 256 K values, each
        // from the 16-byte boundary below (readers skip the lead-in).  A copy brings one row of every group: rows i, i + G, ... of the
        // tile land together, i = 0 .. G - 1.  Rows past n arrive as zeros.  The copies run raw_slots - 1 stages ahead of the
        // dequantisation, across item boundaries.
        if (raw_tma && lane == 0) {
            const uint32_t R = c.raw_slots;
            uint32_t slot = 0, ph = 0, requested = 0;
            bool ok = true;
            for (uint32_t pos = pos0; ok && pos < pos1;) {
                const Item it = load_item(pos);
                pos = it.next;
                for (uint32_t r = 0; r < it.nraw; r++, requested++) {
                    if (requested >= R &&
                        !mbar_wait(&raw_empty[slot], ph ^ 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, wmode_cr)) {
                        ok = false;
                        break;
                    }
                    TRACE(0, 1, requested);
                    const uint32_t kb = (it.r_lo + r) * (KR / QK) * BB;   // byte offset of the stage in a row
                    mbar_expect_tx(&raw_full[slot], raw_stage_bytes);
                    for (uint32_t i = 0; i < 1u << c.row_group; i++)
                        asm volatile(
                            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                            ::"r"(smem_base + c.raw_off + slot * raw_stage_bytes + i * (raw_stage_bytes >> c.row_group)), "l"(&wmap),
                              "r"(((i * row_bytes + kb) & ~15u) >> 2), "r"(it.n0 >> c.row_group), "r"(it.e), "r"(smem_u32(&raw_full[slot]))
                            : "memory");
                    if (++slot == R) { slot = 0; ph ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == kWarpMma0 || warp == kWarpMma1) {
        // ======================= MMA warps: one thread each issues tcgen05.mma =======================
        // A lone thread gets through one of these instructions (MMA, commit, barrier test) every 50-100 cycles, and
        // a K stage costs about thirteen of them, which bounds a narrow tile (NT <= 128: the MMAs themselves are
        // short) well before the tensor core does.  So narrow tiles use two issuing threads: thread w takes the K
        // stages st with st % 2 == w and accumulates them in its own accumulator (columns [w NT, (w+1) NT)); the
        // epilogue adds the two.  NT = 256 keeps one thread (tensor memory has no room for a second accumulator,
        // and there the MMAs are long enough to hide the issue).
        const uint32_t w = warp == kWarpMma0 ? 0u : 1u;
        if (lane == 0 && w < (uint32_t)kNumMma) {
            const uint32_t idesc = umma_idesc_f16(kTcRowsW, nt);
            const uint64_t bd0 = umma_desc_k_sw128(smem_base + c.b_off);
            const uint64_t b_step = b_bytes >> 4;  // descriptor address field is in 16-byte units
            const bool do_mma = !(MLXN_DBG(c) & 4u);
            const uint32_t d_col = tmem_d + w * NT;
            uint32_t sa = 0, aph = 0, sb = 0, bph = 0, nitem = 0;   // ring positions of the stage being looked at
            bool ok = true;
            for (uint32_t pos = pos0; ok && pos < pos1; nitem++) {
                const Item it = load_item(pos);
                pos = it.next;
                // the accumulators of the item before have been read back
                if (nitem > 0 &&
                    !mbar_wait(&acc_empty, (nitem - 1) & 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, wmode_cr))
                    break;
                tc_fence_after();
                TRACE(1 + 3 * w, 1, nitem);
                bool issued = false;
                for (uint32_t st = 0; st < it.nst; st++) {
                    if ((st & (uint32_t)(kNumMma - 1)) == w) {
                        if (!mbar_wait(&a_full[sa], aph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, wmode_cr)) { ok = false; break; }
                        TRACE(1 + 3 * w, 2, st);
                        if (!mbar_wait(&b_full[sb], bph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, wmode_cr)) { ok = false; break; }
                        tc_fence_after();
                        TRACE(1 + 3 * w, 4, st);
                        const uint32_t a_col = tmem_d + kTcAColBase + sa * kTcACols;
                        const uint64_t bd = bd0 + sb * b_step;
                        if (do_mma) {
                            umma_f16_ts(d_col, a_col, bd, idesc, issued ? 1u : 0u);
                            umma_f16_ts(d_col, a_col + 8, bd + 2, idesc, 1u);
                            umma_f16_ts(d_col, a_col + 16, bd + 4, idesc, 1u);
                            umma_f16_ts(d_col, a_col + 24, bd + 6, idesc, 1u);
                        }
                        issued = true;
                        if (2 * st + 1 < it.nck) {
                            const uint32_t sb1 = sb + 1 == c.b_stages ? 0u : sb + 1;
                            const uint32_t bph1 = sb + 1 == c.b_stages ? bph ^ 1u : bph;
                            if (!mbar_wait(&b_full[sb1], bph1, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, wmode_cr)) { ok = false; break; }
                            const uint64_t bd1 = bd0 + sb1 * b_step;
                            if (do_mma) {
                                umma_f16_ts(d_col, a_col + 32, bd1, idesc, 1u);
                                umma_f16_ts(d_col, a_col + 40, bd1 + 2, idesc, 1u);
                                umma_f16_ts(d_col, a_col + 48, bd1 + 4, idesc, 1u);
                                umma_f16_ts(d_col, a_col + 56, bd1 + 6, idesc, 1u);
                            }
                        }
                        TRACE(1 + 3 * w, 5, st);
                        umma_commit(&stage_done[sa]);  // frees the stage's weights and its two activation chunks
                        TRACE(1 + 3 * w, 3, st);
                    }
                    // on to the next stage's ring places (two activation chunk slots per stage, used or not)
                    sb += 2;
                    if (sb >= c.b_stages) { sb -= c.b_stages; bph ^= 1u; }
                    if (++sa == kTcAStages) { sa = 0; aph ^= 1u; }
                }
                if (!ok) break;
                // this thread's share of the item is issued: its accumulator is complete when these MMAs are
                if (issued) umma_commit(&acc_full);
                else mbar_arrive(&acc_full);
            }
        }
        __syncwarp();
    } else {
        // ======================= dequantise warps, then epilogue =======================
        // The 16 warps form two sets of 8; set s fills the K stages st with st % 2 == s, so that a warp has two
        // stage times for each of its turns.  Within a set, thread (warp w, lane l) owns weight row
        // 32 (w % 4) + l of the tile -- the tensor-memory lane its warp may address -- and the 64-element half
        // (w / 4) % 2 of the stage: thirty-two packed f16 pairs = one 32-column store.
        const uint32_t dw = warp - kCtrlWarps;   // 0..15
        const uint32_t q4 = dw & 3u, half = (dw >> 2) & 1u, set = dw >> 3;
        const uint32_t rr = q4 * 32 + lane;
        const uint32_t srow = ((rr & ((1u << c.row_group) - 1u)) << (7 - c.row_group)) + (rr >> c.row_group);   // the row's place in a raw stage
        // Raw weight rows are short (144..272 bytes per stage and row), too short for one bulk copy each to be
        // efficient, so all dequantising threads stream them as 16-byte cp.async chunks, a few raw stages ahead
        // of the one being dequantised.  Each row is fetched as the 16-byte aligned superset of its (only
        // 2-byte aligned) segment; readers skip the lead-in bytes.
        // The (row, 16-byte chunk) pairs a thread copies are the same in every raw stage and every item; per item
        // only the rows' base addresses change, per stage only the K offset.
        constexpr int kRawSlots = 5;            // (128 rows x at most 19 chunks) / 512 threads, rounded up
        constexpr uint32_t kSegFull = (KR / QK) * BB;
        constexpr uint32_t kCmax = (kSegFull + 30u) >> 4;  // most 16-byte chunks a row segment can need
        static_assert(kTcRowsW * kCmax <= kRawSlots * kTcDequantWarps * 32, "raw copy slots");
        static_assert(KR == 256, "a raw stage feeds one K stage of each set");
        const uint8_t *slot_src[kRawSlots];     // start of the thread's row (global), for the item being requested
        uint32_t slot_dst[kRawSlots];           // row's place inside a raw stage + chunk offset (shared, relative)
        uint32_t slot_cc[kRawSlots];            // chunk index within the row, 0xFFFFFFFF = unused in this item
        // request cursor: runs ahead of the dequantisation, across item boundaries
        uint32_t q_pos = pos0, q_next = pos0, q_r = 0, q_nraw = 0, q_rlo = 0;
        auto open_request_item = [&]() {
            const Item it = load_item(q_pos);
            q_next = it.next;
            const uint32_t rows_here = min((uint32_t)kTcRowsW, a.n - it.n0);
#pragma unroll
            for (int i = 0; i < kRawSlots; i++) {
                const uint32_t idx = tid + i * (kTcDequantWarps * 32);
                const uint32_t row = idx / kCmax, cc = idx - row * kCmax;
                const bool used = row < rows_here;
                slot_src[i] = it.wbase + (size_t)(it.n0 + (used ? row : 0)) * row_bytes;
                slot_dst[i] = row * c.seg_stride + cc * 16u;
                slot_cc[i] = used ? cc : 0xFFFFFFFFu;
            }
            q_r = 0;
            q_nraw = it.nraw;
            q_rlo = it.r_lo;
        };
        if (!raw_tma && q_pos < pos1) open_request_item();
        auto issue_raw = [&](uint32_t r, uint32_t slot) {
            const uint32_t k0 = r * KR;
            const uint32_t seg_bytes = (min((uint32_t)KR, a.k - k0) / QK) * BB;
            const uint32_t koff = (k0 / QK) * BB;
            const uint32_t dst0 = smem_base + c.raw_off + slot * raw_stage_bytes;
#pragma unroll
            for (int i = 0; i < kRawSlots; i++) {
                const uint8_t *src = slot_src[i] + koff;
                const uint32_t pre_b = (uint32_t)((uintptr_t)src & 15u);
                if (slot_cc[i] != 0xFFFFFFFFu && slot_cc[i] * 16u < pre_b + seg_bytes && !(MLXN_DBG(c) & 2u))
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + slot_dst[i]),
                                 "l"(src - pre_b + slot_cc[i] * 16u)
                                 : "memory");
            }
            // the thread's arrival on the slot's barrier fires once its copies have landed; nobody blocks on it
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[slot])) : "memory");
        };
        // raw ring: a stage is requested raw_slots-1 stages before it is read; slots and phases count on across items
        const uint32_t R = c.raw_slots, D = R - 1;
        uint32_t islot = 0, iph = 0;   // slot / use-parity of the next stage to request
        uint32_t requested = 0, consumed = 0;
        uint32_t rs = 0, rph = 0;      // slot / parity of the raw stage being read
        uint32_t J0 = 0;               // K stages of the items before this one (tensor-memory ring position)
        uint32_t nitem = 0;
        bool ok = true;
        const uint32_t a_dst = tmem_d + ((q4 * 32) << 16) + kTcAColBase + 32 * half;
        const uint32_t g = dw >> 2;
        for (uint32_t pos = pos0; ok && pos < pos1; nitem++) {
            const Item it = load_item(pos);
            pos = it.next;
            const uint32_t n0 = it.n0;
            const bool row_ok = n0 + rr < a.n;
            const uint32_t row_lo4 = (uint32_t)((uintptr_t)(it.wbase + (size_t)(n0 + rr) * row_bytes) & 15u);
            // the item's output-row table: every thread fetches the entries it will publish now (the loads stay in
            // flight behind the K loop) and stores them just before the epilogue
            static_assert(NT <= kTcDequantWarps * 32, "one output-row entry per thread");
            if (q4 == 0 && half == 0) TRACE(2 + set, 1, nitem);
            uint32_t o_nrows = a.m;
            int32_t o_id = -1;
            const uint32_t o_row = it.mt * nt + tid;
            if (a.hids && tid < nt) {
                o_nrows = a.htpe[it.e];
                if (o_row < a.hids_stride) o_id = a.hids[(size_t)it.e * a.hids_stride + o_row];
            }
            for (uint32_t r = 0; ok && r < it.nraw; r++) {
                // keep D raw stages requested ahead of the one being read
                while (!raw_tma && q_pos < pos1 && requested - consumed < D + 1) {
                    if (requested >= R &&
                        !mbar_wait(&raw_empty[islot], iph ^ 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, wmode_dq)) {
                        ok = false;
                        break;
                    }
                    issue_raw(q_rlo + q_r, islot);
                    requested++;
                    if (++islot == R) { islot = 0; iph ^= 1u; }
                    if (++q_r == q_nraw) {
                        q_pos = q_next;
                        if (q_pos < pos1) open_request_item();
                    }
                }
                if (!ok) break;
                if (!mbar_wait(&raw_full[rs], rph, &abort_flag, a.status, ST_WAIT_FULL_TIMEOUT, wmode_dq)) { ok = false; break; }
                if (q4 == 0 && half == 0) TRACE(2 + set, 2, r);
                const uint32_t st = 2 * r + set;       // this set's K stage inside raw stage r
                if (st < it.nst) {
                    const uint32_t J = J0 + st;        // its number in the CTA's whole run
                    const uint32_t sa = J % kTcAStages;
                    // the MMAs that read this ring place's previous contents (K stage J - 4) have completed
                    if (J >= kTcAStages &&
                        !mbar_wait(&stage_done[sa], ((J / kTcAStages) & 1u) ^ 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT,
                                   wmode_dq)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (q4 == 0 && half == 0) TRACE(2 + set, 3, r);
                    const uint32_t r_abs = it.r_lo + r;
                    const uint32_t pre = (row_lo4 + ((r_abs * KR) / QK) * BB) & 15u;
                    const uint32_t seg = smem_base + c.raw_off + rs * raw_stage_bytes + srow * c.seg_stride + pre;
                uint32_t regs[32];
                if (T != GT_Q4_K && c.aligned && row_ok && !(MLXN_DBG(c) & 1u)) {   // (Q4_K: the generic extraction below)
                    const uint32_t stage_row = smem_base + c.raw_off + rs * raw_stage_bytes + srow * c.seg_stride;
                    if constexpr (T == GT_Q6_K) {
                        dequant64_q6k_aligned_p(r_abs & 7u, stage_row, set, half, regs);
                    } else if constexpr (T != GT_Q4_K) {
                        switch (2 * set + half) {  // uniform per warp
                        case 0: dequant64_aligned<T, 0>(stage_row, regs); break;
                        case 1: dequant64_aligned<T, 1>(stage_row, regs); break;
                        case 2: dequant64_aligned<T, 2>(stage_row, regs); break;
                        default: dequant64_aligned<T, 3>(stage_row, regs); break;
                        }
                    }
                } else {
#pragma unroll
                    for (uint32_t hh = 0; hh < 2; hh++) {
                        uint4 v[4];
                        const uint32_t e0 = 128 * set + 64 * half + 32 * hh;  // element offset inside the raw stage
                        if (row_ok && r_abs * KR + e0 < a.k && !(MLXN_DBG(c) & 1u)) {
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
                    if (q4 == 0 && half == 0) TRACE(2 + set, 8, r);
                    tmem_st_32x32_x32(a_dst + sa * kTcACols, regs);
                    tmem_st_wait();
                    if (q4 == 0 && half == 0) TRACE(2 + set, 9, r);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_full[sa]);
                    if (q4 == 0 && half == 0) TRACE(2 + set, 4, r);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[rs]);  // this warp is done reading the raw stage
                if (q4 == 0 && half == 0) TRACE(2 + set, 10, r);
                consumed++;
                if (++rs == R) { rs = 0; rph ^= 1u; }
            }
            if (!ok) break;
            J0 += it.nst;
            // ---- epilogue: TMEM -> registers -> y ----
            {   // double-buffered: the table of the item before may still be in use by a warp that is behind
                int32_t *wtab = orow[nitem & 1u];
                if (tid < NT) {
                    int32_t o = -1;
                    if (tid < nt && o_row < o_nrows) {
                        if (a.hids) {
                            if (o_id >= 0 && (uint32_t)o_id < a.total_rows) o = o_id;
                        } else {
                            o = (int32_t)o_row;
                        }
                    }
                    wtab[tid] = o;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&orow_ready[nitem & 1u]);
            }
            if (!mbar_wait(&orow_ready[nitem & 1u], (nitem >> 1) & 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, wmode_dq)) break;
            if (q4 == 0 && half == 0) TRACE(2 + set, 5, nitem);
            if (!mbar_wait(&acc_full, nitem & 1u, &abort_flag, a.status, ST_WAIT_MMA_TIMEOUT, wmode_dq)) break;
            tc_fence_after();
            if (q4 == 0 && half == 0) TRACE(2 + set, 6, nitem);
            const int32_t *tab = orow[nitem & 1u];
            const uint32_t wrow = n0 + rr;
            const bool part = it.nraw < nraw_all;   // another CTA has the rest of this tile's K
            if (c.stage_off) {
                // Staged read-back (narrow tiles): the accumulator goes to shared memory as [activation row][weight
                // row], tensor memory is handed back to the MMA warps at once, and every warp then writes whole
                // 512-byte output rows with 16-byte stores (the direct form below writes 128 bytes per instruction).
                constexpr uint32_t kPitch = kTcRowsW + 4;   // floats per staged row
                float *stg = reinterpret_cast<float *>(smem + c.stage_off) + (nitem & 1u) * (NT * kPitch);
#pragma unroll 1
                for (uint32_t col = g * 32; col < nt; col += (kTcDequantWarps / 4) * 32) {
                    uint32_t v[32];
                    tmem_ld_32x32(tmem_d + ((q4 * 32) << 16) + col, v);
                    if (kNumMma == 2 && it.nst >= 2) {
                        uint32_t v1[32];
                        tmem_ld_32x32(tmem_d + ((q4 * 32) << 16) + NT + col, v1);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(v1[j]));
                    }
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) stg[(col + j) * kPitch + rr] = __uint_as_float(v[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&acc_empty);                      // the MMA warps may start the next item
                    mbar_arrive(&stage_ready[nitem & 1u]);        // this warp's part of the staged tile is written
                }
                if (!mbar_wait(&stage_ready[nitem & 1u], (nitem >> 1) & 1u, &abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT, wmode_dq)) break;
                if (!(MLXN_DBG(c) & 256u)) {
                    const uint32_t c4 = n0 + 4 * lane;
                    for (uint32_t r = dw; r < NT; r += kTcDequantWarps) {
                        const int32_t o = tab[r];
                        if (o < 0) continue;
                        const float4 val = *reinterpret_cast<const float4 *>(stg + r * kPitch + 4 * lane);
                        // (the staged form is never chosen for a call that also stores to peers)
                        float *dst = SH ? a.y + ((size_t)o * qmm_ld(a) + a.y_col0 + c4) : a.y + ((size_t)o * a.n + c4);
                        if (c4 + 3 < a.n) {
                            *reinterpret_cast<float4 *>(dst) = val;
                        } else {
                            if (c4 < a.n) dst[0] = val.x;
                            if (c4 + 1 < a.n) dst[1] = val.y;
                            if (c4 + 2 < a.n) dst[2] = val.z;
                        }
                    }
                }
                if (q4 == 0 && half == 0) TRACE(2 + set, 7, nitem);
                continue;
            }
#pragma unroll 1
            for (uint32_t col = g * 32; col < nt; col += (kTcDequantWarps / 4) * 32) {
                uint32_t v[32];
                tmem_ld_32x32(tmem_d + ((q4 * 32) << 16) + col, v);
                if (kNumMma == 2 && it.nst >= 2) {   // the odd K stages went into the second accumulator
                    uint32_t v1[32];
                    tmem_ld_32x32(tmem_d + ((q4 * 32) << 16) + NT + col, v1);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(v1[j]));
                }
                tmem_ld_wait();
                if (wrow < a.n && !(MLXN_DBG(c) & 256u)) {
                    if constexpr (!SH) {   // a plain [m, n] result of this GPU: nothing between the 32 stores
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const int32_t o = tab[col + j];
                            if (o >= 0) {
                                if (part) atomicAdd(&a.y[(size_t)o * a.n + wrow], __uint_as_float(v[j]));
                                else a.y[(size_t)o * a.n + wrow] = __uint_as_float(v[j]);
                            }
                        }
                    } else {           // row-sharded: leading dimension, column offset, the same tile to every peer
#pragma unroll 4
                        for (int j = 0; j < 32; j++) {
                            const int32_t o = tab[col + j];
                            if (o >= 0) {
                                const size_t off = (size_t)o * qmm_ld(a) + a.y_col0 + wrow;
                                a.y[off] = __uint_as_float(v[j]);
                                for (uint32_t pr = 0; pr < a.n_peer; pr++) peer_y[pr][off] = __uint_as_float(v[j]);
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);   // the MMA warp may start the next item's accumulation
            if (q4 == 0 && half == 0) TRACE(2 + set, 7, nitem);
        }
    }
    if (abort_flag) {  // let copies in flight land before the CTA's shared memory is released
        for (int i = 0; i < 200; i++) __nanosleep(5000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kWarpMma0) {
        tc_fence_after();
        tmem_dealloc(tmem_d, kTcTmemCols);
    }
}

// =================================================================================================
// host-side launchers
// =================================================================================================
static thread_local const char *t_mat_mat = "";
static thread_local uint32_t t_mat_mat_rows = 0;
void note_mat_mat(const char *kernel, uint32_t tile_rows) {
    t_mat_mat = kernel;
    t_mat_mat_rows = tile_rows;
}

static inline uint32_t round_up_u(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }
int sm_count_of_device() {
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return sms[dev] ? sms[dev] : 148;
}

// Bytes of scratch the tcgen05 path needs for one call (tile list + packed activations).
size_t qmm_tc_scratch_bytes(const QmmArgs &a, uint32_t nt, bool routed) {
    const uint32_t nchunks = (a.k + 63) / 64;
    size_t tiles;
    size_t header = 0;
    if (routed) {
        tiles = (size_t)a.total_rows / nt + a.n_experts;
        if (tiles > a.total_rows) tiles = a.total_rows;
        if (tiles == 0) tiles = 1;
        header = ((1 + 2 * tiles) * 4 + 1023) / 1024 * 1024;
    } else {
        tiles = (a.m + nt - 1) / nt;
    }
    return header + tiles * nchunks * (size_t)nt * 128;
}

// Activation rows per tile and the CTAs' shares.  Routed calls use tiles of 64 rows, whole.  A dense call takes the combination
// that costs least.  A K stage of 128 values costs nt + 390 (units of 1.74 ns: 4096 x 4096 Q4_0 in one wave takes 30 us with 64
// rows, 33 with 128, 38 with 192 and 41 with 256: the chain from raw block to tensor memory bounds a stage, the multiplication adds
// to it), an item 2000 beside its stages.
//   * whole tiles: waves x tile.
//   * shared tiles, as many CTAs as SMs: no last wave, but one more hand-off, and the shared tiles are zeroed and added up in y.  Has
//     to promise 11 %: Q4_0 512 x 12288 x 4096 (1.3 waves of 256 rows) takes 66 us where whole tiles of 128 rows took 86; Q6_K 2048 x
//     4096 x 12288 (1.7 waves) took 300 us for the whole call, with whole tiles 295.
//   * every tile in two halves, where all halves fit on the chip at once and K is long enough (8 raw stages).
// Rows are spread evenly: 333 rows are two tiles of 176, not 256 and 77.
struct TcPlan {
    uint32_t nt, ctas, shared;
};
static uint64_t tc_plan(uint32_t nt, uint64_t rows, uint64_t n, uint64_t k, uint64_t sms, bool sharded, TcPlan &p) {
    const uint64_t tiles = (n + kTcRowsW - 1) / kTcRowsW * ((rows + nt - 1) / nt), nraw = (k + 255) / 256;
    const uint64_t tile = 2 * nraw * (nt + 390);   // a tile's stages
    uint64_t best = (tiles + sms - 1) / sms * (tile + 2000);
    p = {nt, (uint32_t)(tiles < sms ? tiles : sms), 0};
    if (sharded || tiles * nraw >= (1ull << 31)) return best;
    if (tiles > sms && nraw >= 2) {
        const uint64_t cost = (tiles * tile / sms + (tiles / sms + 2) * 3000) * 111 / 100;
        if (cost < best) {
            best = cost;
            p = {nt, (uint32_t)sms, 1};
        }
    } else if (2 * tiles <= sms && nraw >= 8) {
        const uint64_t cost = tile / 2 + 4600;
        if (cost < best) {
            best = cost;
            p = {nt, (uint32_t)(2 * tiles), 1};
        }
    }
    return best;
}

// The tiles that a dense call is offered, what the kernel on single SMs takes with them, and its choice.
struct TcChoice {
    uint32_t count, best, rows[9];
    uint64_t cost[9];
    TcPlan plan;   // of the chosen one
};
static void tc_choose(const QmmArgs &a, int sm_count, bool sharded, TcChoice &c) {
    uint64_t best_cost = ~0ull;
    c.count = 0;
    for (uint32_t tt = (a.m + 255) / 256; c.count < 9; tt++) {
        const uint32_t i = c.count++;
        TcPlan p;
        c.rows[i] = ((a.m + tt - 1) / tt + 15) / 16 * 16;
        c.cost[i] = tc_plan(c.rows[i], a.m, a.n, a.k, (uint64_t)sm_count, sharded, p);
        if (best_cost == ~0ull || c.cost[i] * 103 / 100 < best_cost) {   // (near a tie, the larger tile: it converts less in all)
            best_cost = c.cost[i];
            c.best = i;
            c.plan = p;
        }
        if (c.rows[i] == 16) break;
    }
}
static uint32_t tc_chain_limit(const QmmArgs &a, const TcChoice &c) {
    const uint32_t nraw = (a.k + 255) / 256, nt = c.rows[c.best];
    const uint64_t tiles = (uint64_t)((a.n + kTcRowsW - 1) / kTcRowsW) * ((a.m + nt - 1) / nt);
    const bool halves = c.plan.shared && c.plan.ctas == 2 * tiles;
    const uint32_t has = chain_mean(nraw, halves ? 2 : 1, nt > 128 ? 1 : 2, tiles, c.plan.shared && !halves ? c.plan.ctas - 1 : 0);
    const uint32_t least = a.k <= 512 ? kChainAny : (uint32_t)(4096ull * 512 * 512 / ((uint64_t)a.k * a.k));
    return has > least ? has : least;
}
uint32_t qmm_chain_limit(const QmmArgs &a, int sm_count) {
    TcChoice c;
    tc_choose(a, sm_count, false, c);
    return tc_chain_limit(a, c);
}

// The tile, of either kernel, with which a dense call takes least.  `limit`: what launch_qmm_tc is to be given with it.
uint32_t qmm_tc_pick_nt(int ggml_type, const QmmArgs &a, int sm_count, bool sharded, uint32_t *limit) {
    TcChoice c;
    tc_choose(a, sm_count, sharded, c);
    *limit = tc_chain_limit(a, c);
    if (!qmm_duo_takes(ggml_type, a)) return c.rows[c.best];
    uint32_t best = 256;
    uint64_t best_cost = ~0ull;
    for (uint32_t i = 0; i < c.count; i++)
        for (int duo = 0; duo < 2; duo++) {
            const uint32_t nt = duo ? (c.rows[i] + 31) / 32 * 32 : c.rows[i];
            const uint64_t cost = duo ? qmm_duo_cost(ggml_type, a, nt, *limit) : c.cost[i];
            if (best_cost == ~0ull || cost * 103 / 100 < best_cost) {
                best_cost = cost;
                best = nt;
            }
        }
    return best;
}

// Products of the same activations (and block type) as one launch on pairs of SMs: the tile, 0 where one of them does not go there, and
// the limit on its chains, the shortest of the products'.
uint32_t qmm_duo_pick_nt(int ggml_type, const QmmArgs *ops, int nops, int sm_count, uint32_t *limit) {
    QmmArgs all = ops[0];
    *limit = kChainAny;
    for (int i = 0; i < nops; i++) {
        if (!qmm_duo_takes(ggml_type, ops[i])) return 0;
        const uint32_t own = qmm_chain_limit(ops[i], sm_count);
        if (own < *limit) *limit = own;
        if (i) all.n = (all.n + 255) / 256 * 256 + ops[i].n;   // (as many weight tiles)
    }
    all.n = (all.n + 255) / 256 * 256;
    uint32_t best = 0;
    uint64_t best_cost = ~0ull;
    for (uint32_t tt = (all.m + 255) / 256, last = tt + 8; tt <= last; tt++) {
        const uint32_t nt = ((all.m + tt - 1) / tt + 31) / 32 * 32;
        const uint64_t cost = qmm_duo_cost(ggml_type, all, nt, *limit);
        if (cost != ~0ull && (best == 0 || cost * 103 / 100 < best_cost)) {
            best_cost = cost;
            best = nt;
        }
        if (nt == 32) break;
    }
    return best;
}

bool qmm_tc_supported(const QmmArgs &a) {
    if (a.k % 32 != 0 || a.k < 32) return false;
    if (((uintptr_t)a.w & 1u) || (a.expert_stride & 1u)) return false;
    return true;
}

template <int T, int NT, bool SH>
static cudaError_t launch_tc_tn(QmmArgs a, bool routed, uint32_t nt, uint8_t *scratch, cudaStream_t st, int *launches) {
    constexpr int QK = BlockTraits<T>::QK, BB = BlockTraits<T>::BYTES, KR = TcTraits<T>::KR;
    TcCfg c{};
    c.nt = nt;
    TcPlan plan;
    tc_plan(nt, a.m, a.n, a.k, (uint64_t)sm_count_of_device(), SH || routed, plan);
    {
        const char *dbg = exp_env("MLXN_TC_DEBUG");
        c.debug = dbg ? (uint32_t)atoi(dbg) : 0u;
    }
    {
        const uint32_t row_bytes = (a.k / QK) * BB;
        c.aligned = ((((uintptr_t)a.w | a.expert_stride) & 15u) == 0 && row_bytes % 16 == 0 && a.k % 256 == 0) ? 1u : 0u;
        if (exp_env("MLXN_TC_NO_ALIGNED")) c.aligned = 0;  // experiment switch
    }
    c.nchunks = (a.k + 63) / 64;
    c.seg_stride = round_up_u((KR / QK) * BB + 15, 16) + 16;
    if ((c.seg_stride / 16) % 2 == 0) c.seg_stride += 16;  // odd multiple of 16 B: rows spread over the banks
    // The weights arrive by tensor copies instead of 16-byte copies from every thread.  A copy has to start on a 16-byte boundary, which
    // every G-th row does (G = 1, 2, 4 or 8): the map's rows are groups of G weight rows, and a raw stage is G copies, each of one row
    // of every group.  The box is a stage's bytes of a row and the lead-in, an odd multiple of 16 (the rows' pitch in shared memory).
    // A 3-D map [expert][row group][words]; dense calls are one expert.  Needs n to be a multiple of G.
    alignas(64) CUtensorMap wmap;
    memset(&wmap, 0, sizeof(wmap));
    {
        EncodeTiledFn enc = encode_tiled_fn();
        const uint32_t row_bytes = (a.k / QK) * BB;
        uint32_t lg = 0;
        while ((row_bytes << lg) & 15u) lg++;
        constexpr uint32_t kSeg = (KR / QK) * BB;
        const uint32_t box_bytes = lg == 0 && kSeg % 16 == 0 ? kSeg : ((kSeg + 14 + 15) / 16 | 1u) * 16;
        const uint32_t n_exp = routed ? a.n_experts : 1u;
        const uint64_t estride = routed ? a.expert_stride : (uint64_t)a.n * row_bytes;
        const bool fits = (((uintptr_t)a.w | estride) & 15u) == 0 && a.n % (1u << lg) == 0 && (uint64_t)row_bytes * a.n <= estride;
        if (enc && n_exp >= 1 && fits && !exp_env("MLXN_TC_NO_TMA")) {
            const cuuint64_t gdim[3] = {((uint64_t)row_bytes << lg) / 4, a.n >> lg, n_exp};
            const cuuint64_t gstride[2] = {(uint64_t)row_bytes << lg, estride};
            const cuuint32_t box[3] = {box_bytes / 4, (cuuint32_t)(kTcRowsW >> lg), 1};
            const cuuint32_t estr[3] = {1, 1, 1};
            if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t *>(a.w), gdim, gstride, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS) {
                c.raw_tma = 1;
                c.row_group = lg;
                c.seg_stride = box_bytes;
            }
        }
    }
    const uint32_t b_bytes = nt * 128;  // one 64-wide K chunk of the activation tile
    const uint32_t raw_slot = kTcRowsW * c.seg_stride;
    uint32_t limit = 222 * 1024;   // + 1 KB alignment slack + 1 to 3 KB of static shared memory: 227 KB
    // narrow tiles stage their result in shared memory (two tiles of NT x 132 floats) and write whole output rows
    const uint32_t stage_bytes = 2u * NT * (kTcRowsW + 4) * 4u;
    // (the row-sharded form never shares tiles: they go straight to every rank's buffer)
    const bool staged = NT == 64 && !plan.shared &&
                        ((((uintptr_t)a.y) | ((uintptr_t)qmm_ld(a) * 4u) | ((uintptr_t)a.y_col0 * 4u)) & 15u) == 0 && a.n_peer == 0 &&
                        !exp_env("MLXN_TC_NO_STAGED_OUT");
    if (staged) limit -= stage_bytes;
    // activation ring first (at least two raw slots kept back), the rest goes to the raw weight ring
    uint32_t b_stages = (limit - 2 * raw_slot) / b_bytes;
    // (a 64-row tile's chunks are 8 KB: eight of them where four raw slots still fit beside them, the loop being
    // bound by how far the copies run ahead of the MMAs)
    const uint32_t b_cap = (NT == 64 && limit >= 8 * b_bytes + 4 * raw_slot) ? 8u : 6u;
    if (b_stages > b_cap) b_stages = b_cap;
    if (const char *e = exp_env("MLXN_TC_STAGES")) {  // experiment switch
        const uint32_t v = (uint32_t)atoi(e);
        if (v >= 4 && v <= b_stages) b_stages = v;
    }
    if (b_stages < 4) return cudaErrorInvalidConfiguration;   // (shallower rings are untested)
    uint32_t raw_slots = (limit - b_stages * b_bytes) / raw_slot;
    if (raw_slots > 6) raw_slots = 6;
    if (const char *e = exp_env("MLXN_TC_RAW")) {  // experiment switch
        const uint32_t v = (uint32_t)atoi(e);
        if (v >= 2 && v <= raw_slots) raw_slots = v;
    }
    const uint32_t raw_bytes = raw_slots * raw_slot;
    c.b_stages = b_stages;
    c.raw_slots = raw_slots;
    c.b_off = 0;
    c.raw_off = b_stages * b_bytes;
    if (staged) c.stage_off = c.raw_off + raw_bytes;
    const size_t smem = (size_t)c.raw_off + raw_bytes + (staged ? stage_bytes : 0u) + 1024;  // + slack for manual 1024-byte alignment

    size_t tiles;
    uint8_t *xpack = scratch;
    if (routed) {
        tiles = (size_t)a.total_rows / nt + a.n_experts;
        if (tiles > a.total_rows) tiles = a.total_rows;
        if (tiles == 0) tiles = 1;
        const size_t header = ((1 + 2 * tiles) * 4 + 1023) / 1024 * 1024;
        uint32_t *tl = reinterpret_cast<uint32_t *>(scratch);
        if (!(a.reuse & 1u)) {   // (an earlier call of the same layer built the list: same buckets, same NT)
            const cudaError_t e = launch_overlapped(build_tiles_kernel, dim3(1), dim3(256), 0, st, a.htpe, a.n_experts, nt, (uint32_t)tiles, tl);
            if (e != cudaSuccess) return e;
            (*launches)++;
        }
        a.tiles = tl;
        xpack = scratch + header;
    } else {
        tiles = (a.m + nt - 1) / nt;
        a.tiles = nullptr;
    }
    c.n_wt = (a.n + kTcRowsW - 1) / kTcRowsW;
    c.ntiles = (uint32_t)tiles;
    const uint32_t nraw = (a.k + KR - 1) / KR;
    if (plan.shared) c.share = {plan.ctas, c.n_wt, nraw, (uint32_t)(c.n_wt * tiles * nraw), kTcRowsW, nt};
    if (!(a.reuse & 2u)) {   // (... or packed the same activation rows already)
        // enough CTAs to fill the GPU a few times over, few enough that a tile's routing lookups are amortised
        uint32_t lanes = c.nchunks;
        const uint64_t slices = (uint64_t)tiles * ((nt + kPackRows - 1) / kPackRows);
        while (lanes > 1 && (uint64_t)lanes * slices > 2048) lanes = (lanes + 1) / 2;
        dim3 grid((unsigned)slices, lanes);
        (*launches)++;
        TcOut res{};
        res.y[0] = a.y;
        res.n[0] = a.n;
        res.wt_end[0] = c.n_wt;
        cudaError_t e = launch_overlapped(a.x2 ? pack_x_kernel<true> : pack_x_kernel<false>, grid, dim3(256), 0, st, a, xpack, c.nchunks, nt, c.share, res);
        if (e != cudaSuccess) return e;
    }
    if (routed && !SH && qmm_duo_routed_fits(T, a)) return launch_qmm_duo_routed(T, a, (uint32_t)tiles, xpack, st, launches);
    static size_t attr_smem[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (smem > attr_smem[dev]) {
        cudaError_t e = cudaFuncSetAttribute(qmm_tc_kernel<T, NT, SH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        attr_smem[dev] = smem;
    }
    // persistent CTAs, one per SM, each walking its items
    uint32_t ctas = plan.ctas;
    if (routed) {
        const uint64_t items = (uint64_t)c.n_wt * tiles;
        ctas = (uint32_t)sm_count_of_device();
        if (items < ctas) ctas = (uint32_t)items;
    }
    if (ctas == 0) return cudaSuccess;
    (*launches)++;
    note_mat_mat(routed ? "qmm_tc_id" : "qmm_tc", nt);
    return launch_overlapped(qmm_tc_kernel<T, NT, SH>, dim3(ctas), dim3(kTcThreads), smem, st, a, c, xpack, wmap);
}

template <int T> static cudaError_t launch_tc_t(const QmmArgs &a, bool routed, uint32_t nt, uint8_t *scratch, cudaStream_t st,
                                                int *launches) {
    if (nt == 0 || nt % 16 != 0 || nt > 256 || (routed && nt != kRoutedTile)) return cudaErrorInvalidValue;
    if (a.y_ld != 0 || a.n_peer != 0) {   // row-sharded result: the instantiation with the peer stores
        if (nt <= 64) return launch_tc_tn<T, 64, true>(a, routed, nt, scratch, st, launches);
        if (nt <= 128) return launch_tc_tn<T, 128, true>(a, routed, nt, scratch, st, launches);
        return launch_tc_tn<T, 256, true>(a, routed, nt, scratch, st, launches);
    }
    if (nt <= 64) return launch_tc_tn<T, 64, false>(a, routed, nt, scratch, st, launches);
    if (nt <= 128) return launch_tc_tn<T, 128, false>(a, routed, nt, scratch, st, launches);
    return launch_tc_tn<T, 256, false>(a, routed, nt, scratch, st, launches);
}

// tcgen05 mat-mat.  `scratch` must hold qmm_tc_scratch_bytes(a, nt, routed) bytes and start on a 256-byte boundary (the packed
// tiles in it are sources of bulk copies: 16-byte alignment is what the hardware needs; their offsets are multiples of 1024).
cudaError_t launch_qmm_tc(int ggml_type, const QmmArgs &a, bool routed, uint32_t nt, uint32_t limit, uint8_t *scratch, cudaStream_t st,
                          int *launches) {
    if (!routed) {
        TcPlan plan;
        if (qmm_duo_cost(ggml_type, a, nt, limit) < tc_plan(nt, a.m, a.n, a.k, (uint64_t)sm_count_of_device(), a.y_ld != 0 || a.n_peer != 0, plan))
            return launch_qmm_duo(ggml_type, &a, 1, nt, limit, scratch, st, launches);
    }
    switch (ggml_type) {
    case GT_Q4_0: return launch_tc_t<GT_Q4_0>(a, routed, nt, scratch, st, launches);
    case GT_Q8_0: return launch_tc_t<GT_Q8_0>(a, routed, nt, scratch, st, launches);
    case GT_Q6_K: return launch_tc_t<GT_Q6_K>(a, routed, nt, scratch, st, launches);
    case GT_Q4_K: return launch_tc_t<GT_Q4_K>(a, routed, nt, scratch, st, launches);
    default: return cudaErrorInvalidValue;
    }
}

template <int T> static cudaError_t launch_simt_t(const QmmArgs &a, bool routed, uint32_t max_rows, cudaStream_t st) {
    dim3 grid((max_rows + 63) / 64, (a.n + 63) / 64, routed ? a.n_experts : 1);
    qmm_simt_kernel<T><<<grid, 256, 0, st>>>(a);
    return cudaGetLastError();
}

// CUDA-core mat-mat.  max_rows: a.m (dense) or the largest possible rows per expert (routed).
cudaError_t launch_qmm_simt(int ggml_type, const QmmArgs &a, bool routed, uint32_t max_rows, cudaStream_t st) {
    switch (ggml_type) {
    case GT_Q4_0: return launch_simt_t<GT_Q4_0>(a, routed, max_rows, st);
    case GT_Q8_0: return launch_simt_t<GT_Q8_0>(a, routed, max_rows, st);
    case GT_Q6_K: return launch_simt_t<GT_Q6_K>(a, routed, max_rows, st);
    case GT_Q4_K: return launch_simt_t<GT_Q4_K>(a, routed, max_rows, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace mlxn

extern "C" const char *mlxn_debug_last_mat_mat(uint32_t *tile_rows) {
    if (tile_rows) *tile_rows = mlxn::t_mat_mat_rows;
    return mlxn::t_mat_mat;
}

// =================================================================================================
// mat-mat entry point that allocates nothing
// =================================================================================================
// Some callers may not allocate device memory at the moment they need a mat-mat: code running inside a
// memory-budgeted serving process whose allocator owns every byte of HBM, a real-time loop that must not
// hit the driver's allocation lock, or a plug-in that is only handed pointers.  For them the packed
// activation tiles of the tensor-core path live in this fixed array instead of the encoder's arena.
// Every GPU that loads the library carries the array until the process exits.
#include <cstdio>
#include <mutex>

#include "../../include/mlxn_b200.h"

int mlxn_detail_fail(int status, const char *msg);
void mlxn_detail_count_launches(int launches);

#define MLXN_NOALLOC_SCRATCH_BYTES (16u * 1024u * 1024u)
static __device__ __align__(256) uint8_t g_noalloc_scratch[MLXN_NOALLOC_SCRATCH_BYTES];

namespace {
std::mutex g_noalloc_mu;
uint8_t *g_noalloc_ptr[64] = {};  // device address of g_noalloc_scratch, per device ordinal
int g_noalloc_sms[64] = {};
}  // namespace

extern "C" size_t mlxn_noalloc_scratch_limit(void) { return MLXN_NOALLOC_SCRATCH_BYTES; }

extern "C" int mlxn_quantized_matmul_ggml_mm_noalloc(void *cuda_stream, const void *input_dev, const void *weight_dev,
                                                     void *output_dev, const mlxn_qmm_params *params) {
    using namespace mlxn;
    if (!input_dev || !weight_dev || !output_dev || !params)
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, "Invalid argument: pointers and params must not be null");
    const int t = (int)params->ggml_type;
    if (t != GT_Q4_0 && t != GT_Q8_0 && t != GT_Q6_K)
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, "Invalid argument: quantized_matmul_ggml_mm_noalloc supports Q4_0, Q8_0 and Q6_K only");
    if (params->m == 0 || params->k == 0 || params->n == 0)
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, "Invalid argument: M, K, and N must all be > 0");
    if (params->k % ggml_qk(t) != 0 || params->k % 32 != 0)
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, "Invalid argument: K must be divisible by the block QK and by 32");
    if (((uintptr_t)weight_dev & 1u) || ((uintptr_t)input_dev & 3u) || ((uintptr_t)output_dev & 3u))
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, "Invalid argument: weights must be 2-byte aligned, f32 buffers 4-byte aligned");
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return mlxn_detail_fail(MLXN_DEVICE_NOT_FOUND, "No usable current CUDA device for quantized_matmul_ggml_mm_noalloc");
#if CUDART_VERSION >= 12080
    {
        // the kernels are launched on the CURRENT device: a stream of another device would be refused by the launch with an
        // error that does not say why
        int sdev = -1;
        if (cudaStreamGetDevice(static_cast<cudaStream_t>(cuda_stream), &sdev) == cudaSuccess && sdev != dev) {
            char msg[160];
            snprintf(msg, sizeof(msg), "Invalid argument: quantized_matmul_ggml_mm_noalloc: the stream belongs to device %d but device %d is current",
                     sdev, dev);
            return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, msg);
        }
        cudaGetLastError();
    }
#endif
    uint8_t *scratch = nullptr;
    int sms = 0;
    {
        // first call on this device (with the device current): look up where the array lives on it.
        // The array's name is a host-side stand-in; only the address returned here may be given to a kernel.
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) {
                cudaGetLastError();
                return mlxn_detail_fail(MLXN_COMMAND_BUFFER_ERROR, "Command buffer error: cudaGetSymbolAddress failed for the static scratch array");
            }
            int n = 0;
            e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess || n <= 0) {
                cudaGetLastError();
                return mlxn_detail_fail(MLXN_COMMAND_BUFFER_ERROR, "Command buffer error: cannot query the SM count");
            }
            g_noalloc_sms[dev] = n;
            g_noalloc_ptr[dev] = static_cast<uint8_t *>(p);
        }
        scratch = g_noalloc_ptr[dev];
        sms = g_noalloc_sms[dev];
    }
    QmmArgs a{};
    a.w = static_cast<const uint8_t *>(weight_dev);
    a.x = static_cast<const float *>(input_dev);
    a.y = static_cast<float *>(output_dev);
    a.m = params->m;
    a.n = params->n;
    a.k = params->k;
    a.top_k = 1;
    a.n_experts = 1;
    a.total_rows = params->m;
    a.status = nullptr;  // no status word: a wait that gives up still ends the kernel, but is not reported
    uint32_t limit = 0, nt = qmm_tc_pick_nt(t, a, sms, false, &limit);
    size_t need = qmm_tc_scratch_bytes(a, nt, false);
    // (the fastest tile may pad the rows more than another one that still fits; tiles of 16 rows pad least)
    for (uint32_t other = 256; other >= 16 && need > MLXN_NOALLOC_SCRATCH_BYTES; other -= 16) need = qmm_tc_scratch_bytes(a, nt = other, false);
    if (need > MLXN_NOALLOC_SCRATCH_BYTES) {
        char msg[256];
        snprintf(msg, sizeof(msg),
                 "Invalid argument: quantized_matmul_ggml_mm_noalloc needs %zu bytes of packed activations for m=%u k=%u, "
                 "the static scratch holds %u (about m*k <= 8M elements); use quantized_matmul_ggml instead",
                 need, a.m, a.k, MLXN_NOALLOC_SCRATCH_BYTES);
        return mlxn_detail_fail(MLXN_INVALID_ARGUMENT, msg);
    }
    int launches = 0;
    cudaError_t e = launch_qmm_tc(t, a, false, nt, limit, scratch, static_cast<cudaStream_t>(cuda_stream), &launches);
    if (e != cudaSuccess) {
        cudaGetLastError();
        char msg[256];
        snprintf(msg, sizeof(msg), "Command buffer error: mat-mat launch: %s", cudaGetErrorString(e));
        return mlxn_detail_fail(MLXN_COMMAND_BUFFER_ERROR, msg);
    }
    mlxn_detail_count_launches(launches);
    return MLXN_OK;
}
