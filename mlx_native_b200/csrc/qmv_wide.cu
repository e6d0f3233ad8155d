// Q4_K products of many activation rows: y[m, n] = x[m, k] . W[n, k]^T, m > 8.
//
// Upstream has no dense mat-mat for Q4_K and takes the mat-vec at any m (src/ops/quantized_matmul_ggml.rs:350-360), so results
// are 32-bit sums of exact products here too: codes as integers in f16, activations as f16 hi + lo halves, scales outside the multiply.
// That is the arithmetic of qmv_split.cuh, whose kernel unpacks the weights again for every eight rows (96 rows of 4096 x 4096: 12
// passes, 110 us).  Here
//
//  * a CTA takes 128 or 256 weight rows and 16 to 48 activation rows, K in stages of a super-block of 256: one tensor copy of the raw
//    blocks, one bulk copy each of the packed activations and of their sums (written by qmv_pack_kernel);
//  * a warp unpacks two 16-row tiles once per 32 values (a third of its instructions) for all its sets of eight activation rows: the
//    columns of an MMA, multiplied with their hi and their lo halves;
//  * K may be split over a cluster: 4096 x 4096 with 9 rows has 32 tiles for 148 SMs.  The ranks' sums are added in rank order through
//    distributed shared memory: no atomics, results are bit-reproducible.
//
// Graph replay of dependent calls, packing included, us before / now: 9 rows of 4096 x 4096 26 / 14, 32 43 / 19, 96 111 / 37, 512 547 / 152,
// 2048 2166 / 571; 16 rows of 12288 x 4096 57 / 32, 100 of 256 x 4096 17 / 11.  What bounds it: mma.sync (2 cycles on an SM per 16 x 8 x 16) is
// busy for 40 % of the time, instruction issue for 44 % (96 rows); the rest is waiting of one on the other.  Relative error against 64 bits (K 1024 ..
// 14336) 0.9..1.1e-7, the other kernel's 0.9..1.2e-7; with hi and lo summed by one chain of multiplies it was 1.0..1.2e-7 (35 us).
#include "qmv_split.cuh"

namespace mlxn {

constexpr int kWdOps = 8;
constexpr uint32_t kWdSuper = 144;                   // bytes of a super-block
constexpr uint32_t kWdStages = 2;

struct WdOp {
    const uint8_t *w;
    const float *x;
    float *y;
    const uint8_t *xp;        // packed activations [super-block][row][1024 bytes], see qmv_pack_kernel
    const float *xsum, *xinv; // [super-block][row][8], [row]
    uint32_t n, k;
    uint32_t tile_end;        // tiles of the ops up to and including this one
};
struct WdArgs {
    WdOp op[kWdOps];
    uint32_t nops, m;
    uint32_t m_pad;           // rows of the packed arrays
    uint32_t early_weights;
    uint32_t *status;
};

// The scales d sc and the offsets 8 d sc - dmin m (codes are taken less 8) of a unit's two sub-blocks, each twice: operands of packed
// arithmetic.  rb: the row's super-block (the 6-bit fields as in src/gguf/mod.rs:440-452).
__device__ __forceinline__ void wd_table_row(uint32_t dst, uint32_t rb, uint32_t u) {
    uint32_t dd, s0, s1, s2;
    lds128(rb, dd, s0, s1, s2);
    const float d = f16lo_to_float(dd), dmin = f16hi_to_float(dd);
    const uint32_t sh = 16u * (u & 1u);
    const uint32_t a = s0 >> sh, b = s1 >> sh, c = s2 >> sh;
    uint32_t sc, mn;   // two fields each, a byte apart
    if (u < 2) {
        sc = a & 0x3F3Fu;
        mn = b & 0x3F3Fu;
    } else {
        sc = (c & 0x0F0Fu) | ((a >> 2) & 0x3030u);
        mn = ((c >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u);
    }
    const float e0 = d * (float)(sc & 255u), e1 = d * (float)((sc >> 8) & 255u);   // (17 bits: exact, as the products with the minima)
    const float o0 = fmaf(8.f, e0, -(dmin * (float)(mn & 255u))), o1 = fmaf(8.f, e1, -(dmin * (float)((mn >> 8) & 255u)));
    auto put = [](uint32_t at, float e, float o) { sts128(at, __float_as_uint(e), __float_as_uint(e), __float_as_uint(o), __float_as_uint(o)); };
    put(dst, e0, o0);
    put(dst + 16, e1, o1);
}

// RG row groups of 32 weight rows x two column groups of S sets of eight activation rows, a warp each.
template <int RG, int S> struct WdShape {
    static constexpr uint32_t threads = RG * 64, rows = RG * 32, cols = S * 16;
    static constexpr uint32_t xoff = rows * kWdSuper, soff = xoff + cols * 1024, stage = soff + cols * 32, tab = kWdStages * stage;
    static constexpr uint32_t pitch = rows + 4;      // floats of a result column in shared memory
    static constexpr uint32_t smem = 128 + tab + RG * 2 * 1024;
    static_assert(cols * pitch * 4 <= tab, "the tile's sums take the place of the stages");
};

template <int RG, int S>
__global__ void __launch_bounds__(WdShape<RG, S>::threads, RG == 4 ? 2 : 1) qmv_wide_kernel(const __grid_constant__ WdArgs A, const __grid_constant__ SpMaps maps) {
    using H = WdShape<RG, S>;
    constexpr uint32_t WARPS = RG * 2, BN = H::cols;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;   // (the same in every CTA of a cluster)
    __shared__ __align__(8) uint64_t full[kWdStages];
    __shared__ uint32_t readers[kWdStages];
    __shared__ volatile uint32_t abort_flag;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t ranks;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    const uint32_t rank = sp::cluster_rank();
    if (tid == 0) {
        abort_flag = 0;
        for (uint32_t s = 0; s < kWdStages; s++) {
            mbar_init(&full[s], 1);
            readers[s] = 0;
        }
        mbar_init_fence();
    }
    __syncthreads();
    allow_dependents();
    // the cluster's tile: activation tiles of one weight tile are neighbours, so that its blocks come from HBM but once
    const uint32_t at = blockIdx.x / ranks;
    uint32_t op = 0;
    while (at >= A.op[op].tile_end) op++;
    const WdOp &P = A.op[op];
    const uint32_t tile = at - (op ? A.op[op - 1].tile_end : 0u), ncol = (A.m + BN - 1) / BN;
    const uint32_t n0 = tile / ncol * H::rows, c0 = tile % ncol * BN;
    const uint32_t nsb = P.k / 256u, sb0 = nsb * rank / ranks, mine = nsb * (rank + 1) / ranks - sb0;

    auto weights = [&](uint32_t i) {   // stage i of the CTA's share of K
        const uint32_t s = i % kWdStages;
        mbar_expect_tx(&full[s], H::stage);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(base + s * H::stage),
                     "l"(&maps.m[op]), "r"((sb0 + i) * (kWdSuper / 4u)), "r"(n0), "r"(smem_u32(&full[s]))
                     : "memory");
    };
    auto rows = [&](uint32_t i) {
        const uint32_t s = i % kWdStages;
        const size_t r = (size_t)(sb0 + i) * A.m_pad + c0;
        bulk_g2s_a(base + s * H::stage + H::xoff, P.xp + r * 1024u, BN * 1024u, &full[s]);
        bulk_g2s_a(base + s * H::stage + H::soff, P.xsum + r * 8u, BN * 32u, &full[s]);
    };
    if (tid == 0) {
        if (!A.early_weights) grid_dependency_wait();
        for (uint32_t i = 0; i < min(kWdStages, mine); i++) weights(i);
        grid_dependency_wait();   // the packed activations are the kernel's ahead
        for (uint32_t i = 0; i < min(kWdStages, mine); i++) rows(i);
    }
    __syncwarp();

    const uint32_t g = lane >> 2, t = lane & 3u, wr = warp % RG, wc = warp / RG;
    // [tile][set][weight row g, g + 8]: sums for the activation rows 2t, 2t + 1; `acc` over a super-block, `sum` over all of them: short
    // chains of additions (one chain over K = 4096 had an error of 2.6e-7 against 64 bits, chains of 8 and 16 have 1.0e-7)
    uint64_t acc[2][S][2], sum[2][S][2];
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int v = 0; v < S; v++) acc[j][v][0] = acc[j][v][1] = sum[j][v][0] = sum[j][v][1] = 0ull;
    const uint32_t tab = base + H::tab + warp * 1024u, tr = tab + g * 32u;
    uint32_t s = 0, ph = 0;
    for (uint32_t i = 0; i < mine; i++) {
        if (!mbar_wait(&full[s], ph, &abort_flag, A.status, ST_WAIT_FULL_TIMEOUT, 0u)) break;
        const uint32_t st = base + s * H::stage, wrow = st + wr * 32u * kWdSuper;
        const uint32_t q0 = wrow + g * kWdSuper + 16u + 4u * t;
        const uint32_t xa = st + H::xoff + (wc * S * 8u + g) * 1024u + t * 32u + (g & 1u) * 16u, xl = xa ^ 16u;   // hi, lo
        const uint32_t ca = st + H::soff + wc * S * 256u + t * 8u;
#pragma unroll 1
        for (uint32_t u = 0; u < 4; u++) {
            __syncwarp();   // the table of the unit before has been read
            wd_table_row(tab + lane * 32u, wrow + lane * kWdSuper, u);
            uint32_t x[2][4];   // [tile]: the unit's code bytes of rows g and g + 8, first and second 16
            static_for<0, 2>([&](auto J) {
                constexpr int j = decltype(J)::value;
                constexpr uint32_t o = j * 16u * kWdSuper, o8 = o + 8u * kWdSuper;
                const uint32_t qa = q0 + 32u * u;
                x[j][0] = lds32i<o>(qa); x[j][1] = lds32i<o8>(qa);
                x[j][2] = lds32i<o + 16>(qa); x[j][3] = lds32i<o8 + 16>(qa);
            });
            __syncwarp();
            static_for<0, 2>([&](auto HALF) {   // a sub-block: the low or the high nibbles
                constexpr uint32_t hf = decltype(HALF)::value;
                uint32_t a[2][2][4], p[2][2][4];   // [tile]: codes; scale and offset, twice each, of rows g and g + 8
                static_for<0, 2>([&](auto J) {
                    constexpr int j = decltype(J)::value;
                    lds128i<j * 512u + hf * 16u>(tr, p[j][0]);
                    lds128i<j * 512u + 256u + hf * 16u>(tr, p[j][1]);
#pragma unroll
                    for (int e = 0; e < 2; e++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint32_t z = x[j][2 * e + h], y = z >> 8;
                            a[j][e][h] = hf ? sp::hi4(z) : sp::lo4(z);
                            a[j][e][h + 2] = hf ? sp::hi4(y) : sp::lo4(y);
                        }
                });
                static_for<0, S>([&](auto V) {
                    constexpr int v = decltype(V)::value;
                    constexpr float zero[4] = {0.f, 0.f, 0.f, 0.f};
                    uint32_t bh[4], bl[4], c[2];
                    lds128i<v * 8192u + hf * 128u>(xa + u * 256u, bh);
                    lds128i<v * 8192u + hf * 128u>(xl + u * 256u, bl);
                    lds64i<v * 256u + hf * 32u>(ca + u * 64u, c[0], c[1]);
                    const uint64_t cc = pack2u(c[0], c[1]);
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        float r[4], l[4];   // products with the hi and with the lo halves
                        mma16816(r, a[j][0][0], a[j][0][1], a[j][0][2], a[j][0][3], bh[0], bh[1], zero);
                        mma16816(l, a[j][0][0], a[j][0][1], a[j][0][2], a[j][0][3], bl[0], bl[1], zero);
                        mma16816(r, a[j][1][0], a[j][1][1], a[j][1][2], a[j][1][3], bh[2], bh[3], r);
                        mma16816(l, a[j][1][0], a[j][1][1], a[j][1][2], a[j][1][3], bl[2], bl[3], l);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint32_t(&f)[4] = p[j][h];
                            uint64_t z = ffma2(pack2u(f[0], f[1]), pack2(l[2 * h], l[2 * h + 1]), fmul2(pack2u(f[2], f[3]), cc));
                            z = ffma2(pack2u(f[0], f[1]), pack2(r[2 * h], r[2 * h + 1]), z);
                            acc[j][v][h] = fadd2(acc[j][v][h], z);
                        }
                    }
                });
            });
        }
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int v = 0; v < S; v++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    sum[j][v][h] = fadd2(sum[j][v][h], acc[j][v][h]);
                    acc[j][v][h] = 0ull;
                }
        __syncwarp();
        if (lane == 0) {   // the last of the warps to have read a stage asks for the one that takes its place
            __threadfence_block();
            if ((atomicAdd(&readers[s], 1u) & (WARPS - 1u)) == WARPS - 1u && i + kWdStages < mine) {
                __threadfence_block();
                weights(i + kWdStages);
                rows(i + kWdStages);
            }
        }
        __syncwarp();
        if (++s == kWdStages) {
            s = 0;
            ph ^= 1u;
        }
    }
    __syncwarp();
    if (abort_flag)   // let copies in flight land before anything else is written there
        for (int i = 0; i < 200; i++) __nanosleep(5000);
    __syncthreads();      // the stages have been read
    const uint32_t d = base + ((wc * S * 8u + 2u * t) * H::pitch + wr * 32u + g) * 4u;
    static_for<0, S>([&](auto V) {
        constexpr uint32_t v = decltype(V)::value, o = v * 32u * H::pitch;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float lo, hi;
                unpack2(sum[j][v][h], lo, hi);
                sts32(d + o + j * 64u + h * 32u, __float_as_uint(lo));
                sts32(d + o + H::pitch * 4u + j * 64u + h * 32u, __float_as_uint(hi));
            }
    });
    if (ranks > 1) sp::cluster_sync();
    else __syncthreads();
    grid_dependency_wait();   // (all threads: y may be what the kernels ahead still read)
    // every rank finishes its share of the columns, four rows a thread
    const uint32_t share = BN / ranks, lo = rank * share;
    for (uint32_t q = tid; q < share * (H::rows / 4u); q += H::threads) {
        const uint32_t col = lo + q / (H::rows / 4u), row = q % (H::rows / 4u) * 4u, out = c0 + col;
        if (out >= A.m || n0 + row >= P.n) continue;
        const uint32_t a = base + (col * H::pitch + row) * 4u;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (uint32_t r = 0; r < ranks; r++) {
            float z[4];
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(z[0]), "=f"(z[1]), "=f"(z[2]), "=f"(z[3]) : "r"(sp::map_rank(a, r)));
#pragma unroll
            for (int e = 0; e < 4; e++) v[e] += z[e];
        }
        const float inv = __ldcg(P.xinv + out);
        float *y = P.y + (size_t)out * P.n + n0 + row;
        const uint32_t cnt = min(4u, P.n - n0 - row);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            v[e] *= inv;
            // (an infinite activation times codes and offset may cancel where the weight has a sign: formed again, weight by weight)
            if (v[e] != v[e] && e < (int)cnt)
                v[e] = sp_again<GT_Q4_K>(P.w + (size_t)(n0 + row + e) * (nsb * kWdSuper), P.x + (size_t)out * P.k, P.k, 0, 1);
        }
        if (cnt == 4 && ((uintptr_t)y & 15u) == 0) {
            *reinterpret_cast<float4 *>(y) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (e < (int)cnt) y[e] = v[e];
        }
    }
    // nobody leaves while a peer may still read here
    if (ranks > 1) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
struct WdPick {
    uint32_t shape, ranks;   // 0: 128 x 16, 1: 128 x 32, 2: 256 x 48
};
static constexpr uint32_t kWdShapeRows[3] = {128, 128, 256}, kWdShapeCols[3] = {16, 32, 48};
static uint64_t wd_tiles(uint32_t shape, uint32_t m, uint32_t n) {
    return (uint64_t)((n + kWdShapeRows[shape] - 1) / kWdShapeRows[shape]) * ((m + kWdShapeCols[shape] - 1) / kWdShapeCols[shape]);
}
// Time of a geometry: the CTAs of the fullest SM, one after another, times their stages and what a CTA costs beside them.  Measured
// (K = 4096 in one, two, four and eight parts, 9 to 2048 rows): a stage of 128 x 16 takes 1.9 us on an SM of its own and 1.6 where two
// share it, 128 x 32 2.6 and 2.4, 256 x 48 (three times the work) 6.1.  One to eight parts, us, 96 rows of 4096 x 4096: 128 x 16 57 / 47 / 51
// / 62, 128 x 32 47 / 43 / 42 / 45, 256 x 48 104 / 57 / 35 / 61; 9 rows 35 / 21 / 14 / 13, 46 / 27 / 17 / 16, 102 / 56 / 32 / 38; 2048 rows in one
// part 717, 510, 522.
static WdPick wd_pick(const QmvArgs *ops, int nops, int sm_count) {
    WdPick best{1, 1};
    static const double alone[3] = {1.9, 2.6, 6.1}, shared[3] = {1.62, 2.37, 6.1};
    static const double beside[3][4] = {{0.0, 0.5, 1.1, 1.7}, {0.0, 0.4, 1.3, 2.1}, {6.0, 6.0, 6.5, 7.0}};
    double least = 1e30;
    uint32_t sb = 1;
    for (int i = 0; i < nops; i++) sb = ops[i].k / 256 > sb ? ops[i].k / 256 : sb;
    for (uint32_t s = 0; s < 3; s++)
        for (uint32_t l = 0; l < 4 && (1u << l) <= sb; l++) {
            uint64_t ctas = 0;
            for (int i = 0; i < nops; i++) ctas += wd_tiles(s, ops[0].m, ops[i].n) << l;
            const uint64_t per = (ctas + sm_count - 1) / sm_count;
            const double cost = (double)per * ((sb + (1u << l) - 1) / (1u << l) * (per > 1 ? shared[s] : alone[s]) + beside[s][l]);
            if (cost < least) {
                least = cost;
                best = {s, 1u << l};
            }
        }
    return best;
}

// Sizes and addresses that the kernel takes: dense Q4_K, every row on a 16-byte boundary.
bool qmv_wide_supported(int ggml_type, const QmvArgs &a) {
    if (ggml_type != GT_Q4_K || a.ids || a.x2 || a.y_ld || a.n_peer) return false;
    if (a.m == 0 || a.n == 0 || a.k == 0 || a.k % 256 != 0) return false;
    if (((uintptr_t)a.x & 7u) || ((uintptr_t)a.w & 15u)) return false;
    if ((uint64_t)a.k / 256 * kWdSuper >= (1ull << 31) || (uint64_t)a.m * a.k >= (1ull << 31)) return false;
    if (((uint64_t)a.m + 15) / 16 * ((a.n + 127) / 128) * 8 >= (1ull << 31)) return false;
    return encode_tiled_fn() != nullptr;
}
// Below 256 x 4096 there are a handful of tiles, and a launch is all latency with either kernel.
bool qmv_wide_pays(const QmvArgs &a) { return (uint64_t)a.n * a.k >= 1u << 20; }

static uint32_t wd_pad(uint32_t m) { return (m + 95) / 96 * 96; }   // (whole tiles)
static size_t wd_pack_bytes(uint32_t m, uint32_t k) {
    const size_t sb = k / 256, rows = wd_pad(m);
    return (sb * rows * (1024 + 32) + rows * 4 + 255) / 256 * 256;
}
size_t qmv_wide_scratch_bytes(const QmvArgs *ops, int nops) {
    size_t n = 0;
    for (int i = 0; i < nops; i++) n += wd_pack_bytes(ops[i].m, ops[i].k);
    return n;
}

template <int RG, int S> static cudaError_t wd_launch(const WdArgs &A, const SpMaps &maps, uint32_t ranks, uint32_t clusters, int sm_count, cudaStream_t st) {
    using H = WdShape<RG, S>;
    auto kernel = qmv_wide_kernel<RG, S>;
    // Where every CTA can have an SM of its own it has to ask for more than half of the shared memory: the blocks of the packing kernel
    // are still there when CTAs are placed, and these then shared the SMs that were left (96 CTAs: 88 us instead of 57).
    constexpr uint32_t alone = 120 * 1024;
    const uint32_t smem = RG == 4 && clusters * ranks <= (uint32_t)sm_count ? alone : H::smem;
    static std::atomic<uint32_t> prepared[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(RG == 4 ? alone : H::smem));
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
    cfg.gridDim = dim3(clusters * ranks);
    cfg.blockDim = dim3(H::threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, A, maps);
}

// `ops`: dense products of the same number of rows.
cudaError_t launch_qmv_wide(const QmvArgs *ops, int nops, int sm_count, uint8_t *scratch, int *launches, cudaStream_t st) {
    if (nops < 1 || nops > kWdOps) return cudaErrorInvalidValue;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return cudaErrorNotSupported;
    static thread_local SpBatch pk;
    static thread_local WdArgs A;
    alignas(64) static thread_local SpMaps maps;
    A.nops = (uint32_t)nops;
    A.m = ops[0].m;
    A.m_pad = wd_pad(A.m);
    A.status = ops[0].status;
    A.early_weights = 1;
    pk.nops = (uint32_t)nops;
    const WdPick pick = wd_pick(ops, nops, sm_count);
    uint32_t rows = 0;
    for (int i = 0; i < nops; i++) {
        const QmvArgs &a = ops[i];
        WdOp &P = A.op[i];
        SpOp &Q = pk.op[i];
        P.w = a.w;
        P.x = Q.x = a.x;
        P.y = a.y;
        P.n = a.n;
        P.k = Q.k = a.k;
        if (!a.early_weights) A.early_weights = 0;
        int same = -1;
        for (int q = 0; q < i && same < 0; q++)
            if (ops[q].x == a.x && ops[q].k == a.k) same = q;
        if (same >= 0) {
            P.xp = A.op[same].xp;
            P.xsum = A.op[same].xsum;
            P.xinv = A.op[same].xinv;
        } else {
            const size_t n = (size_t)(a.k / 256) * A.m_pad;
            P.xp = scratch;
            P.xsum = reinterpret_cast<const float *>(scratch + n * 1024);
            P.xinv = P.xsum + n * 8;
            scratch += wd_pack_bytes(a.m, a.k);
            rows += A.m;
        }
        Q.xp = P.xp;
        Q.xsum = P.xsum;
        Q.xinv = P.xinv;
        Q.units = Q.pk_units = a.k / 64;
        Q.row_end = rows;
        Q.xp_row = 1024;
        Q.xp_super = (uint64_t)A.m_pad * 1024;
        Q.wide_rows = A.m_pad;
        const cuuint64_t dim[2] = {a.k / 256 * (kWdSuper / 4), a.n}, stride[1] = {a.k / 256 * kWdSuper};
        const cuuint32_t box[2] = {kWdSuper / 4, kWdShapeRows[pick.shape]}, one[2] = {1, 1};
        if (enc(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t *>(a.w), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    uint32_t clusters = 0;
    for (int i = 0; i < nops; i++) A.op[i].tile_end = clusters += (uint32_t)wd_tiles(pick.shape, A.m, A.op[i].n);
    cudaError_t e = launch_overlapped(qmv_pack_kernel<GT_Q4_K, true>, dim3(rows), dim3(256), 0, st, pk);
    if (e != cudaSuccess) return e;
    *launches = 2;
    switch (pick.shape) {
    case 0: return wd_launch<4, 1>(A, maps, pick.ranks, clusters, sm_count, st);
    case 1: return wd_launch<4, 2>(A, maps, pick.ranks, clusters, sm_count, st);
    default: return wd_launch<8, 3>(A, maps, pick.ranks, clusters, sm_count, st);
    }
}

}  // namespace mlxn
