// Sigmoid attention with mixed heads over a portion of a prompt, on the tensor cores, in one of two ways (gate_flash_pays): one
// head at a time, mixed in the outputs (gate_flash_kernel, gate_mix_kernel), or all heads of a pair at once, as follows.
//
// Mixing couples every head at every (query, key) pair, so a CTA owns a tile of 128 queries x BN keys for
// ALL heads: each head's scores land in their own TMEM columns (heads x BN <= 512), then a thread reads
// one query row's scores of all heads for four keys at a time, forms the sigmoids in fp32, and the mixed
// weights are written as bf16.  Up to 8 heads are mixed in registers (packed fma.rn.f32x2).  With more
// heads the mixing is a small product per key, mix[h][query] = sum_g T[h][g] w[g][query]: T is bf16 as
// stored, and the fp32 weights go in as two bf16 parts, high and low (16 bits of mantissa together), in
// two rounds of mma.sync over the same accumulator; their operand layout is what the TMEM rows give
// after one pass through shared memory.  The product with the raw keys is a
// batched gemm_tc over heads (its causal bound skips the zero part), against keys transposed once per
// call.  Queries go in blocks, so that the weights of a block stay within the workspace.
#include <algorithm>

#include "gemm_tc.h"
#include "layered_ops.cuh"
#include "umma.cuh"

namespace mg {

namespace {

constexpr int kThreads = 320;       // TMA warp, MMA warp, 8 epilogue warps

struct ScoreArgs {
    CUtensorMap q, k;               // [rows][heads][dim_s] in boxes of 128 rows; [max_seq][kv][dim_s] in boxes of BN rows
    GateAttn at;
    int row0, rows, pos0;           // queries [row0, row0 + rows) of the portion, at positions pos0 + row
    int ldp;                        // columns of a weight row (a multiple of 64)
    long long head_stride;          // elements between heads of the weights
    __nv_bfloat16* w;               // [heads][.][ldp]
    int* status;
};

template <int HP>
struct Geo {
    static constexpr bool tensor_mix = HP >= 16;
    static constexpr int bn = HP <= 8 ? 32 : 16;
    static constexpr int cols = HP * bn < 32 ? 32 : HP * bn;
    static constexpr int per_sm = cols <= 256 ? 2 : 1;
    static constexpr int stages = HP == 32 ? 8 : HP == 16 ? 5 : 4;
    static constexpr int stage = 128 * 128 + bn * 128;
    static constexpr int ring = stages * stage;
    // the epilogue's operand rows take the ring's place: per warp 4 keys x 32 queries x {high, low}
    static constexpr int point = HP * 2 + 16;               // bytes of a row of bf16 weights, padded against conflicts
    static constexpr int part = 4 * 32 * point;
    static constexpr int mix_bytes = tensor_mix ? 8 * 2 * part : 0;
    static constexpr int body = ring > mix_bytes ? ring : mix_bytes;
    static constexpr int talk_bytes = tensor_mix ? 0 : 8 * HP * HP;    // mixing pairs {t, t}
    static constexpr int bytes = body + 1024 + 256 + talk_bytes + (2 * HP + bn * HP) * 4;
};

// 1 / (1 + 2^t)
__device__ __forceinline__ float sigmoid_of_exp2(float t) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return r;
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&p);
}

template <int HP>
__global__ void __launch_bounds__(kThreads, Geo<HP>::per_sm) gate_scores_kernel(const __grid_constant__ ScoreArgs a) {
    pdl_wait();
    using G = Geo<HP>;
    constexpr int BN = G::bn, kStages = G::stages;
    const GateAttn& A = a.at;
    const int tile_row = blockIdx.y * 128, j0 = blockIdx.x * BN;
    const int tile_rows = min(128, a.rows - tile_row);
    // the product reads whole steps of 64 columns up to the last query of the row tile
    if (j0 >= pad_to(a.pos0 + a.row0 + tile_row + tile_rows, 64)) return;

    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + G::body);
    uint64_t* empty = full + kStages;
    uint64_t* done = empty + kStages;
    uint32_t* tmem_base = reinterpret_cast<uint32_t*>(done + 1);
    ulonglong2* talk = reinterpret_cast<ulonglong2*>(base + G::body + 256);     // [h][g / 2]: {t, t} of two g
    float2* line = reinterpret_cast<float2*>(base + G::body + 256 + G::talk_bytes);  // per head: slope, -bias, in units of log2 e
    float* kr = reinterpret_cast<float*>(line + HP);                            // [head][key]: -1 / rms of the key, likewise
    static_assert((2 * kStages + 1) * 8 + 4 <= 256, "barriers fit their place");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int H = A.heads, group = H / A.kv_heads;
    const int kb = (A.dim_s + 63) / 64, steps = H * kb;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; i++) { bar_init(full + i, 1); bar_init(empty + i, 1); }
        bar_init(done, 1);
        bar_init_fence();
        tma_prefetch_map(&a.q);
        tma_prefetch_map(&a.k);
    }
    if (warp == 1) tmem_alloc(tmem_base, G::cols);
    constexpr float kLog2e = 1.4426950408889634f;
    if constexpr (!G::tensor_mix) {
        for (int i = threadIdx.x; i < HP * HP / 2; i += kThreads) {
            const int h = i / (HP / 2), g = 2 * (i % (HP / 2));
            const float t0 = h < H && g < H ? A.talk[h * H + g] : 0.f, t1 = h < H && g + 1 < H ? A.talk[h * H + g + 1] : 0.f;
            talk[i] = make_ulonglong2(pack2(t0, t0), pack2(t1, t1));
        }
    }
    for (int i = threadIdx.x; i < HP; i += kThreads)
        line[i] = i < H ? make_float2(A.slopes[i] * kLog2e, -A.head_bias[i] * kLog2e) : make_float2(0.f, 0.f);
    const int len = a.pos0 + a.row0 + a.rows;       // keys the block's queries can see
    for (int i = threadIdx.x; i < BN * HP; i += kThreads) {
        const int p = i % BN, h = i / BN;
        kr[i] = h < H && j0 + p < len ? -kLog2e * A.cache_r[(size_t)(j0 + p) * A.kv_heads + h / group] : 0.f;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t acc = *tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < steps; i++) {
                const int s = i % kStages, use = i / kStages, h = i / kb, x = (i - h * kb) * 64;
                if (use > 0 && !bar_wait(empty + s, (use - 1) & 1, a.status)) break;
                bar_expect(full + s, G::stage);
                uint8_t* st = base + s * G::stage;
                tma_load_3d(st, &a.q, x, h, a.row0 + tile_row, full + s);
                tma_load_3d(st + 128 * 128, &a.k, x, h / group, j0, full + s);
                issued = i + 1;
            }
            for (int i = max(0, issued - kStages); i < issued; i++) bar_wait(full + i % kStages, (i / kStages) & 1, a.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            for (int i = 0; i < steps; i++) {
                const int s = i % kStages, h = i / kb;
                if (!bar_wait(full + s, (i / kStages) & 1, a.status)) break;
                tc_fence_after();
                const uint64_t da = tile_desc(base + s * G::stage), db = tile_desc(base + s * G::stage + 128 * 128);
#pragma unroll
                for (int k = 0; k < 4; k++) mma_bf16(acc + h * BN, da + 2 * k, db + 2 * k, mma_desc(BN), i > h * kb || k > 0);
                mma_commit(empty + s);
            }
            mma_commit(done);
        }
        __syncwarp();
    } else {
        // mixing matrix as MMA operands: rows h, columns g
        constexpr int MT = HP >= 16 ? HP / 16 : 1;
        uint32_t ta[MT][MT][4];
        if constexpr (G::tensor_mix) {
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int k = 0; k < MT; k++)
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int h = m * 16 + (lane >> 2) + (r & 1) * 8, g = k * 16 + (lane & 3) * 2 + (r >> 1) * 8;
                        ta[m][k][r] = bf16_pair(h < H && g < H ? A.talk[h * H + g] : 0.f, h < H && g + 1 < H ? A.talk[h * H + g + 1] : 0.f);
                    }
        }
        const bool ok = __all_sync(0xffffffffu, bar_wait(done, 0, a.status));
        tc_fence_after();
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const int row = tile_row + quarter * 32 + lane;
        const int pos = a.pos0 + a.row0 + row;
        uint8_t* mine = base + (warp - 2) * 2 * G::part;
        if (ok) {
#pragma unroll 1
            for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 4) {
                constexpr int GB = HP < 8 ? HP : 8;         // heads per round of loads
                unsigned long long w[G::tensor_mix ? 1 : HP][2];
                const float dist = (float)(pos - (j0 + c));
#pragma unroll
                for (int g0 = 0; g0 < HP; g0 += GB) {
                    uint32_t s[GB][4];
                    float v[GB][4];
#pragma unroll
                    for (int g = 0; g < GB; g++)
                        if (g0 + g < H) tmem_load4_async(acc + ((uint32_t)(quarter * 32) << 16) + (g0 + g) * BN + c, s[g]);
                    tmem_wait_load();
#pragma unroll
                    for (int g = 0; g < GB; g++) {
                        const float2 ln = line[g0 + g];
                        const float4 k4 = *reinterpret_cast<const float4*>(kr + (g0 + g) * BN + c);
                        const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float t = fmaf(__uint_as_float(s[g][i]), kk[i], fmaf(ln.x, dist - (float)i, ln.y));
                            v[g][i] = g0 + g < H && dist >= (float)i ? sigmoid_of_exp2(t) : 0.f;
                        }
                    }
                    if constexpr (G::tensor_mix) {
                        // eight heads are 16 bytes of a point's row, as bf16 and what bf16 leaves over
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            uint32_t hi4[4], lo4[4];
#pragma unroll
                            for (int g = 0; g < GB; g += 2) {
                                const uint32_t p = bf16_pair(v[g][i], v[g + 1][i]);
                                hi4[g / 2] = p;
                                lo4[g / 2] = bf16_pair(v[g][i] - __uint_as_float(p << 16), v[g + 1][i] - __uint_as_float(p & 0xffff0000u));
                            }
                            uint8_t* row_at = mine + (i * 32 + lane) * G::point + g0 * 2;
                            *reinterpret_cast<uint4*>(row_at) = make_uint4(hi4[0], hi4[1], hi4[2], hi4[3]);
                            *reinterpret_cast<uint4*>(row_at + G::part) = make_uint4(lo4[0], lo4[1], lo4[2], lo4[3]);
                        }
                    } else {
#pragma unroll
                        for (int g = 0; g < GB; g++) {
                            w[g0 + g][0] = pack2(v[g][0], v[g][1]);
                            w[g0 + g][1] = pack2(v[g][2], v[g][3]);
                        }
                    }
                }
                if constexpr (G::tensor_mix) {
                    __syncwarp();
#pragma unroll 1
                    for (int nt = 0; nt < 4; nt++) {            // eight queries at a time
                        float o[MT][4][4] = {};                 // [h tile][key][accumulator]
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            uint32_t bh[4], bl[4];
                            if constexpr (MT == 2) {
                                const uint32_t at = smem_addr(mine) + (i * 32 + nt * 8 + (lane & 7)) * G::point + (lane >> 3) * 16;
                                ldmatrix4(bh, at);
                                ldmatrix4(bl, at + G::part);
                            } else {                            // high columns 0-7, 8-15, then low
                                uint32_t b4[4];
                                ldmatrix4(b4, smem_addr(mine) + (i * 32 + nt * 8 + (lane & 7)) * G::point + ((lane >> 3) & 1) * 16 + (lane >> 4) * G::part);
                                bh[0] = b4[0]; bh[1] = b4[1]; bl[0] = b4[2]; bl[1] = b4[3];
                            }
#pragma unroll
                            for (int m = 0; m < MT; m++)
#pragma unroll
                                for (int k = 0; k < MT; k++) {
                                    mma_16816(o[m][i], ta[m][k], bh[2 * k], bh[2 * k + 1]);
                                    mma_16816(o[m][i], ta[m][k], bl[2 * k], bl[2 * k + 1]);
                                }
                        }
#pragma unroll
                        for (int m = 0; m < MT; m++)
#pragma unroll
                            for (int r = 0; r < 4; r++) {
                                const int h = m * 16 + (lane >> 2) + (r >> 1) * 8;
                                const int q = tile_row + quarter * 32 + nt * 8 + (lane & 3) * 2 + (r & 1);
                                if (h < H && q < a.rows)
                                    *reinterpret_cast<uint2*>(a.w + h * a.head_stride + (long long)q * a.ldp + j0 + c) =
                                        make_uint2(bf16_pair(o[m][0][r], o[m][1][r]), bf16_pair(o[m][2][r], o[m][3][r]));
                            }
                    }
                    __syncwarp();                               // the rows are free again
                } else {
                    __nv_bfloat16* out = a.w + (long long)row * a.ldp + j0 + c;
#pragma unroll 2
                    for (int h = 0; h < H; h++) {
                        unsigned long long m0 = 0ull, m1 = 0ull;
#pragma unroll
                        for (int g = 0; g < HP; g += 2) {
                            const ulonglong2 t = talk[h * (HP / 2) + g / 2];
                            m0 = fma2(t.x, w[g][0], m0);
                            m1 = fma2(t.x, w[g][1], m1);
                            m0 = fma2(t.y, w[g + 1][0], m0);
                            m1 = fma2(t.y, w[g + 1][1], m1);
                        }
                        if (row < a.rows)
                            *reinterpret_cast<uint2*>(out + h * a.head_stride) = make_uint2(bf16_pair(lo(m0), hi(m0)), bf16_pair(lo(m1), hi(m1)));
                    }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(acc, G::cols);
}

// ---- heads one at a time, mixed behind the product with the keys ---------------------------------------
// sum over keys of (sum over g of T[h][g] w_g) v = sum over g of T[h][g] (sum over keys of w_g v): the weights are
// multiplied by the keys first and the heads are mixed in the outputs.  A head then multiplies the keys of
// EVERY key head, kv_heads times the products, and mixing falls from
// every (query, key) pair to every query.  A CTA owns 128 queries of one head and up to 256 output columns
// (more columns are more CTAs, each of which forms the scores again) and walks the keys in tiles of 64: scores into one of two TMEM buffers, sigmoids in fp32 on sixteen warps
// (a row's 64 keys belong to four threads: a sigmoid is a chain of a dozen instructions; with eight warps, 139 us
// and 34 % tensor-pipe activity for 2048 queries of 32 heads, with sixteen 122 us),
// weights as two bf16 parts, high and low, into one of two shared-memory buffers, O += (P_high + P_low) V
// in TMEM.  The weights carry 16 bits of mantissa into an fp32 sum and are never rounded to 8.
constexpr int kFlashKeys = 64;
constexpr int kFlashCols = 256;
constexpr int kFlashThreads = 576;         // TMA warp, MMA warp, 16 sigmoid warps

struct FlashArgs {
    CUtensorMap q, k, v;            // [rows][heads][dim_s] in boxes of 128 rows; [max_seq][kv][dim_s], 64 rows; [kv * dim][ldv], `cols` rows
    GateAttn at;
    int rows, pos0;                 // queries of the portion, at positions pos0 + row
    int kb;                         // 64-column steps of a query
    int per, cols;                  // key heads per CTA; their columns, padded to 16
    int tmem_cols;
    float* o;                       // [rows][heads][kv_heads * dim]
    int* status;
};

constexpr int flash_smem(int kb, int cols) { return kb * 128 * 128 + 4 * 128 * 128 + 2 * kb * kFlashKeys * 128 + 2 * ((cols * 128 + 1023) & ~1023) + 1024 + 256 + 8 * 2 * 32 * 4; }

__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
    tmem_wait_load();
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__global__ void __launch_bounds__(kFlashThreads, 1) gate_flash_kernel(const __grid_constant__ FlashArgs a) {
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    const GateAttn& A = a.at;
    const int kbytes = a.kb * kFlashKeys * 128, vbytes = pad_to(a.cols * 128, 1024);
    uint8_t* Q = base;
    uint8_t* P = Q + a.kb * 128 * 128;                      // [2][high, low][128 x 64]
    uint8_t* Ks = P + 4 * 128 * 128;
    uint8_t* Vs = Ks + 2 * kbytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(Vs + 2 * vbytes);
    uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 7, *s_full = bars + 9, *p_empty = bars + 11,
             *s_empty = bars + 13, *p_full = bars + 15;
    uint32_t* tmem_base = reinterpret_cast<uint32_t*>(bars + 17);
    float* rms = reinterpret_cast<float*>(Vs + 2 * vbytes + 256);               // [warp][2][16]: -log2 e / rms of the warp's keys

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, c = h / (A.heads / A.kv_heads), c0 = blockIdx.y * a.per;
    const int tile_row = (gridDim.z - 1 - blockIdx.z) * 128;                    // the longest rows of every head first
    const int first = a.pos0 + tile_row;                                        // position of the first query
    const int last = a.pos0 + min(tile_row + 128, a.rows) - 1;
    const int tiles = last / kFlashKeys + 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 17; i++) bar_init(bars + i, i >= 13 ? 16 : 1);
        bar_init_fence();
        tma_prefetch_map(&a.q); tma_prefetch_map(&a.k); tma_prefetch_map(&a.v);
    }
    if (warp == 1) tmem_alloc(tmem_base, a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // behind the allocation of TMEM, as in gemm_tc_kernel
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t S0 = *tmem_base, O = S0 + 2 * kFlashKeys;

    if (warp == 0) {
        if (lane == 0) {
            bar_expect(q_full, a.kb * 128 * 128);
            for (int x = 0; x < a.kb; x++) tma_load_3d(Q + x * 128 * 128, &a.q, x * 64, h, tile_row, q_full);
            int ki = 0, vi = 0;
            for (int j = 0; j < tiles; j++) {
                const int s = j & 1, use = j >> 1;
                if (use > 0 && !bar_wait(k_empty + s, (use - 1) & 1, a.status)) break;
                bar_expect(k_full + s, kbytes);
                for (int x = 0; x < a.kb; x++) tma_load_3d(Ks + s * kbytes + x * kFlashKeys * 128, &a.k, x * 64, c, j * kFlashKeys, k_full + s);
                ki = j + 1;
                if (use > 0 && !bar_wait(v_empty + s, (use - 1) & 1, a.status)) break;
                bar_expect(v_full + s, a.cols * 128);
                tma_load_3d(Vs + s * vbytes, &a.v, j * kFlashKeys, c0 * A.dim, 0, v_full + s);
                vi = j + 1;
            }
            // no copy may be in flight when the CTA leaves
            bar_wait(q_full, 0, a.status);
            for (int i = max(0, ki - 2); i < ki; i++) bar_wait(k_full + (i & 1), (i >> 1) & 1, a.status);
            for (int i = max(0, vi - 2); i < vi; i++) bar_wait(v_full + (i & 1), (i >> 1) & 1, a.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            auto scores = [&](int j) {
                const int b = j & 1;
                if (!bar_wait(k_full + b, (j >> 1) & 1, a.status)) return false;
                if (j >= 2 && !bar_wait(s_empty + b, ((j >> 1) - 1) & 1, a.status)) return false;
                tc_fence_after();
                for (int x = 0; x < a.kb; x++) {
                    const uint64_t da = tile_desc(Q + x * 128 * 128), db = tile_desc(Ks + b * kbytes + x * kFlashKeys * 128);
#pragma unroll
                    for (int k = 0; k < 4; k++) mma_bf16(S0 + b * kFlashKeys, da + 2 * k, db + 2 * k, mma_desc(kFlashKeys), x > 0 || k > 0);
                }
                mma_commit(k_empty + b);
                mma_commit(s_full + b);
                return true;
            };
            bool ok = bar_wait(q_full, 0, a.status) && scores(0);
            for (int j = 0; j < tiles && ok; j++) {
                if (j + 1 < tiles && !(ok = scores(j + 1))) break;
                const int b = j & 1;
                ok = bar_wait(v_full + b, (j >> 1) & 1, a.status) && bar_wait(p_full + b, (j >> 1) & 1, a.status);
                if (!ok) break;
                tc_fence_after();
                const uint64_t dh = tile_desc(P + b * 2 * 128 * 128), dl = tile_desc(P + (b * 2 + 1) * 128 * 128), db = tile_desc(Vs + b * vbytes);
                const uint32_t desc = mma_desc(a.cols);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    mma_bf16(O, dl + 2 * k, db + 2 * k, desc, j > 0 || k > 0);
                    mma_bf16(O, dh + 2 * k, db + 2 * k, desc, true);
                }
                mma_commit(v_empty + b);
                mma_commit(p_empty + b);
            }
        }
        __syncwarp();
    } else {
        constexpr float kLog2e = 1.4426950408889634f;
        const int quarter = warp & 3, part = (warp - 2) >> 2, r = quarter * 32 + lane;
        const uint32_t mine = (uint32_t)(quarter * 32) << 16;
        const float slope = A.slopes[h] * kLog2e, bias = -A.head_bias[h] * kLog2e;
        float* kr = rms + (warp - 2) * 32;
        auto key_rms = [&](int j) {
            const int key = j * kFlashKeys + part * 16 + (lane & 15);
            return key <= last ? -kLog2e * A.cache_r[(size_t)key * A.kv_heads + c] : 0.f;
        };
        const int pos = first + r;
        float next = key_rms(0), later = tiles > 1 ? key_rms(1) : 0.f;
        bool ok = true;
        for (int j = 0; j < tiles; j++) {
            const int b = j & 1, k0 = j * kFlashKeys + part * 16;
            if (lane < 16) kr[b * 16 + lane] = next;
            __syncwarp();
            next = later;
            if (j + 2 < tiles) later = key_rms(j + 2);
            ok = __all_sync(MG_FULL_MASK, bar_wait(s_full + b, (j >> 1) & 1, a.status));
            if (!ok) break;
            tc_fence_after();
            float s[16];
            tmem_load16(S0 + mine + b * kFlashKeys + part * 16, s);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(s_empty + b);
            const int seen = pos - k0 + 1;                  // keys of this part that the row sees
            const bool cut = __any_sync(MG_FULL_MASK, seen < 16);
            if (cut) {                                      // rows of the cache behind the query hold anything
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (i >= seen) s[i] = 0.f;
            }
            // 1 / (1 + 2^t), two at a time: 1 / x = y / (x y).  Exponents are cut off at 60, where a weight is 2^-60.
            const float line = fmaf(slope, (float)(pos - k0), bias);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + b * 16 + i);
                const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
                float e[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    float t = fmaf(s[i + u], kk[u], fmaf(-slope, (float)(i + u), line));
                    asm("min.NaN.f32 %0, %1, 0f42700000;" : "=f"(t) : "f"(t));
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e[u]) : "f"(t));
                    e[u] += 1.0f;
                }
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    float inv;
                    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(e[u] * e[u + 1]));
                    s[i + u] = inv * e[u + 1];
                    s[i + u + 1] = inv * e[u];
                }
            }
            if (cut) {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (i >= seen) s[i] = 0.f;
            }
            if (j >= 2) {
                ok = __all_sync(MG_FULL_MASK, bar_wait(p_empty + b, ((j >> 1) - 1) & 1, a.status));
                if (!ok) break;
            }
            uint8_t* high = P + b * 2 * 128 * 128 + r * 128;
#pragma unroll
            for (int x = 0; x < 2; x++) {
                uint32_t w[4], u[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float p = s[x * 8 + i * 2], q = s[x * 8 + i * 2 + 1];
                    w[i] = bf16_pair(p, q);
                    u[i] = bf16_pair(p - __uint_as_float(w[i] << 16), q - __uint_as_float(w[i] & 0xffff0000u));
                }
                const int at = ((part * 2 + x) ^ (r & 7)) << 4;
                *reinterpret_cast<uint4*>(high + at) = make_uint4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<uint4*>(high + 128 * 128 + at) = make_uint4(u[0], u[1], u[2], u[3]);
            }
            async_proxy_fence();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(p_full + b);
        }
        if (ok) ok = __all_sync(MG_FULL_MASK, bar_wait(p_empty + ((tiles - 1) & 1), ((tiles - 1) >> 1) & 1, a.status));
        if (ok) {
            tc_fence_after();
            // 32 columns of 32 rows through shared memory (queries, weights and keys have been consumed), so that a store is 128
            // bytes of one row
            const int wide = A.kv_heads * A.dim, cols = min(a.per, A.kv_heads - c0) * A.dim;
            float* piece = reinterpret_cast<float*>(base) + (warp - 2) * 32 * 33;
            for (int x = part * 32; x < cols; x += 128) {
                float o[32];
                tmem_load32(O + mine + x, o);
#pragma unroll
                for (int i = 0; i < 32; i++) piece[lane * 33 + i] = o[i];
                __syncwarp();
                float* out = a.o + ((size_t)(tile_row + quarter * 32) * A.heads + h) * wide + c0 * A.dim + x + lane;
#pragma unroll 8
                for (int i = 0; i < 32; i++)
                    if (tile_row + quarter * 32 + i < a.rows && x + lane < cols) out[(size_t)i * A.heads * wide] = piece[i * 33 + lane];
                __syncwarp();
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(S0, a.tmem_cols);
}

// out[row][h][d] = sum over g of T[h][g] o[row][g][key head of h][d]: every element of o is read once, V at a time (dim a
// multiple of V), for eight heads of its group at a time; a CTA takes V rows.
template <int V>
__global__ void __launch_bounds__(256) gate_mix_kernel(GateAttn A, int rows, const float* o, __nv_bfloat16* out, int ld_out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float talk[32][36];            // [g][h], heads of a group side by side
    const int H = A.heads, group = H / A.kv_heads, wide = A.kv_heads * A.dim, units = wide / V;
    for (int i = threadIdx.x; i < 32 * 36; i += 256) {
        const int h = i % 36, g = i / 36;
        talk[g][h] = h < H && g < H ? A.talk[h * H + g] : 0.f;
    }
    __syncthreads();
    const bool quads = (group & 3) == 0;
    for (int u = threadIdx.x; u < V * units; u += 256) {
        const size_t row = (size_t)blockIdx.x * V + u / units;
        if (row >= rows) return;
        const int e = u % units * V, c = e / A.dim, d = e - c * A.dim;
        const float* p = o + row * H * wide + e;
        for (int h0 = 0; h0 < group; h0 += 8) {
            const int first = c * group + h0, n = min(8, group - h0);
            float acc[8][V] = {};
#pragma unroll 8
            for (int g = 0; g < H; g++) {
                float v[V], t[8];
                if constexpr (V == 2) {
                    const float2 f = *reinterpret_cast<const float2*>(p + (size_t)g * wide);
                    v[0] = f.x; v[1] = f.y;
                } else {
                    v[0] = p[(size_t)g * wide];
                }
                if (quads) {                                // heads past the group are in the row, and not stored
                    const float4 x = *reinterpret_cast<const float4*>(&talk[g][first]), y = *reinterpret_cast<const float4*>(&talk[g][first + 4]);
                    t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w; t[4] = y.x; t[5] = y.y; t[6] = y.z; t[7] = y.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 8; i++) t[i] = talk[g][min(first + i, 35)];
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int q = 0; q < V; q++) acc[i][q] = fmaf(t[i], v[q], acc[i][q]);
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i < n) {
                    __nv_bfloat16* to = out + row * ld_out + (size_t)(first + i) * A.dim + d;
                    if constexpr (V == 2) *reinterpret_cast<__nv_bfloat162*>(to) = __floats2bfloat162_rn(acc[i][0], acc[i][1]);
                    else *to = __float2bfloat16_rn(acc[i][0]);
                }
        }
    }
}

// cache [len][kv][dim_s] -> vt [kv][dim][ldv], zero from len to ldv
__global__ void __launch_bounds__(256) key_transpose_kernel(const __nv_bfloat16* cache, int kv_heads, int dim, int dim_s, int len, int ldv,
                                                            __nv_bfloat16* vt) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __nv_bfloat16 t[32][34];
    const int p0 = blockIdx.x * 32, d0 = blockIdx.y * 32, c = blockIdx.z, x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (int i = y; i < 32; i += 8)
        t[i][x] = p0 + i < len && d0 + x < dim ? cache[((size_t)(p0 + i) * kv_heads + c) * dim_s + d0 + x] : __float2bfloat16_rn(0.f);
    __syncthreads();
    for (int i = y; i < 32; i += 8)
        if (d0 + i < dim && p0 + x < ldv) vt[((size_t)c * dim + d0 + i) * ldv + p0 + x] = t[x][i];
}

template <int HP>
cudaError_t scores(const ScoreArgs& a, bool pdl, cudaStream_t s) {
    using G = Geo<HP>;
    launch_pdl(gate_scores_kernel<HP>, dim3(pad_to(a.pos0 + a.row0 + a.rows, 64) / G::bn, (a.rows + 127) / 128), kThreads, G::bytes, pdl, s, a);
    return cudaGetLastError();
}

int flash_key_heads(const GateAttn& at) { return std::min(at.kv_heads, kFlashCols / at.dim); }     // per CTA

// One head at a time where that is the faster way.  Against it: more columns of key heads than a CTA takes are more CTAs (groups) that
// form the same scores; and a CTA walks every key of its rows, while the pairs of the other kernel are dealt over keys
// too, so that few heads behind a long context leave most SMs idle.  B200, Forward of one layer of 256 columns, one head at a time / pairs, us:
// 2048 tokens, 32 heads of 64 with 4, 8, 16 and 32 key heads 243 / 480, 363 / 477, 610 / 481 and 1139 / 485; 512 tokens behind 3584,
// 16, 8 and 4 heads of 64 with 4 key heads 175 / 237, 168 / 153 and 168 / 127; 128 tokens, 32 heads of 96 with 8 (four groups)
// 116 / 142.  The lines were laid through 138 shapes of heads at 13 portions each.
constexpr int kFlashGroups = 4;
int flash_groups(const GateAttn& at) { return (at.kv_heads + flash_key_heads(at) - 1) / flash_key_heads(at); }
bool gate_flash_pays(const GateAttn& at, int pos0, int n) {
    if (at.dim_s > 128) return false;                       // a query, two buffers of weights and two stages of keys fill shared memory
    const long long longest = (pos0 + n + kFlashKeys - 1) / kFlashKeys;
    if (flash_groups(at) > 2) return flash_groups(at) <= kFlashGroups && longest <= 2;
    long long tiles = 0;
    for (int r = 0; r < n; r += 128) tiles += (pos0 + std::min(r + 128, n) + kFlashKeys - 1) / kFlashKeys;
    return (longest - 4) * sm_count() <= 4 * at.heads * tiles;
}

size_t flash_bytes(const GateAttn& at, int max_rows) {
    if (at.dim_s > 128 || flash_groups(at) > kFlashGroups) return 0;
    return (size_t)(flash_groups(at) > 2 ? std::min(max_rows, 2 * kFlashKeys) : max_rows) * at.heads * at.kv_heads * at.dim * 4;
}
size_t pair_bytes(const GateAttn& at, int rows) { return (size_t)rows * at.heads * pad_to(at.max_seq, 64) * 2; }
// Queries of a block whose pairs' weights fit `bytes`.
int pair_rows(const GateAttn& at, int max_rows, size_t bytes) {
    return std::max(128, (int)std::min<size_t>(bytes / pair_bytes(at, 1), (size_t)pad_to(max_rows, 128)) / 128 * 128);
}

cudaError_t launch_flash(const GateAttn& at, const void* qh, int pos0, int n, int max_rows, void* work, const void* vt, int ldv,
                         void* out, int ld_out, int* status, int* launches, bool pdl, cudaStream_t s) {
    FlashArgs a{};
    a.at = at; a.pos0 = pos0; a.rows = n; a.o = (float*)work; a.status = status;
    a.kb = (at.dim_s + 63) / 64;
    a.per = flash_key_heads(at);
    a.cols = pad_to(a.per * at.dim, 16);
    a.tmem_cols = 2 * kFlashKeys + pad_to(a.cols, 32) <= 256 ? 256 : 512;
    if (!make_head_map(&a.q, qh, at.dim_s, at.heads, max_rows, at.dim_s, (long long)at.heads * at.dim_s, 128) ||
        !make_head_map(&a.k, at.cache, at.dim_s, at.kv_heads, at.max_seq, at.dim_s, (long long)at.kv_heads * at.dim_s, kFlashKeys) ||
        !make_tile_map(&a.v, vt, ldv, at.kv_heads * at.dim, 1, ldv, (long long)at.kv_heads * at.dim * ldv, a.cols))
        return cudaErrorInvalidValue;
    launch_pdl(gate_flash_kernel, dim3(at.heads, (at.kv_heads + a.per - 1) / a.per, (n + 127) / 128), kFlashThreads, flash_smem(a.kb, a.cols), pdl, s, a);
    if (at.dim % 2 == 0) launch_pdl(gate_mix_kernel<2>, (n + 1) / 2, 256, 0, pdl, s, at, n, a.o, (__nv_bfloat16*)out, ld_out);
    else launch_pdl(gate_mix_kernel<1>, n, 256, 0, pdl, s, at, n, a.o, (__nv_bfloat16*)out, ld_out);
    *launches += 2;
    return cudaGetLastError();
}

}  // namespace

cudaError_t gate_attn_tc_attrs() {
    if (cudaError_t c = allow_smem(gate_scores_kernel<4>, Geo<4>::bytes)) return c;
    if (cudaError_t c = allow_smem(gate_scores_kernel<8>, Geo<8>::bytes)) return c;
    if (cudaError_t c = allow_smem(gate_scores_kernel<16>, Geo<16>::bytes)) return c;
    if (cudaError_t c = allow_smem(gate_scores_kernel<32>, Geo<32>::bytes)) return c;
    return allow_smem(gate_flash_kernel, flash_smem(2, kFlashCols));
}

bool gate_attn_tc_fits(const GateAttn& at) { return at.heads <= 32; }

size_t gate_attn_tc_bytes(const GateAttn& at, int max_rows, size_t budget) {
    return std::max(pair_bytes(at, pair_rows(at, max_rows, budget)), flash_bytes(at, max_rows));
}

cudaError_t launch_gate_attn_tc(const GateAttn& at, const void* qh, int pos0, int n, int max_rows, void* weights, size_t bytes, void* vt,
                                void* out, int ld_out, int* status, int* launches, bool pdl, cudaStream_t s) {
    const int len = pos0 + n, ldv = pad_to(len, 64);
    launch_pdl(key_transpose_kernel, dim3(ldv / 32, (at.dim + 31) / 32, at.kv_heads), 256, 0, pdl, s, (const __nv_bfloat16*)at.cache, at.kv_heads, at.dim,
                                                                                       at.dim_s, len, ldv, (__nv_bfloat16*)vt);
    *launches += 1;
    if (gate_flash_pays(at, pos0, n)) return launch_flash(at, qh, pos0, n, max_rows, weights, vt, ldv, out, ld_out, status, launches, pdl, s);
    const int block_rows = pair_rows(at, max_rows, bytes);
    const int hp = at.heads <= 4 ? 4 : at.heads <= 8 ? 8 : at.heads <= 16 ? 16 : 32;
    ScoreArgs a{};
    a.at = at; a.pos0 = pos0; a.w = (__nv_bfloat16*)weights; a.status = status;
    if (!make_head_map(&a.q, qh, at.dim_s, at.heads, max_rows, at.dim_s, (long long)at.heads * at.dim_s, 128) ||
        !make_head_map(&a.k, at.cache, at.dim_s, at.kv_heads, at.max_seq, at.dim_s, (long long)at.kv_heads * at.dim_s, hp <= 8 ? 32 : 16))
        return cudaErrorInvalidValue;
    GemmTC g{};
    g.bn = at.dim > 64 ? 128 : 64;
    g.n = at.dim; g.batch = at.heads; g.b_group = at.heads / at.kv_heads; g.ldc = ld_out; g.batch_c = at.dim; g.mode = GEMM_BF16; g.status = status;
    if (!make_tile_map(&g.b, vt, ldv, at.dim, at.kv_heads, ldv, (long long)at.dim * ldv, g.bn)) return cudaErrorInvalidValue;
    for (int q0 = 0; q0 < n; q0 += block_rows) {
        const int rows = std::min(block_rows, n - q0);
        a.row0 = q0; a.rows = rows; a.ldp = pad_to(pos0 + q0 + rows, 64); a.head_stride = (long long)block_rows * a.ldp;
        cudaError_t c = hp == 4 ? scores<4>(a, pdl, s) : hp == 8 ? scores<8>(a, pdl, s) : hp == 16 ? scores<16>(a, pdl, s) : scores<32>(a, pdl, s);
        if (c != cudaSuccess) return c;
        if (!make_tile_map(&g.a, weights, a.ldp, block_rows, at.heads, a.ldp, a.head_stride, 128)) return cudaErrorInvalidValue;
        g.m = rows; g.k = a.ldp; g.causal_pos0 = pos0 + q0;
        g.out = (__nv_bfloat16*)out + (size_t)q0 * ld_out;
        if ((c = launch_gemm_tc(g, pdl, s)) != cudaSuccess) return c;
        *launches += 2;
    }
    return cudaSuccess;
}

}  // namespace mg
