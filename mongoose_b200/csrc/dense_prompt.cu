// Prompts of the fixed seven-matrix decode block, many tokens at a time.  Fed one by one, every token pays
// the decode kernel's chain of dependent steps and streams every weight again; here a weight is read
// once per 64 tokens and multiplied on the tensor cores.
//
// Products.  Activations are fp32 and stay so: a value is the sum of three bf16 parts (8 + 8 + 8 bits of
// mantissa, exact).  Q8_0 and Q4_0 quants are small integers, exact in bf16, and one K = 32 block is two steps
// of tcgen05.mma: per block the tensor cores form sum q * (x0 + x1 + x2) in fp32, smallest part first, and
// the epilogue warps add it to fp32 registers times the block's scale, as the decode kernels do.  fp16
// weights are two bf16 parts (exact), five products, one sum per 64 columns.  No sum in the tensor core runs
// over more than 64 columns, so its truncating accumulator stays at the level of one fp32 rounding.
//
// B200: prompt of 512 tokens, six layers of 1.1B widths, Q8_0: 101 ms one by one, 2.2 ms so (0.25 PFLOP/s counting
// each of the three parts' products).  Short prompts are bound by the nine launches of a layer, long ones by the products.
#include "dense_prompt.h"

#include <type_traits>

#include "gemm_tc.h"
#include "umma.cuh"

namespace mg {

namespace {

// ---- products ------------------------------------------------------------------------------------
// A CTA: 128 weight rows (the M side) x NT tokens, one piece of K in steps of 64 columns.
//   warp 0         TMA of the three activation parts
//   warp 1         tcgen05.mma, one thread
//   warps 2 - 9    accumulators out of TMEM, scales, fp32 sums in registers (32 rows x NT / 2 tokens each)
//   warps 10 - 17  weights: 16-byte loads two steps ahead, quants to bf16, 128-byte-swizzled tile
constexpr int kGemmThreads = 576;
constexpr int kAcc = 4;                 // accumulator slots in TMEM

template <int FMT, int NT>
struct GemmShape {
    static constexpr int w_parts = FMT == FMT_F16 ? 2 : 1;
    static constexpr int w_bytes = w_parts * 128 * 128, x_part = NT * 128, stage = w_bytes + 3 * x_part;
    static constexpr int stages = NT == 32 ? (FMT == FMT_F16 ? 4 : 6) : (FMT == FMT_F16 ? 3 : 5);
    static constexpr int blocks = FMT == FMT_F16 ? 1 : 2;       // sums per step
    static constexpr int slot = blocks * NT;                    // TMEM columns of a slot
    static constexpr int bytes = stages * stage + 1024 + 256;
    static constexpr int loads = FMT == FMT_Q8_0 ? 2 : FMT == FMT_Q4_0 ? 1 : 4;     // 16-byte loads per weight thread and step
};

__device__ __forceinline__ void tmem_load16_async(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}

__device__ __forceinline__ uint32_t bf2_sub(uint32_t a, uint32_t b) {
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&d);
}
// Two int8 in the low bytes of two halfwords -> bf16: 128 + the low seven bits, minus 128, or minus 256 where negative.
__device__ __forceinline__ uint32_t s8x2_bf16(uint32_t h) { return bf2_sub((h & 0x007f007fu) | 0x43004300u, (h & 0x00800080u) | 0x43004300u); }
// Two nibbles -> bf16 of nibble - 8
__device__ __forceinline__ uint32_t u4x2_bf16(uint32_t h) { return bf2_sub(h | 0x43004300u, 0x43084308u); }

__device__ __forceinline__ void store_piece(uint8_t* tile, int row, int piece, uint4 v) {
    *reinterpret_cast<uint4*>(tile + row * 128 + ((piece ^ (row & 7)) << 4)) = v;
}

// The 16-byte loads of weight thread t for step i of 64 columns: rows past the matrix repeat its last one (their results
// are not stored), columns past K are zeros.
template <int FMT>
__device__ __forceinline__ void load_weights(const uint8_t* qs, int row0, int rows, int K, int step, int t, uint4 (&v)[GemmShape<FMT, 64>::loads]) {
    constexpr int per_row = FMT == FMT_Q8_0 ? 4 : FMT == FMT_Q4_0 ? 2 : 8;      // 16-byte pieces of a row and step
    constexpr int weights = 64 / per_row;                                       // per piece
    const size_t row_bytes = FMT == FMT_Q8_0 ? (size_t)K : FMT == FMT_Q4_0 ? (size_t)K / 2 : (size_t)K * 2;
#pragma unroll
    for (int j = 0; j < GemmShape<FMT, 64>::loads; j++) {
        const int id = t + 256 * j, r = id / per_row, c = id % per_row, k = step * 64 + c * weights;
        v[j] = make_uint4(0u, 0u, 0u, 0u);
        if (k < K) v[j] = __ldg(reinterpret_cast<const uint4*>(qs + (size_t)min(row0 + r, rows - 1) * row_bytes) + step * per_row + c);
        else if (FMT == FMT_Q4_0) v[j] = make_uint4(0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u);
    }
}

template <int FMT>
__device__ __forceinline__ void store_weights(uint8_t* tile, int t, const uint4 (&v)[GemmShape<FMT, 64>::loads]) {
#pragma unroll
    for (int j = 0; j < GemmShape<FMT, 64>::loads; j++) {
        const int id = t + 256 * j;
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        uint32_t o[16];
        if (FMT == FMT_Q8_0) {
            const int r = id >> 2, c = id & 3;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                o[2 * i] = s8x2_bf16(__byte_perm(w[i], 0, 0x4140));
                o[2 * i + 1] = s8x2_bf16(__byte_perm(w[i], 0, 0x4342));
            }
            store_piece(tile, r, 2 * c, make_uint4(o[0], o[1], o[2], o[3]));
            store_piece(tile, r, 2 * c + 1, make_uint4(o[4], o[5], o[6], o[7]));
        } else if (FMT == FMT_Q4_0) {
            const int r = id >> 1, c = id & 1;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t lo = w[i] & 0x0f0f0f0fu, hi = (w[i] >> 4) & 0x0f0f0f0fu;
                o[2 * i] = u4x2_bf16(__byte_perm(lo, 0, 0x4140));
                o[2 * i + 1] = u4x2_bf16(__byte_perm(lo, 0, 0x4342));
                o[8 + 2 * i] = u4x2_bf16(__byte_perm(hi, 0, 0x4140));
                o[8 + 2 * i + 1] = u4x2_bf16(__byte_perm(hi, 0, 0x4342));
            }
#pragma unroll
            for (int p = 0; p < 4; p++) store_piece(tile, r, 4 * c + p, make_uint4(o[4 * p], o[4 * p + 1], o[4 * p + 2], o[4 * p + 3]));
        } else {
            const int r = id >> 3, c = id & 7;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
                const __nv_bfloat162 l = __floats2bfloat162_rn(f.x - __low2float(h), f.y - __high2float(h));
                o[i] = *reinterpret_cast<const uint32_t*>(&h);
                o[4 + i] = *reinterpret_cast<const uint32_t*>(&l);
            }
            store_piece(tile, r, c, make_uint4(o[0], o[1], o[2], o[3]));
            store_piece(tile + 128 * 128, r, c, make_uint4(o[4], o[5], o[6], o[7]));
        }
    }
}

template <int FMT, int NT>
__global__ void __launch_bounds__(kGemmThreads, 1) prompt_gemm_kernel(const __grid_constant__ PromptGemm g) {
    using S = GemmShape<FMT, NT>;
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_x = reinterpret_cast<uint64_t*>(base + S::stages * S::stage);
    uint64_t* full_w = full_x + S::stages;
    uint64_t* empty = full_w + S::stages;
    uint64_t* acc_full = empty + S::stages;
    uint64_t* acc_empty = acc_full + kAcc;
    uint64_t* done = acc_empty + kAcc;
    uint32_t* tmem_base = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, m = tile < g.tile_end[0] ? 0 : tile < g.tile_end[1] ? 1 : 2;
    const int row0 = (tile - (m == 0 ? 0 : m == 1 ? g.tile_end[0] : g.tile_end[1])) * 128;
    const int rows = m == 0 ? g.rows[0] : m == 1 ? g.rows[1] : g.rows[2];
    const WeightView w = m == 0 ? g.w[0] : m == 1 ? g.w[1] : g.w[2];
    const int tok0 = blockIdx.y * NT;
    const int step0 = blockIdx.z * g.steps, kt = min(g.steps, (g.K + 63) / 64 - step0);

    if (threadIdx.x == 0) {
        for (int i = 0; i < S::stages; i++) { bar_init(full_x + i, 1); bar_init(full_w + i, 8); bar_init(empty + i, 1); }
        for (int i = 0; i < kAcc; i++) { bar_init(acc_full + i, 1); bar_init(acc_empty + i, 8); }
        bar_init(done, 1);
        bar_init_fence();
        tma_prefetch_map(&g.x);
    }
    if (warp == 1) tmem_alloc(tmem_base, kAcc * S::slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t acc = *tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < kt; i++) {
                const int s = i % S::stages, use = i / S::stages;
                if (use > 0 && !bar_wait(empty + s, (use - 1) & 1, g.status)) break;
                bar_expect(full_x + s, 3 * S::x_part);
                uint8_t* to = base + s * S::stage + S::w_bytes;
#pragma unroll
                for (int p = 0; p < 3; p++) tma_load_3d(to + p * S::x_part, &g.x, (step0 + i) * 64, tok0, p, full_x + s);
                issued = i + 1;
            }
            // no copy may be in flight when the CTA leaves
            for (int i = max(0, issued - S::stages); i < issued; i++) bar_wait(full_x + i % S::stages, (i / S::stages) & 1, g.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            for (int i = 0; i < kt; i++) {
                const int s = i % S::stages, a = i % kAcc;
                if (i >= kAcc && !bar_wait(acc_empty + a, (i / kAcc - 1) & 1, g.status)) break;
                if (!bar_wait(full_w + s, (i / S::stages) & 1, g.status) || !bar_wait(full_x + s, (i / S::stages) & 1, g.status)) break;
                tc_fence_after();
                uint8_t* st = base + s * S::stage;
                const uint64_t dw = tile_desc(st);
                uint64_t dx[3];
#pragma unroll
                for (int p = 0; p < 3; p++) dx[p] = tile_desc(st + S::w_bytes + p * S::x_part);
                const uint32_t to = acc + a * S::slot;
                if (FMT == FMT_F16) {
                    const uint64_t dl = tile_desc(st + 128 * 128);
#pragma unroll
                    for (int k = 0; k < 4; k++) {       // smallest products first
                        mma_bf16(to, dw + 2 * k, dx[2] + 2 * k, mma_desc(NT), k > 0);
                        mma_bf16(to, dl + 2 * k, dx[1] + 2 * k, mma_desc(NT), true);
                        mma_bf16(to, dw + 2 * k, dx[1] + 2 * k, mma_desc(NT), true);
                        mma_bf16(to, dl + 2 * k, dx[0] + 2 * k, mma_desc(NT), true);
                        mma_bf16(to, dw + 2 * k, dx[0] + 2 * k, mma_desc(NT), true);
                    }
                } else {
#pragma unroll
                    for (int b = 0; b < 2; b++)
#pragma unroll
                        for (int p = 2; p >= 0; p--)
#pragma unroll
                            for (int k = 0; k < 2; k++)
                                mma_bf16(to + b * NT, dw + 4 * b + 2 * k, dx[p] + 4 * b + 2 * k, mma_desc(NT), p < 2 || k > 0);
                }
                mma_commit(empty + s);
                mma_commit(acc_full + a);
            }
            // nothing may be in flight when the accumulators are given back
            mma_commit(done);
            bar_wait(done, 0, g.status);
        }
        __syncwarp();
    } else if (warp < 10) {
        constexpr int C = NT / 2;                       // tokens per thread
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const int row = row0 + quarter * 32 + lane;
        const unsigned short* ds = FMT == FMT_F16 ? nullptr : w.ds + (size_t)min(row, rows - 1) * (g.K / 32);
        const int nb = g.K / 32;
        float sum[C];
#pragma unroll
        for (int i = 0; i < C; i++) sum[i] = 0.f;
        auto scale = [&](int b) { return b < nb ? half_bits_to_float(__ldg(ds + b)) : 0.f; };
        float d0 = 1.f, d1 = 1.f;
        if (FMT != FMT_F16) { d0 = scale(2 * step0); d1 = scale(2 * step0 + 1); }
        for (int i = 0; i < kt; i++) {
            const int a = i % kAcc;
            float n0 = 1.f, n1 = 1.f;
            if (FMT != FMT_F16 && i + 1 < kt) { n0 = scale(2 * (step0 + i + 1)); n1 = scale(2 * (step0 + i + 1) + 1); }
            if (!__all_sync(MG_FULL_MASK, bar_wait(acc_full + a, (i / kAcc) & 1, g.status))) break;
            tc_fence_after();
            const uint32_t from = acc + ((uint32_t)(quarter * 32) << 16) + a * S::slot + half * C;
            uint32_t v[C / 16][S::blocks][16];
#pragma unroll
            for (int c = 0; c < C / 16; c++)
#pragma unroll
                for (int b = 0; b < S::blocks; b++) tmem_load16_async(from + b * NT + c * 16, v[c][b]);
            tmem_wait_load();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(acc_empty + a);
#pragma unroll
            for (int c = 0; c < C / 16; c++)
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    float& s = sum[c * 16 + j];
                    if (FMT == FMT_F16) s += __uint_as_float(v[c][0][j]);
                    else s = fmaf(d1, __uint_as_float(v[c][S::blocks - 1][j]), fmaf(d0, __uint_as_float(v[c][0][j]), s));
                }
            d0 = n0; d1 = n1;
        }
        if (row < rows) {
            const int col = (m == 0 ? g.col[0] : m == 1 ? g.col[1] : g.col[2]) + row;
            float* out = g.out + blockIdx.z * g.stride + (size_t)(tok0 + half * C) * g.ld + col;
#pragma unroll
            for (int i = 0; i < C; i++)
                if (tok0 + half * C + i < g.tokens) out[(size_t)i * g.ld] = sum[i];
        }
        tc_fence_before();
    } else {
        const int t = threadIdx.x - 320;
        uint4 v0[S::loads], v1[S::loads], v2[S::loads];
        load_weights<FMT>(w.qs, row0, rows, g.K, step0, t, v0);
        load_weights<FMT>(w.qs, row0, rows, g.K, step0 + 1, t, v1);         // past K: zeros
        for (int i = 0; i < kt; i++) {
            const int s = i % S::stages, use = i / S::stages;
            load_weights<FMT>(w.qs, row0, rows, g.K, step0 + i + 2, t, v2);
            if (use > 0 && !__all_sync(MG_FULL_MASK, bar_wait(empty + s, (use - 1) & 1, g.status))) break;
            store_weights<FMT>(base + s * S::stage, t, v0);
            async_proxy_fence();
            __syncwarp();
            if (lane == 0) bar_arrive(full_w + s);
#pragma unroll
            for (int j = 0; j < S::loads; j++) { v0[j] = v1[j]; v1[j] = v2[j]; }
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(acc, kAcc * S::slot);
}

template <int FMT, int NT>
cudaError_t run_gemm(const PromptGemm& g, cudaStream_t s) {
    using S = GemmShape<FMT, NT>;
    prompt_gemm_kernel<FMT, NT><<<dim3(g.tile_end[2], (g.tokens + NT - 1) / NT, g.pieces), kGemmThreads, S::bytes, s>>>(g);
    return cudaGetLastError();
}

// ---- rows ------------------------------------------------------------------------------------------

__device__ __forceinline__ float piece_sum(const PieceSums& a, size_t t, int i) {
    const float* p = a.p + t * a.ld + i;
    float v = p[0];
    for (int s = 1; s < a.n; s++) v += p[s * a.stride];
    return v;
}

__device__ __forceinline__ void store_split(const SplitRows& o, size_t t, int i, float v) {
    __nv_bfloat16* p = o.p + t * o.width + i;
    const __nv_bfloat16 a = __float2bfloat16_rn(v);
    const float r = v - __bfloat162float(a);
    const __nv_bfloat16 b = __float2bfloat16_rn(r);
    p[0] = a;
    p[o.part] = b;
    p[2 * o.part] = __float2bfloat16_rn(r - __bfloat162float(b));
}

__global__ void __launch_bounds__(256) prompt_norm_kernel(const PromptNorm a) {
    extern __shared__ __align__(16) float y[];
    __shared__ float red[40];
    const size_t t = blockIdx.x;
    const int n = a.out.width;
    float* x = a.x + t * n;
    const int token = a.tokens ? a.tokens[t] : 0;
    float ss = 0.f;
    for (int i = threadIdx.x; i < n; i += 256) {
        float v = a.tokens ? embed_value(a.embed, a.embed_fmt, n, token, i) : x[i];
        if (a.add.n) v += piece_sum(a.add, t, i);
        x[i] = v;
        y[i] = v;
        ss = fmaf(v, v, ss);
    }
    const float r = 1.0f / sqrtf(block_sum(ss, red) / (float)n + a.eps);
    for (int i = threadIdx.x; i < n; i += 256) store_split(a.out, t, i, y[i] * r * a.w[i]);
}

__global__ void __launch_bounds__(256) prompt_rope_kernel(const PromptRope a) {
    const size_t t = blockIdx.x;
    const int pos = a.pos0 + (int)t, half = a.head_dim / 2;
    const int pairs = (a.q_dim + 2 * a.kv_dim) / 2;
    for (int i = a.first / 2 + threadIdx.x; i < pairs; i += 256) {
        const int m = i < a.q_dim / 2 ? 0 : i < (a.q_dim + a.kv_dim) / 2 ? 1 : 2;
        const int base = m == 0 ? 0 : m == 1 ? a.q_dim : a.q_dim + a.kv_dim;
        const int k = i - base / 2;
        int r0 = 2 * k, r1 = r0 + 1;
        if (m < 2) {
            const int head = k / half, j = k - head * half;
            r0 = head * a.head_dim + j;
            r1 = r0 + half;
        }
        float v0 = piece_sum(a.qkv, t, base + r0 - a.first), v1 = piece_sum(a.qkv, t, base + r1 - a.first);
        const float* bias = m == 0 ? a.bias[0] : m == 1 ? a.bias[1] : a.bias[2];
        if (bias) { v0 += bias[r0]; v1 += bias[r1]; }
        if (m < 2) {
            const int j = k % half;
            const float c = a.cos_tab[(size_t)pos * half + j], s = a.sin_tab[(size_t)pos * half + j];
            const float u0 = v0 * c - v1 * s, u1 = v0 * s + v1 * c;
            v0 = u0; v1 = u1;
        }
        if (m == 0) {
            a.q[t * a.q_dim + r0] = v0;
            a.q[t * a.q_dim + r1] = v1;
        } else {
            __half* o = (m == 1 ? a.kc : a.vc) + (size_t)pos * a.kv_dim;
            o[r0] = __float2half_rn(v0);
            o[r1] = __float2half_rn(v1);
        }
    }
}

__global__ void __launch_bounds__(256) prompt_swiglu_kernel(const PieceSums gu, const SplitRows out) {
    const size_t t = blockIdx.y;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= out.width) return;
    const float g = piece_sum(gu, t, i), u = piece_sum(gu, t, out.width + i);
    store_split(out, t, i, g / (1.0f + expf(-g)) * u);
}

// ---- attention -------------------------------------------------------------------------------------
// One head, 32 queries, tiles of 64 cached rows; all fp32 on the CUDA cores (queries and probabilities have
// 32 bits, and a prompt's scores are a hundredth of its products).  Thread (ty, tx) owns queries 4 ty .. 4 ty + 3;
// of the scores, keys tx + 16 j; of the output, elements 4 tx + 64 j (HD = 32: 2 tx).  Rows of K are HD + 4 floats
// apart, so that the 16 rows an access touches fall on distinct banks.
constexpr int kAttnQ = 32, kAttnK = 64;

template <int HD>
constexpr int attn_smem() { return (kAttnQ * HD + kAttnK * (HD + 4) + kAttnK * HD + kAttnQ * (kAttnK + 4)) * 4; }

template <int HD>
__global__ void __launch_bounds__(128) prompt_attn_kernel(const PromptAttn a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int KS = HD + 4, PS = kAttnK + 4, E = HD / 16;
    float *Q = sm, *K = Q + kAttnQ * HD, *V = K + kAttnK * KS, *P = V + kAttnK * HD;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int head = blockIdx.x, kvh = head / (a.n_heads / a.n_kv_heads);
    const int q0 = (gridDim.y - 1 - blockIdx.y) * kAttnQ;          // the longest rows first
    const int q_dim = a.n_heads * HD;
    const float scale = rsqrtf((float)HD);
    for (int i = threadIdx.x; i < kAttnQ * HD / 4; i += 128) {
        const int r = i / (HD / 4), c = i % (HD / 4);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q0 + r < a.tokens) v = *reinterpret_cast<const float4*>(a.q + (size_t)(q0 + r) * q_dim + head * HD + 4 * c);
        reinterpret_cast<float4*>(Q)[i] = v;
    }
    const int first = a.pos0 + q0, last = a.pos0 + min(q0 + kAttnQ, a.tokens) - 1;      // positions of the first and the last query
    float o[4][E] = {}, mx[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) { mx[i] = -INFINITY; l[i] = 0.f; }

    for (int k0 = 0; k0 <= last; k0 += kAttnK) {
        __syncthreads();
        for (int i = threadIdx.x; i < kAttnK * HD / 8; i += 128) {
            const int r = i / (HD / 8), c = i % (HD / 8);
            uint4 kk = make_uint4(0u, 0u, 0u, 0u), vv = kk;
            if (k0 + r <= last) {
                const size_t at = (size_t)(k0 + r) * a.kv_dim + kvh * HD + 8 * c;
                kk = *reinterpret_cast<const uint4*>(a.kc + at);
                vv = *reinterpret_cast<const uint4*>(a.vc + at);
            }
            const __half2 *kh = reinterpret_cast<const __half2*>(&kk), *vh = reinterpret_cast<const __half2*>(&vv);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float2 x = __half22float2(kh[2 * j]), y = __half22float2(kh[2 * j + 1]);
                *reinterpret_cast<float4*>(K + r * KS + 8 * c + 4 * j) = make_float4(x.x, x.y, y.x, y.y);
                const float2 z = __half22float2(vh[2 * j]), w = __half22float2(vh[2 * j + 1]);
                *reinterpret_cast<float4*>(V + r * HD + 8 * c + 4 * j) = make_float4(z.x, z.y, w.x, w.y);
            }
        }
        __syncthreads();
        float s[4][4] = {};
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            float4 q[4], k[4];
#pragma unroll
            for (int i = 0; i < 4; i++) q[i] = *reinterpret_cast<const float4*>(Q + (4 * ty + i) * HD + d);
#pragma unroll
            for (int j = 0; j < 4; j++) k[j] = *reinterpret_cast<const float4*>(K + (tx + 16 * j) * KS + d);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    s[i][j] = fmaf(q[i].w, k[j].w, fmaf(q[i].z, k[j].z, fmaf(q[i].y, k[j].y, fmaf(q[i].x, k[j].x, s[i][j]))));
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int pos = first + 4 * ty + i;
            float m = mx[i];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                s[i][j] = k0 + tx + 16 * j <= pos ? s[i][j] * scale : -INFINITY;
                m = fmaxf(m, s[i][j]);
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(MG_FULL_MASK, m, x));
            // key 0 is visible to every query, so m is finite (or NaN, or infinite as its scores are) from the first tile on
            const float keep = expf(mx[i] - m);
            mx[i] = m;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float p = expf(s[i][j] - m);
                P[(4 * ty + i) * PS + tx + 16 * j] = p;
                sum += p;
            }
            l[i] = l[i] * keep + sum;
#pragma unroll
            for (int e = 0; e < E; e++) o[i][e] *= keep;
        }
        __syncwarp();                                   // a query's 16 threads are in one warp
        const int n = min(kAttnK, (last - k0 + 4) & ~3);        // rows past `last` are zeros with zero weight
        auto add_values = [&](auto masked) {
            for (int k = 0; k < n; k += 4) {
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] = *reinterpret_cast<const float4*>(P + (4 * ty + i) * PS + k);
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    const float* v = V + (k + kk) * HD;
                    float x[E];
                    if (HD == 32) {
                        *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(v + 2 * tx);
                    } else {
#pragma unroll
                        for (int e = 0; e < E / 4; e++) *reinterpret_cast<float4*>(x + 4 * e) = *reinterpret_cast<const float4*>(v + 4 * tx + 64 * e);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (decltype(masked)::value && k0 + k + kk > first + 4 * ty + i) continue;
                        const float w = kk == 0 ? p[i].x : kk == 1 ? p[i].y : kk == 2 ? p[i].z : p[i].w;
#pragma unroll
                        for (int e = 0; e < E; e++) o[i][e] = fmaf(w, x[e], o[i][e]);
                    }
                }
            }
        };
        // a row behind a query counts for nothing, not for zero times what it holds: its values may have overflowed fp16
        if (k0 + n - 1 <= first) add_values(std::false_type{});
        else add_values(std::true_type{});
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float sum = l[i];
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(MG_FULL_MASK, sum, x);
        const int t = q0 + 4 * ty + i;
        if (t >= a.tokens) continue;
        const float inv = 1.0f / sum;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int d = HD == 32 ? 2 * tx + e : 4 * tx + (e & 3) + 64 * (e >> 2);
            store_split(a.out, t, head * HD + d, o[i][e] * inv);
        }
    }
}

template <int HD>
cudaError_t run_attn(const PromptAttn& a, cudaStream_t s) {
    prompt_attn_kernel<HD><<<dim3(a.n_heads, (a.tokens + kAttnQ - 1) / kAttnQ), 128, attn_smem<HD>(), s>>>(a);
    return cudaGetLastError();
}

template <int FMT, int NT>
cudaError_t allow_gemm() {
    return cudaFuncSetAttribute((const void*)prompt_gemm_kernel<FMT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmShape<FMT, NT>::bytes);
}
template <int HD>
cudaError_t allow_attn() {
    return cudaFuncSetAttribute((const void*)prompt_attn_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_smem<HD>());
}

}  // namespace

cudaError_t prompt_kernel_attrs() {
    const cudaError_t all[] = {allow_gemm<FMT_Q8_0, 64>(), allow_gemm<FMT_Q4_0, 64>(), allow_gemm<FMT_F16, 64>(), allow_gemm<FMT_Q8_0, 32>(),
                               allow_gemm<FMT_Q4_0, 32>(), allow_gemm<FMT_F16, 32>(), allow_attn<32>(), allow_attn<64>(), allow_attn<128>(),
                               cudaFuncSetAttribute((const void*)prompt_norm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPromptMaxWidth * 4)};
    for (cudaError_t e : all)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t launch_prompt_gemm(const PromptGemm& g, cudaStream_t s) {
    if (g.n_tile == 32) return g.fmt == FMT_Q8_0 ? run_gemm<FMT_Q8_0, 32>(g, s) : g.fmt == FMT_Q4_0 ? run_gemm<FMT_Q4_0, 32>(g, s) : run_gemm<FMT_F16, 32>(g, s);
    return g.fmt == FMT_Q8_0 ? run_gemm<FMT_Q8_0, 64>(g, s) : g.fmt == FMT_Q4_0 ? run_gemm<FMT_Q4_0, 64>(g, s) : run_gemm<FMT_F16, 64>(g, s);
}

cudaError_t launch_prompt_norm(const PromptNorm& a, int tokens, cudaStream_t s) {
    prompt_norm_kernel<<<tokens, 256, (size_t)a.out.width * 4, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_prompt_rope(const PromptRope& a, int tokens, cudaStream_t s) {
    prompt_rope_kernel<<<tokens, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_prompt_attn(const PromptAttn& a, int head_dim, cudaStream_t s) {
    return head_dim == 64 ? run_attn<64>(a, s) : head_dim == 128 ? run_attn<128>(a, s) : run_attn<32>(a, s);
}

cudaError_t launch_prompt_swiglu(const PieceSums& gu, const SplitRows& out, int tokens, cudaStream_t s) {
    prompt_swiglu_kernel<<<dim3((out.width + 255) / 256, tokens), 256, 0, s>>>(gu, out);
    return cudaGetLastError();
}

}  // namespace mg
