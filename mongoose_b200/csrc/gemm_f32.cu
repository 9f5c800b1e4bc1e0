// out = epilogue(A W^T) for fp32 A [n][K] and bf16 W [rows][K], with fp32's accuracy on the tensor cores: a value of A is
// the exact sum of three bf16 parts (8 + 8 + 8 bits of mantissa), a product of two bf16 values is exact in fp32, and the
// three parts' products meet in one accumulator, smallest first.  A sum in the tensor core runs over 64 columns; the
// epilogue adds it to fp32 registers, so the truncating accumulator stays at the level of one fp32 rounding.
// (The 64 x 64 tiles on the CUDA cores that this replaces left most SMs idle for a prompt's portion of a few dozen to a
// few hundred tokens and walked K sixteen columns at a time, each behind two barriers.)
//
// A CTA: 128 rows of W (the M side) x NT tokens.  Warp 0 copies W (TMA), warp 1 issues tcgen05.mma, warps 2 - 9 take the
// accumulators out of TMEM, warps 10 - 17 load A two steps ahead and store its parts as swizzled tiles.  Where tiles are
// fewer than SMs, the CTAs of a cluster share K, and each adds up its share of the tokens over the cluster, in order.
#include <algorithm>

#include "gemm_tc.h"
#include "layered_ops.cuh"
#include "umma.cuh"

namespace mg {

namespace {

constexpr int kThreads = 576;
constexpr int kAcc = 4;                 // accumulator slots in TMEM

struct Args {
    GemmF32 g;
    CUtensorMap w;                      // [matrix][rows][K] in boxes of 128 rows
    int steps;                          // steps of 64 columns per CTA
};

template <int NT>
struct Shape {
    static constexpr int w_bytes = 128 * 128, x_part = NT * 128, stage = w_bytes + 3 * x_part;
    static constexpr int stages = NT == 32 ? 6 : 5;
    static constexpr int bytes = stages * stage + 1024 + 256;
    static constexpr int values = NT / 4;           // of A per loading thread and step
};

__device__ __forceinline__ void tmem_load16_async(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void store_to_cta(uint32_t addr, int rank, float v) {
    asm volatile("{\n.reg .b32 p;\nmapa.shared::cluster.u32 p, %0, %1;\nst.shared::cluster.f32 [p], %2;\n}" ::"r"(addr), "r"(rank), "f"(v) : "memory");
}

__device__ __forceinline__ void finish(const GemmF32& g, int token, int row, float v) {
    if (token >= g.n || row >= g.rows) return;
    const size_t at = (size_t)token * g.ldc + row;
    if (g.epi == F32_GELU) v = gelu_tanh(v);
    else if (g.epi == F32_SILU_MUL) v *= silu(g.aux[at]);
    else if (g.epi == F32_DECAY) v = expf(-expf(v + g.bias[row]));
    g.out[at] = v;
}

// The thread's V values of row `token` from column k on; zeros past the tokens and the columns.
template <int V>
__device__ __forceinline__ void load_a(const GemmF32& g, int token, int k, float4 (&v)[V / 4]) {
    const float* p = g.A + (size_t)token * g.lda + k;
#pragma unroll
    for (int i = 0; i < V; i += 4) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (token < g.n) {
            if (k + i + 4 <= g.K) {
                t = __ldg(reinterpret_cast<const float4*>(p + i));
            } else {
                if (k + i < g.K) t.x = p[i];
                if (k + i + 1 < g.K) t.y = p[i + 1];
                if (k + i + 2 < g.K) t.z = p[i + 2];
            }
        }
        v[i / 4] = t;
    }
}

// Two values to three pairs of bf16 parts.  An infinity is its first part alone.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&o)[3]) {
#pragma unroll
    for (int p = 0; p < 3; p++) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        o[p] = *reinterpret_cast<const uint32_t*>(&b);
        const float hx = __uint_as_float(o[p] << 16), hy = __uint_as_float(o[p] & 0xffff0000u);
        x = fabsf(hx) == INFINITY ? 0.f : x - hx;
        y = fabsf(hy) == INFINITY ? 0.f : y - hy;
    }
}

template <int NT>
__global__ void __launch_bounds__(kThreads, 1) gemm_f32_kernel(const __grid_constant__ Args a) {
    using S = Shape<NT>;
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_w = reinterpret_cast<uint64_t*>(base + S::stages * S::stage);
    uint64_t* full_x = full_w + S::stages;
    uint64_t* empty = full_x + S::stages;
    uint64_t* acc_full = empty + S::stages;
    uint64_t* acc_empty = acc_full + kAcc;
    uint64_t* done = acc_empty + kAcc;
    uint32_t* tmem_base = reinterpret_cast<uint32_t*>(done + 1);

    const GemmF32& g = a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * 128, tok0 = blockIdx.y * NT, parts = gridDim.z;
    int matrix = 0;
    if (g.group) {
        matrix = g.group[tok0 / 128];
        if (matrix < 0) return;                     // the whole cluster: it shares the tokens
    }
    const int step0 = blockIdx.z * a.steps, kt = max(0, min(a.steps, (g.K + 63) / 64 - step0));

    if (threadIdx.x == 0) {
        for (int i = 0; i < S::stages; i++) { bar_init(full_w + i, 1); bar_init(full_x + i, 8); bar_init(empty + i, 1); }
        for (int i = 0; i < kAcc; i++) { bar_init(acc_full + i, 1); bar_init(acc_empty + i, 8); }
        bar_init(done, 1);
        bar_init_fence();
        tma_prefetch_map(&a.w);
    }
    if (warp == 1) tmem_alloc(tmem_base, kAcc * NT);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t acc = *tmem_base;

    constexpr int C = NT / 2;                       // tokens per epilogue thread
    const int quarter = warp & 3, half = (warp - 2) >> 2, row = quarter * 32 + lane;
    float sum[C];
#pragma unroll
    for (int i = 0; i < C; i++) sum[i] = 0.f;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < kt; i++) {
                const int s = i % S::stages, use = i / S::stages;
                if (use > 0 && !bar_wait(empty + s, (use - 1) & 1, g.status)) break;
                bar_expect(full_w + s, S::w_bytes);
                tma_load_3d(base + s * S::stage, &a.w, (step0 + i) * 64, row0, matrix, full_w + s);
                issued = i + 1;
            }
            // no copy may be in flight when the CTA leaves
            for (int i = max(0, issued - S::stages); i < issued; i++) bar_wait(full_w + i % S::stages, (i / S::stages) & 1, g.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            for (int i = 0; i < kt; i++) {
                const int s = i % S::stages, b = i % kAcc;
                if (i >= kAcc && !bar_wait(acc_empty + b, (i / kAcc - 1) & 1, g.status)) break;
                if (!bar_wait(full_w + s, (i / S::stages) & 1, g.status) || !bar_wait(full_x + s, (i / S::stages) & 1, g.status)) break;
                tc_fence_after();
                uint8_t* st = base + s * S::stage;
                const uint64_t dw = tile_desc(st);
#pragma unroll
                for (int p = 2; p >= 0; p--) {
                    const uint64_t dx = tile_desc(st + S::w_bytes + p * S::x_part);
#pragma unroll
                    for (int k = 0; k < 4; k++) mma_bf16(acc + b * NT, dw + 2 * k, dx + 2 * k, mma_desc(NT), p < 2 || k > 0);
                }
                mma_commit(empty + s);
                mma_commit(acc_full + b);
            }
            // nothing may be in flight when the accumulators are given back
            mma_commit(done);
            bar_wait(done, 0, g.status);
        }
        __syncwarp();
    } else if (warp < 10) {
        for (int i = 0; i < kt; i++) {
            const int b = i % kAcc;
            if (!__all_sync(MG_FULL_MASK, bar_wait(acc_full + b, (i / kAcc) & 1, g.status))) break;
            tc_fence_after();
            uint32_t v[C / 16][16];
#pragma unroll
            for (int c = 0; c < C / 16; c++) tmem_load16_async(acc + ((uint32_t)(quarter * 32) << 16) + b * NT + half * C + c * 16, v[c]);
            tmem_wait_load();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(acc_empty + b);
#pragma unroll
            for (int c = 0; c < C; c++) sum[c] += __uint_as_float(v[c / 16][c % 16]);
        }
        if (parts == 1) {
#pragma unroll
            for (int i = 0; i < C; i++) finish(g, tok0 + half * C + i, row0 + row, sum[i]);
        }
        tc_fence_before();
    } else {
        constexpr int V = S::values, per = 64 / V;          // threads per row
        const int t = threadIdx.x - 320, r = t / per, c = t % per;
        const bool bend = g.epi == F32_DECAY;
        float4 v0[V / 4], v1[V / 4], v2[V / 4];
        load_a<V>(g, tok0 + r, step0 * 64 + c * V, v0);
        load_a<V>(g, tok0 + r, (step0 + 1) * 64 + c * V, v1);
        for (int i = 0; i < kt; i++) {
            const int s = i % S::stages, use = i / S::stages;
            load_a<V>(g, tok0 + r, (step0 + i + 2) * 64 + c * V, v2);
            if (use > 0 && !__all_sync(MG_FULL_MASK, bar_wait(empty + s, (use - 1) & 1, g.status))) break;
            uint8_t* tile = base + s * S::stage + S::w_bytes + r * 128;
#pragma unroll
            for (int q = 0; q < V / 8; q++) {
                const float x[8] = {v0[2 * q].x, v0[2 * q].y, v0[2 * q].z, v0[2 * q].w, v0[2 * q + 1].x, v0[2 * q + 1].y, v0[2 * q + 1].z, v0[2 * q + 1].w};
                uint32_t o[4][3];
#pragma unroll
                for (int k = 0; k < 4; k++) split_pair(bend ? tanhf(x[2 * k]) : x[2 * k], bend ? tanhf(x[2 * k + 1]) : x[2 * k + 1], o[k]);
                const int at = ((c * (V / 8) + q) ^ (r & 7)) << 4;
#pragma unroll
                for (int p = 0; p < 3; p++) *reinterpret_cast<uint4*>(tile + p * S::x_part + at) = make_uint4(o[0][p], o[1][p], o[2][p], o[3][p]);
            }
            async_proxy_fence();
            __syncwarp();
            if (lane == 0) bar_arrive(full_x + s);
#pragma unroll
            for (int j = 0; j < V / 4; j++) { v0[j] = v1[j]; v1[j] = v2[j]; }
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(acc, kAcc * NT);
    if (parts == 1) return;

    // CTA p of the cluster adds up tokens [p * share, (p + 1) * share); the rings are free once every CTA is here
    const int share = NT / parts;
    float* mail = reinterpret_cast<float*>(base);   // [sender][token of the share][row]
    cluster_sync();
    if (warp >= 2 && warp < 10) {
#pragma unroll
        for (int i = 0; i < C; i++) {
            const int t = half * C + i, to = t / share;
            store_to_cta(smem_addr(mail + ((size_t)blockIdx.z * share + t - to * share) * 128 + row), to, sum[i]);
        }
    }
    cluster_sync();
    for (int i = threadIdx.x; i < share * 128; i += kThreads) {
        float v = mail[i];
        for (int q = 1; q < parts; q++) v += mail[(size_t)q * share * 128 + i];
        finish(g, tok0 + blockIdx.z * share + i / 128, row0 + i % 128, v);
    }
}

template <int NT>
cudaError_t run(const Args& a, int parts, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((a.g.rows + 127) / 128, (a.g.n + NT - 1) / NT, parts);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Shape<NT>::bytes;
    cfg.stream = s;
    cudaLaunchAttribute cluster[1];
    cluster[0].id = cudaLaunchAttributeClusterDimension;
    cluster[0].val.clusterDim.x = 1;
    cluster[0].val.clusterDim.y = 1;
    cluster[0].val.clusterDim.z = (unsigned)parts;
    cfg.attrs = cluster;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gemm_f32_kernel<NT>, a);
}

}  // namespace

cudaError_t gemm_f32_attrs() {
    if (cudaError_t c = allow_smem(gemm_f32_kernel<32>, Shape<32>::bytes)) return c;
    return allow_smem(gemm_f32_kernel<64>, Shape<64>::bytes);
}

cudaError_t launch_gemm_f32(const GemmF32& g, cudaStream_t s) {
    Args a{};
    a.g = g;
    if (!make_tile_map(&a.w, g.W, g.ldw, g.rows, g.group ? g.groups : 1, g.ldw, g.group ? g.group_stride : (long long)g.rows * g.ldw, 128))
        return cudaErrorInvalidValue;
    const int nt = g.n <= 32 ? 32 : 64, tiles = (g.rows + 127) / 128 * ((g.n + nt - 1) / nt), steps = (g.K + 63) / 64;
    int parts = 1;
    while (parts < 8 && tiles * parts * 2 <= sm_count() && steps >= 3 * parts * 2) parts *= 2;
    a.steps = (steps + parts - 1) / parts;
    return nt == 32 ? run<32>(a, parts, s) : run<64>(a, parts, s);
}

}  // namespace mg
