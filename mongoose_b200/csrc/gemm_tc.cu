// out = A B^T for bf16 A [m][k] and B [n][k], fp32 accumulation.  One CTA per SM walks tiles of 128 x BN: warp 0 streams both
// operands with TMA into a ring of 64-column stages that runs on from tile to tile, one thread of warp 1 issues
// tcgen05.mma into one of two accumulators in TMEM, warps 2-9 read the other back and store it row by row through
// shared memory.  A tile's first copies and its results are thus hidden behind the products of its neighbours;
// with a CTA per tile (two to an SM) they were a third of the time.  What bounds a product is how often its operands come
// from L2, (128 + BN) x 128 bytes for 128 x BN x 64 products, so the widest tile that keeps the SMs busy is taken.
// B200: the 31 products of a 2048-token prompt at 1.1B widths (six layers) 1403 -> 1190 us, 0.92 PFLOP/s on average; the
// 118 of a 1500-token one in two portions, whose tiles are few, 2711 -> 2409 us.
#include "gemm_tc.h"
#include "layered_ops.cuh"
#include "umma.cuh"

namespace mg {

namespace {

constexpr int kThreads = 320;
constexpr int kEpiWarps = 8;

// gelu for results that are rounded to bf16: tanh from one fast exponential
__device__ __forceinline__ float gelu_tanh_fast(float z) {
    const float u = 0.7978845608028654f * (z + 0.044715f * z * z * z);
    return z - z * __fdividef(1.0f, 1.0f + __expf(2.0f * u));
}

__device__ __forceinline__ float silu_fast(float z) { return z * __fdividef(1.0f, 1.0f + __expf(-z)); }

template <int BN>
struct Geo {
    static constexpr int a_bytes = 128 * 128, b_bytes = BN * 128, stage = a_bytes + b_bytes;
    static constexpr int stages = BN == 256 ? 4 : BN == 128 ? 6 : 8;
    static constexpr int rows = kEpiWarps * 32 * 33 * 4;            // a 32 x 32 piece per epilogue warp
    static constexpr int bytes = stages * stage + rows + 1024 + 256;
};

struct Tile {
    int col0, row0, z, zb, kt;
};

// Tile t in the order columns, rows, batches; false: it has no matrix.
template <int BN>
__device__ __forceinline__ bool tile_at(const GemmTC& g, int t, int gx, int gy, Tile* o) {
    const int x = t % gx, yz = t / gx, y = yz % gy;
    o->z = yz / gy;
    o->col0 = x * (g.mode == GEMM_SILU_BF16 ? BN / 2 : BN);
    o->row0 = y * 128;
    o->zb = o->z / g.b_group;
    if (g.group && (o->zb = g.group[y]) < 0) return false;
    o->kt = (g.k + 63) / 64;
    if (g.causal_pos0 >= 0) o->kt = min(o->kt, (g.causal_pos0 + min(o->row0 + 128, g.m) + 63) / 64);
    return true;
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_kernel(const __grid_constant__ GemmTC g, int gx, int gy, int tiles) {
    using G = Geo<BN>;
    constexpr int kStages = G::stages;
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    float* pieces = reinterpret_cast<float*>(base + kStages * G::stage);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + kStages * G::stage + G::rows);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* done = acc_empty + 2;
    uint32_t* tmem_base = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool dual = g.mode == GEMM_SILU_BF16;
    Tile t;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; i++) { bar_init(full + i, 1); bar_init(empty + i, 1); }
        for (int i = 0; i < 2; i++) { bar_init(acc_full + i, 1); bar_init(acc_empty + i, kEpiWarps); }
        bar_init(done, 1);
        bar_init_fence();
        tma_prefetch_map(&g.a);
        tma_prefetch_map(&g.b);
        if (dual) tma_prefetch_map(&g.b2);
    }
    if (warp == 1) tmem_alloc(tmem_base, 2 * BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // behind the allocation of TMEM: a dependent that took its share first would wait for this kernel, and this one for it
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t acc = *tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            int n = 0, s = 0, par = 1;          // copies issued, their stage, parity of the wait for its last use
            bool ok = true;
            for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
                if (!tile_at<BN>(g, i, gx, gy, &t)) continue;
                for (int k = 0; k < t.kt; k++) {
                    if (n >= kStages && !(ok = bar_wait(empty + s, par, g.status))) break;
                    bar_expect(full + s, G::stage);
                    uint8_t* st = base + s * G::stage;
                    tma_load_3d(st, &g.a, k * 64, t.row0, t.z, full + s);
                    tma_load_3d(st + G::a_bytes, &g.b, (g.b_steps ? k % g.b_steps : k) * 64, t.col0, t.zb, full + s);
                    if (dual) tma_load_3d(st + G::a_bytes + G::b_bytes / 2, &g.b2, k * 64, t.col0, t.zb, full + s);
                    n++;
                    if (++s == kStages) { s = 0; par ^= 1; }
                }
            }
            // no copy may be in flight when the CTA leaves
            for (int i = max(0, n - kStages); i < n; i++) bar_wait(full + i % kStages, (i / kStages) & 1, g.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            int n = 0, s = 0, par = 0;
            bool ok = true;
            for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
                if (!tile_at<BN>(g, i, gx, gy, &t)) continue;
                const int b = n & 1;
                if (n >= 2 && !(ok = bar_wait(acc_empty + b, ((n >> 1) - 1) & 1, g.status))) break;
                tc_fence_after();
                for (int k = 0; k < t.kt; k++) {
                    if (!(ok = bar_wait(full + s, par, g.status))) break;
                    tc_fence_after();
                    const uint64_t da = tile_desc(base + s * G::stage), db = tile_desc(base + s * G::stage + G::a_bytes);
#pragma unroll
                    for (int q = 0; q < 4; q++) mma_bf16(acc + b * BN, da + 2 * q, db + 2 * q, mma_desc(BN), k > 0 || q > 0);
                    mma_commit(empty + s);
                    if (++s == kStages) { s = 0; par ^= 1; }
                }
                mma_commit(acc_full + b);
                n++;
            }
            // nothing may be in flight when the accumulators are given back
            mma_commit(done);
            bar_wait(done, 0, g.status);
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        float* tile = pieces + (warp - 2) * 32 * 33;
        int n = 0;
        for (int i = blockIdx.x; i < tiles; i += gridDim.x) {
            if (!tile_at<BN>(g, i, gx, gy, &t)) continue;
            const int b = n & 1;
            if (!__all_sync(MG_FULL_MASK, bar_wait(acc_full + b, (n >> 1) & 1, g.status))) break;
            n++;
            tc_fence_after();
            const uint32_t from = acc + ((uint32_t)(quarter * 32) << 16) + b * BN;
#pragma unroll 1
            for (int c = half * 32; c < (dual ? BN / 2 : BN) && t.col0 + c < g.n; c += 64) {
                float v[32];
                tmem_load32(from + c, v);
                if (dual) {
                    float u[32];
                    tmem_load32(from + BN / 2 + c, u);
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = silu_fast(v[j]) * u[j];
                }
#pragma unroll
                for (int j = 0; j < 32; j++) tile[lane * 33 + j] = v[j];
                __syncwarp();
                if (g.mode == GEMM_F32 || g.mode == GEMM_DECAY_F32) {
                    const int col = t.col0 + c + lane;
                    float* out = static_cast<float*>(g.out) + t.z * g.batch_c + col;
                    const float bias = g.mode == GEMM_DECAY_F32 && col < g.n ? g.bias[col] : 0.f;
#pragma unroll 8
                    for (int r = 0; r < 32; r++) {
                        const int row = t.row0 + quarter * 32 + r;
                        float x = tile[r * 33 + lane];
                        if (g.mode == GEMM_DECAY_F32) x = expf(-expf(x + bias));
                        if (row < g.m && col < g.n) out[row * g.ldc] = x;
                    }
                } else {                            // two columns per lane, two rows at a time
                    const int col = t.col0 + c + 2 * (lane & 15);
                    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(g.out) + t.z * g.batch_c + col;
                    const bool pair = (reinterpret_cast<uintptr_t>(out) & 3) == 0 && (g.ldc & 1) == 0 && col + 1 < g.n;
#pragma unroll 4
                    for (int r = lane >> 4; r < 32; r += 2) {
                        const int row = t.row0 + quarter * 32 + r;
                        float x = tile[r * 33 + 2 * (lane & 15)], y = tile[r * 33 + 2 * (lane & 15) + 1];
                        if (g.mode == GEMM_GELU_BF16) { x = gelu_tanh_fast(x); y = gelu_tanh_fast(y); }
                        if (row >= g.m) break;
                        if (pair) {
                            *reinterpret_cast<__nv_bfloat162*>(out + row * g.ldc) = __floats2bfloat162_rn(x, y);
                        } else {
                            if (col < g.n) out[row * g.ldc] = __float2bfloat16_rn(x);
                            if (col + 1 < g.n) out[row * g.ldc + 1] = __float2bfloat16_rn(y);
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(acc_empty + b);
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(acc, 2 * BN);
}

typedef CUresult (*encode_fn_t)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_fn_t encode_fn() {
    static encode_fn_t fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return (encode_fn_t)p;
    }();
    return fn;
}

bool encode(CUtensorMap* map, const void* base, const cuuint64_t dims[3], const cuuint64_t strides[2], const cuuint32_t box[3],
            CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
    const cuuint32_t ones[3] = {1, 1, 1};
    encode_fn_t fn = encode_fn();
    return fn && fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, ones,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
cudaError_t run(const GemmTC& g, bool pdl, cudaStream_t s) {
    const int cols = g.mode == GEMM_SILU_BF16 ? BN / 2 : BN, gx = (g.n + cols - 1) / cols, gy = (g.m + 127) / 128, tiles = gx * gy * g.batch;
    return launch_pdl(gemm_tc_kernel<BN>, tiles < sm_count() ? tiles : sm_count(), kThreads, Geo<BN>::bytes, pdl, s, g, gx, gy, tiles);
}

}  // namespace

bool make_tile_map(CUtensorMap* map, const void* base, int k, int rows, int batch, long long row_stride, long long batch_stride, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, (cuuint64_t)batch};
    const cuuint64_t strides[2] = {(cuuint64_t)row_stride * 2, (cuuint64_t)batch_stride * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    return encode(map, base, dims, strides, box);
}

bool make_head_map(CUtensorMap* map, const void* base, int k, int batch, int rows, long long batch_stride, long long row_stride, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)batch, (cuuint64_t)rows};
    const cuuint64_t strides[2] = {(cuuint64_t)batch_stride * 2, (cuuint64_t)row_stride * 2};
    const cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows};
    return encode(map, base, dims, strides, box);
}

bool make_rows_map(CUtensorMap* map, const void* base, int row_len, int rows, int batch, int box_cols, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)row_len, (cuuint64_t)rows, (cuuint64_t)batch};
    const cuuint64_t strides[2] = {(cuuint64_t)row_len * 2, (cuuint64_t)rows * row_len * 2};
    const cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
    return encode(map, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

int gemm_tc_bn(int m, int n, int batch) {
    if (n <= 64) return 64;
    // Rounds of tiles over the SMs, times what a tile of each width takes.  Measured on B200, 2048 columns of K: 11.5, 13.5 and 18.9 us where
    // a CTA walks several tiles, 12, 15.5 and 24.4 where it has one, whose copies and results nothing hides.  Over the 504 products
    // of prompts of 128 to 2048 tokens of six models the choices take 17.5 ms and the best ones 17.1; the furthest off are
    // gated products of experts (75 us for 51), whose row tiles are counted as if every expert's last one were used.
    const int rows = (m + 127) / 128 * batch;
    int best = 64;
    float least = 0.f;
    for (int bn : {64, 128, 256}) {
        const int tiles = (n + bn - 1) / bn * rows;
        const float t = (float)((tiles + sm_count() - 1) / sm_count()) * (bn == 64 ? 1.0f : bn == 128 ? 1.4f : 2.2f);
        if (bn == 64 || t < least) { best = bn; least = t; }
    }
    return best;
}

cudaError_t gemm_tc_attrs() {
    if (cudaError_t c = allow_smem(gemm_tc_kernel<64>, Geo<64>::bytes)) return c;
    if (cudaError_t c = allow_smem(gemm_tc_kernel<128>, Geo<128>::bytes)) return c;
    return allow_smem(gemm_tc_kernel<256>, Geo<256>::bytes);
}

cudaError_t launch_gemm_tc(const GemmTC& g, bool pdl, cudaStream_t s) {
    if (g.bn == 64 && g.mode != GEMM_SILU_BF16) return run<64>(g, pdl, s);
    if (g.bn == 128) return run<128>(g, pdl, s);
    if (g.bn == 256) return run<256>(g, pdl, s);
    return cudaErrorInvalidValue;
}

}  // namespace mg
