// Matvecs on caller-owned RAW quantized blocks (GGUF Q4_0 18-byte blocks,
// Q8_0 34-byte blocks), the int8-activation (dp4a) family, and the fused
// per-token dispatch over caller-owned buffers.
//
// The Go side declares these entry points (kernels.go:62-67, 206-211;
// cuda_graph.go:211-234) but the reference ships no source for them; the
// block layout is the one cuda_q4_0.go:13-17 uploads.  Raw blocks are only
// 2-byte aligned; the engine (mg_*) re-packs blocks at upload and does not
// use this file's kernels.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "../../include/mongoose_kernels.h"
#include "mg_common.cuh"

using namespace mg;

namespace {

struct __align__(8) ActBlock {   // 40 bytes per 32 activations
    float d;                     // amax / 127
    float s;                     // d * sum(q)
    int8_t q[32];
};
static_assert(sizeof(ActBlock) == 40, "activation block is 40 bytes");

// ---------------- fp32-activation matvecs on raw blocks ----------------
// Raw GGUF blocks (34 / 18 bytes) are only 2-byte aligned, so a lane cannot fetch its block with a
// vector load.  Instead a warp takes a CHUNK of 32 consecutive blocks of a row - a contiguous byte
// range - and copies the aligned 16-byte pieces that cover it into a ring of its own in shared memory
// (cp.async, kRawStages deep, running on over chunks and rows, so that a row's end does not drain it);
// each lane then pulls the words of ITS block out of shared memory, re-aligns them with a funnel shift
// by 16 or 32 bits, and multiplies them with the activation slice staged once per CTA.  A warp takes R
// rows at a time, which share the activation reads; where rows are fewer than warps, `ks` warps share
// a row and their sums meet in shared memory, in order.
//
// Two chunks per row are under way while a third is multiplied.  The activation slices of a warp's lanes
// are 36 floats apart: 32 floats apart, all lanes of an access fell on the same four banks and the reads
// alone took 60 of 104 us of a 3584 x 18944 Q4_0 product.
constexpr int kRawStages = 3;
constexpr int kXStride = 36;                                // floats between the activation slices of two blocks
// Where the kernel reads activations: slices kXStride apart; slices without gaps, the eight 16-byte pieces of block b in the
// order of piece ^ (b mod 8), which takes a ninth less room and an instruction per read; global memory.
enum RawInput : int { RAW_PADDED, RAW_SWIZZLED, RAW_GLOBAL };
__host__ __device__ constexpr int block_bytes(int fmt) { return fmt == FMT_Q8_0 ? 34 : 18; }
__host__ __device__ constexpr int chunk_ring(int fmt) { return 32 * block_bytes(fmt) + 16; }        // bytes: whole pieces cover a chunk, whatever its alignment

// Copies bytes [src, src + n) so that they start at dst + (address of src mod V); nothing behind them is read.
template <int V>
__device__ __forceinline__ void copy_chunk(uint8_t* dst, const uint8_t* src, int n, int lane) {
    const int lead = (int)(reinterpret_cast<uintptr_t>(src) & (V - 1));
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    for (int i = lane * V; i < lead + n; i += 32 * V) {
        const int left = min(V, lead + n - i);
        if (V == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + i), "l"(src - lead + i), "r"(left) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + i), "l"(src - lead + i), "r"(left) : "memory");
    }
}

// V: bytes per copy; 16 where the matrix starts on a 16-byte boundary (so no piece starts before it), else 4.
// X: where the activations are (RawInput).  ks: warps per row.
template <int FMT, int R, int V, int X>
__global__ void __launch_bounds__(512) raw_block_matvec_kernel(const float* __restrict__ act, const uint8_t* __restrict__ w, float* out, int N,
                                                               int K, int ks) {
    constexpr int BB = block_bytes(FMT), QW = FMT == FMT_Q8_0 ? 8 : 4;       // bytes, 4-byte words of quants per block
    constexpr int ring = chunk_ring(FMT);
    extern __shared__ __align__(16) float raw_xs[];         // activation slices, 16 R partial sums, then the rings
    const int nb = K / 32, chunks = (nb + 31) / 32;
    float* sums = raw_xs + (size_t)nb * (X == RAW_PADDED ? kXStride : X == RAW_SWIZZLED ? 32 : 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint8_t* stage = reinterpret_cast<uint8_t*>(sums + 16 * R) + (size_t)warp * kRawStages * R * ring;
    const int slots = warps / ks, slot = warp / ks, part = warp - slot * ks;
    const int tiles = (N + R - 1) / R;
    const int mine = blockIdx.x < tiles ? (tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;        // tiles of this CTA
    const int rounds = (mine + slots - 1) / slots;
    pdl_launch_dependents();
    pdl_wait();

    int iround = 0, ichunk = part;                          // the next chunk to be copied
    auto issue = [&](int s) {
        const int k = iround * slots + slot;
        if (k < mine) {
            const int row0 = (blockIdx.x + k * gridDim.x) * R, n = min(32, nb - ichunk * 32) * BB;
#pragma unroll
            for (int r = 0; r < R; r++)
                if (row0 + r < N) copy_chunk<V>(stage + (s * R + r) * ring, w + ((size_t)(row0 + r) * nb + ichunk * 32) * BB, n, lane);
            ichunk += ks;
            if (ichunk >= chunks) { ichunk = part; iround++; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < kRawStages - 1; s++) issue(s);

    if (X != RAW_GLOBAL) {
        auto place = [&](int b, int piece) {                // four floats of block b
            return raw_xs + (X == RAW_PADDED ? b * kXStride + piece * 4 : b * 32 + (piece ^ (b & 7)) * 4);
        };
        if ((reinterpret_cast<uintptr_t>(act) & 15) == 0) {
#pragma unroll 4
            for (int i = threadIdx.x; i < nb * 8; i += blockDim.x) *reinterpret_cast<float4*>(place(i >> 3, i & 7)) = reinterpret_cast<const float4*>(act)[i];
        } else {
            for (int i = threadIdx.x; i < K; i += blockDim.x) place(i >> 5, (i & 31) >> 2)[i & 3] = act[i];
        }
        __syncthreads();
    }

    int s = 0;
    for (int round = 0; round < rounds; round++) {
        const int k = round * slots + slot;
        const bool has = k < mine;
        const int row0 = (blockIdx.x + k * gridDim.x) * R;
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.f;
        for (int c = part; has && c < chunks; c += ks) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRawStages - 2) : "memory");
            __syncwarp();
            const int b = c * 32 + lane;
            if (b < nb) {
                uint32_t q[R][QW];
                float d[R], sum[R];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const int row = min(row0 + r, N - 1);
                    const int off = (int)(reinterpret_cast<uintptr_t>(w + ((size_t)row * nb + c * 32) * BB) & (V - 1)) + lane * BB;
                    const uint32_t* p = reinterpret_cast<const uint32_t*>(stage + (s * R + r) * ring) + (off >> 2);
                    const int sh = (off & 2) ? 32 : 16;                 // quants start 2 bytes after the scale
                    uint32_t lo = p[0];
                    d[r] = half_bits_to_float((unsigned short)((off & 2) ? (lo >> 16) : (lo & 0xffffu)));
#pragma unroll
                    for (int i = 0; i < QW; i++) {
                        // the word behind a block that ends on a word's end is another's, or was never written: it is shifted out
                        const uint32_t hi = p[i + 1];
                        q[r][i] = __funnelshift_rc(lo, hi, sh);
                        lo = hi;
                    }
                    sum[r] = 0.f;
                }
                const float* xb = X == RAW_PADDED ? raw_xs + b * kXStride : X == RAW_SWIZZLED ? raw_xs + b * 32 : act + (size_t)b * 32;
                auto x4 = [&](int i) {
                    if (X == RAW_GLOBAL) return make_float4(xb[4 * i], xb[4 * i + 1], xb[4 * i + 2], xb[4 * i + 3]);
                    return *reinterpret_cast<const float4*>(xb + 4 * (X == RAW_PADDED ? i : i ^ (lane & 7)));
                };
                if (FMT == FMT_Q8_0) {
#pragma unroll
                    for (int i = 0; i < QW; i++) {
                        const float4 x = x4(i);
#pragma unroll
                        for (int r = 0; r < R; r++) sum[r] = dot4_s8(q[r][i], x, sum[r]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < QW; i++) {                      // low nibbles: elements 4i .., high ones: 16 + 4i ..
                        const float4 x = x4(i), y = x4(4 + i);
#pragma unroll
                        for (int r = 0; r < R; r++) sum[r] = dot4_u4(q[r][i] >> 4 & 0x0f0f0f0fu, y, dot4_u4(q[r][i] & 0x0f0f0f0fu, x, sum[r]));
                    }
                }
#pragma unroll
                for (int r = 0; r < R; r++) acc[r] = fmaf(d[r], sum[r], acc[r]);
            }
            __syncwarp();
            issue(s == 0 ? kRawStages - 1 : s - 1);
            s = s == kRawStages - 1 ? 0 : s + 1;
        }
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = warp_sum(acc[r]);
        if (ks == 1) {
            if (lane == 0 && has) {
#pragma unroll
                for (int r = 0; r < R; r++)
                    if (row0 + r < N) out[row0 + r] = acc[r];
            }
            continue;
        }
        if (round > 0) __syncthreads();                     // the last round's sums have been read
        if (lane == 0) {
#pragma unroll
            for (int r = 0; r < R; r++) sums[warp * R + r] = acc[r];
        }
        __syncthreads();
        if (lane == 0 && part == 0 && has) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                float v = 0.f;
                for (int p = 0; p < ks; p++) v += sums[(warp + p) * R + r];
                if (row0 + r < N) out[row0 + r] = v;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------- activation quantizer: one warp per block of 32 ----------------
__global__ void __launch_bounds__(256) quantize_act_kernel(const float* __restrict__ act, ActBlock* out,
                                                          int nblocks_total) {
    const int lane = threadIdx.x & 31;
    const int blk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (blk >= nblocks_total) return;
    const float v = act[(size_t)blk * 32 + lane];
    const float amax = warp_max(fabsf(v));
    const float d = amax / 127.0f;
    const int q = amax > 0.f ? __float2int_rn(v / d) : 0;
    int sum = q;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(MG_FULL_MASK, sum, o);
    out[blk].q[lane] = (int8_t)q;
    if (lane == 0) {
        out[blk].d = d;
        out[blk].s = d * (float)sum;
    }
}

// ---------------- Q4_0 x int8 activations, integer dot products ----------------
// out[b][row] = sum_blocks d_w * (d_a * sum_j nib_j * qa_j - 8 * s_a)
__global__ void __launch_bounds__(256) q4_0_dp4a_kernel(const uint8_t* __restrict__ w,
                                                       const ActBlock* __restrict__ q8, float* out, int N, int K,
                                                       int B) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= N) return;
    const int nb = K / 32;
    const uint8_t* wr = w + (size_t)row * nb * 18;
    for (int bi = 0; bi < B; bi++) {
        const ActBlock* qa = q8 + (size_t)bi * nb;
        float acc = 0.f;
        for (int b = lane; b < nb; b += 32) {
            const unsigned short* p = reinterpret_cast<const unsigned short*>(wr + (size_t)b * 18);
            const float dw = half_bits_to_float(p[0]);
            const int* aq = reinterpret_cast<const int*>(qa[b].q);
            int sumi = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t word = (uint32_t)p[1 + 2 * i] | ((uint32_t)p[2 + 2 * i] << 16);
                const int lo = (int)(word & 0x0f0f0f0fu), hi = (int)((word >> 4) & 0x0f0f0f0fu);
                sumi = __dp4a(lo, aq[i], sumi);
                sumi = __dp4a(hi, aq[4 + i], sumi);
            }
            acc = fmaf(dw, qa[b].d * (float)sumi - 8.0f * qa[b].s, acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) out[(size_t)bi * N + row] = acc;
    }
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// ---- scratch that lives in the library image, for callers that must not allocate ----
// 40 bytes per 32 activations; 32768 input features at most.
constexpr int kStaticMaxK = 32768;
constexpr size_t kStaticScratchBytes = (size_t)(kStaticMaxK / 32) * sizeof(ActBlock);
static __device__ __align__(256) unsigned char g_static_act_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_ptr[kMaxDevices] = {};      // device address of g_static_act_scratch on each device
thread_local char g_static_err[256] = "";

int static_fail(int code, const char* fmt, int a, int b) {
    snprintf(g_static_err, sizeof g_static_err, fmt, a, b);
    return code;
}

// Two rows per warp where every warp has a row; where tiles are fewer than warps, several warps share a row (pair) each.  CTAs
// of 8 warps, three per SM (two where no more fit: Q8_0 8192 x 5376 19 us, 29 with a third left for a second round), while the activations are small; wide inputs, whose copy a CTA's warps share, take one
// CTA of 16, and those that do not fit beside its rings take, in this order, slices without gaps, single rows and 8 warps: Q8_0
// from 27872 columns on (39648 where rows are single anyway), Q4_0 from 38784 (45120); beyond 51200 (54272) the
// activations stay in global memory.
// Measured on B200, weights in no cache, activations read from global memory / from such slices: Q8_0 8192 x 28672 573 / 74 us, 8192 x
// 40960 817 / 112 us, 256 x 32768 99 / 7 us.  Elsewhere: 4864 x 896 Q8_0 4.7 us (the launch), 18944 x 3584 Q8_0 27 us = 2.7 TB/s;
// at 18944 columns of Q8_0, 2368 rows 17 us (two warps a pair), 2400 to 4736 rows 27 to 29 us (the walk of one warp over its pair).
struct RawShape {
    int grid, threads, ks, input;
    bool pairs;
    size_t smem;
};
constexpr size_t kRawSmem = 226 * 1024, kSmSmem = 228 * 1024;      // of a CTA; of an SM, 1 KB of it for each CTA

template <int FMT>
RawShape raw_shape(int N, int K, int sms) {
    RawShape p{};
    const int nb = K / 32, chunks = cdiv(nb, 32);
    size_t x = (size_t)nb * kXStride * 4;
    auto rest = [&](int warps, int R) { return (size_t)16 * R * 4 + (size_t)warps * kRawStages * R * chunk_ring(FMT); };
    const bool wide = x > 24 * 1024;
    int warps = wide ? 16 : 8, most = sms * (wide ? 1 : 3);
    p.pairs = N >= most * warps;
    if (x + rest(warps, p.pairs ? 2 : 1) > kRawSmem) {
        p.input = RAW_SWIZZLED;
        x = (size_t)K * 4;
        if (x + rest(warps, p.pairs ? 2 : 1) > kRawSmem) p.pairs = false;
        if (x + rest(warps, 1) > kRawSmem) warps = 8;
        if (x + rest(warps, 1) > kRawSmem) { p.input = RAW_GLOBAL; x = 0; most = sms * 3; p.pairs = N >= most * warps; }
    }
    const int R = p.pairs ? 2 : 1, tiles = cdiv(N, R);
    p.smem = x + rest(warps, R);
    most = std::min(most, sms * (int)(kSmSmem / (p.smem + 1024)));         // no second round of CTAs
    p.ks = 1;
    while (2 * p.ks <= warps && 2 * p.ks <= chunks && (long long)tiles * 2 * p.ks <= (long long)most * warps) p.ks *= 2;
    p.grid = std::min(cdiv(tiles, warps / p.ks), most);
    p.threads = warps * 32;
    return p;
}

template <int FMT, int R, int V, int X>
void run_raw_matvec(const RawShape& p, int dev, const float* act, const uint8_t* w, float* out, int N, int K, cudaStream_t stream) {
    auto kern = raw_block_matvec_kernel<FMT, R, V, X>;
    static std::atomic<bool> raised[kMaxDevices];
    if (p.smem > 48 * 1024 && !(dev < kMaxDevices && raised[dev].load(std::memory_order_relaxed))) {
        cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (dev < kMaxDevices) raised[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];        // a launch may begin while the one before it ends; the kernel waits before it reads
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, act, w, out, N, K, p.ks);
}

template <int FMT>
void launch_raw_matvec(const float* act, const void* w_blocks, float* out, int N, int K, cudaStream_t stream) {
    if (N <= 0 || K < 32 || K % 32) return;
    static std::atomic<int> sm_count[kMaxDevices];
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (dev < kMaxDevices) sms = sm_count[dev].load(std::memory_order_relaxed);
    if (sms <= 0) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
        if (dev < kMaxDevices) sm_count[dev].store(sms, std::memory_order_relaxed);
    }
    const RawShape p = raw_shape<FMT>(N, K, sms);
    const uint8_t* w = static_cast<const uint8_t*>(w_blocks);
    auto go = [&](auto r, auto v) {
        constexpr int R = decltype(r)::value, V = decltype(v)::value;
        if (p.input == RAW_PADDED) run_raw_matvec<FMT, R, V, RAW_PADDED>(p, dev, act, w, out, N, K, stream);
        else if (p.input == RAW_SWIZZLED) run_raw_matvec<FMT, R, V, RAW_SWIZZLED>(p, dev, act, w, out, N, K, stream);
        else run_raw_matvec<FMT, R, V, RAW_GLOBAL>(p, dev, act, w, out, N, K, stream);
    };
    using std::integral_constant;
    const bool v16 = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    if (p.pairs) v16 ? go(integral_constant<int, 2>{}, integral_constant<int, 16>{}) : go(integral_constant<int, 2>{}, integral_constant<int, 4>{});
    else v16 ? go(integral_constant<int, 1>{}, integral_constant<int, 16>{}) : go(integral_constant<int, 1>{}, integral_constant<int, 4>{});
}

}  // namespace

extern "C" {

void mongoose_q4_0_matvec(const float* act, const void* w_blocks, float* out, int N, int K, cudaStream_t stream) {
    launch_raw_matvec<FMT_Q4_0>(act, w_blocks, out, N, K, stream);
}

void mongoose_q8_0_matvec(const float* act, const void* w_blocks, float* out, int N, int K, cudaStream_t stream) {
    launch_raw_matvec<FMT_Q8_0>(act, w_blocks, out, N, K, stream);
}

void mongoose_q8_quantize_act(const float* act, void* q8_out, int K, cudaStream_t stream) {
    if (K < 32) return;
    quantize_act_kernel<<<cdiv(K / 32, 8), 256, 0, stream>>>(act, (ActBlock*)q8_out, K / 32);
}

void mongoose_q8_quantize_act_batch(const float* acts, void* q8_out, int K, int B, cudaStream_t stream) {
    if (K < 32 || B <= 0) return;
    const int total = (K / 32) * B;
    quantize_act_kernel<<<cdiv(total, 8), 256, 0, stream>>>(acts, (ActBlock*)q8_out, total);
}

void mongoose_q4_0_matvec_dp4a_preq(const void* w_blocks, const void* q8, float* out, int N, int K,
                                    cudaStream_t stream) {
    if (N <= 0 || K < 32) return;
    q4_0_dp4a_kernel<<<cdiv(N, 8), 256, 0, stream>>>((const uint8_t*)w_blocks, (const ActBlock*)q8, out, N, K, 1);
}

void mongoose_q4_0_matvec_dp4a_batch(const void* w_blocks, const void* q8, float* out, int N, int K, int B,
                                     cudaStream_t stream) {
    if (N <= 0 || K < 32 || B <= 0) return;
    q4_0_dp4a_kernel<<<cdiv(N, 8), 256, 0, stream>>>((const uint8_t*)w_blocks, (const ActBlock*)q8, out, N, K, B);
}

void mongoose_q4_0_matvec_dp4a(const float* act, const void* w_blocks, float* out, int N, int K, void* scratch,
                               cudaStream_t stream) {
    if (N <= 0 || K < 32 || !scratch) return;
    mongoose_q8_quantize_act(act, scratch, K, stream);
    mongoose_q4_0_matvec_dp4a_preq(w_blocks, scratch, out, N, K, stream);
}

// Q4_0 integer-dot matvec that allocates nothing.
//
// Who needs it: code that may not call cudaMalloc at the moment it wants a matvec - a capture-time
// or latency-critical section that forbids allocator calls, a plugin host that owns the memory
// budget and hands out no more, or a caller running after the pool it was given is exhausted.  The
// activation blocks (40 bytes per 32 inputs) that mongoose_q4_0_matvec_dp4a wants in a caller
// buffer live instead in a fixed array inside the library image (40 KiB, room for K <= 32768),
// present on every GPU that loads the library until the process exits.
//
// The array's name is only a host-side handle; the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current.  That lookup happens on the FIRST call on a
// device, so make the first call outside any stream capture.  The address is remembered per device
// for the life of the process: after cudaDeviceReset() the library must not be used on that device
// again (the remembered address belongs to the destroyed context).  Every call overwrites the whole
// region it uses before reading it, so nothing needs clearing between calls, but all calls share
// the one array: two calls that overlap on the GPU (different streams, different threads) race.
// Returns MG_OK, MG_ERR_ARG (NULL pointer, K not a multiple of 32, or K > 32768) or MG_ERR_CUDA;
// mongoose_static_scratch_error() has the text.
int mongoose_q4_0_matvec_dp4a_static(const float* act, const void* w_blocks, float* out, int N, int K,
                                     cudaStream_t stream) {
    g_static_err[0] = 0;
    if (!act || !w_blocks || !out) return static_fail(MG_ERR_ARG, "NULL pointer argument (N=%d K=%d)", N, K);
    if (N <= 0 || K < 32 || K % 32) return static_fail(MG_ERR_ARG, "N=%d must be positive and K=%d a multiple of 32", N, K);
    if (K > kStaticMaxK)
        return static_fail(MG_ERR_ARG, "K=%d exceeds the built-in scratch limit of %d input features", K, kStaticMaxK);
    int dev = -1;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return static_fail(MG_ERR_CUDA, "cudaGetDevice failed or device ordinal %d is out of range (%d)", dev, (int)ce);
    void* scratch;
    {
        std::lock_guard<std::mutex> lk(g_static_mu);
        if (!g_static_ptr[dev]) {
            void* p = nullptr;
            ce = cudaGetSymbolAddress(&p, g_static_act_scratch);
            if (ce != cudaSuccess || !p)
                return static_fail(MG_ERR_CUDA, "cudaGetSymbolAddress failed on device %d (error %d)", dev, (int)ce);
            g_static_ptr[dev] = p;
        }
        scratch = g_static_ptr[dev];
    }
    // Each launch's own status is checked: an error that an earlier, unrelated call left behind is
    // cleared first so that it is not taken for one of ours (a sticky error - a faulted context -
    // comes back from the next check all the same, and is reported as what it is).
    (void)cudaGetLastError();
    quantize_act_kernel<<<cdiv(K / 32, 8), 256, 0, stream>>>(act, (ActBlock*)scratch, K / 32);
    if ((ce = cudaGetLastError()) != cudaSuccess)
        return static_fail(MG_ERR_CUDA, "launch of the activation quantizer failed on device %d (CUDA error %d)", dev, (int)ce);
    q4_0_dp4a_kernel<<<cdiv(N, 8), 256, 0, stream>>>((const uint8_t*)w_blocks, (const ActBlock*)scratch, out, N, K, 1);
    if ((ce = cudaGetLastError()) != cudaSuccess)
        return static_fail(MG_ERR_CUDA, "launch of the matvec failed on device %d (CUDA error %d)", dev, (int)ce);
    return MG_OK;
}

const char* mongoose_static_scratch_error(void) { return g_static_err; }

// The reference's per-token op order (cuda_fused_infer.go:414-444 / cuda_fused_infer_q4.go:103-131)
// issued from one C call on caller-owned buffers.
void mongoose_partial_step_q4_fused_graph(
    const float** norm1, const void** wq, const void** wk, const void** wv, const void** wo,
    const float** norm2, const void** wgate, const void** wup, const void** wdown,
    float** kCache, float** vCache,
    float* hidden, float* normed, float* Q, float* K, float* V,
    float* attnOut, float* proj, float* normed2,
    float* gatePre, float* upOut, float* ffnMid,
    void* q8Scratch,
    const float* cosTab, const float* sinTab,
    int dim, int kvDim, int headDim, int ffnDim, int nHeads, int nKVHeads, int halfHead,
    int pos, int layerStart, int layerEnd,
    cudaStream_t stream) {
    (void)q8Scratch;   // fp32 activations throughout: no activation quantization on this path
    const float* cosRow = cosTab + (size_t)pos * halfHead;
    const float* sinRow = sinTab + (size_t)pos * halfHead;
    for (int l = layerStart; l < layerEnd; l++) {
        mongoose_rmsnorm_out(hidden, normed, norm1[l], 1, dim, stream);
        mongoose_q4_0_matvec(normed, wq[l], Q, dim, dim, stream);
        mongoose_q4_0_matvec(normed, wk[l], K, kvDim, dim, stream);
        mongoose_q4_0_matvec(normed, wv[l], V, kvDim, dim, stream);
        mongoose_rope(Q, cosRow, sinRow, 1, dim, headDim, nHeads, stream);
        mongoose_rope(K, cosRow, sinRow, 1, kvDim, headDim, nKVHeads, stream);
        mongoose_kv_cache_write(kCache[l], K, pos, kvDim, stream);
        mongoose_kv_cache_write(vCache[l], V, pos, kvDim, stream);
        mongoose_decode_attention(Q, kCache[l], vCache[l], attnOut, pos + 1, dim, kvDim, nHeads, nKVHeads, stream);
        mongoose_q4_0_matvec(attnOut, wo[l], proj, dim, dim, stream);
        mongoose_add_inplace(hidden, proj, dim, stream);
        mongoose_rmsnorm_out(hidden, normed2, norm2[l], 1, dim, stream);
        mongoose_q4_0_matvec(normed2, wgate[l], gatePre, ffnDim, dim, stream);
        mongoose_q4_0_matvec(normed2, wup[l], upOut, ffnDim, dim, stream);
        mongoose_silu_gate_mul(gatePre, upOut, ffnMid, ffnDim, stream);
        mongoose_q4_0_matvec(ffnMid, wdown[l], proj, dim, ffnDim, stream);
        mongoose_add_inplace(hidden, proj, dim, stream);
    }
}

}  // extern "C"
