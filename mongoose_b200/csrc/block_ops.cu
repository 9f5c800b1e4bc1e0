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
#include "umma.cuh"

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

// ---------------- the same on the integer tensor path: matrices that keep every SM busy ----------------
// Above, a lane converts every weight to fp32: about eight instructions per weight of a lane, and the issue slots are what
// bounds a large product.  Here a warp multiplies 16 rows x one block of 32 columns by ONE mma.sync (m16n8k32, int8): A = the
// quants as they lie in the block (4-bit ones as 16 (q - 8)), B = the activations as fixed point, two whole numbers of three signed byte
// digits each in six of the eight columns.  A block's activations share a power of two, which puts the largest at 2^20 .. 2^21: the first number is what is
// whole of that, the second what is left, in steps of 2^-22.  So the digits hold EVERY bit of an element that has 2^-19 of its block's largest or more.
// A block with an element of which they do not is PLAIN (scale 0): multiplied in fp32 as the kernel above does; so is one that is not finite, lies
// below 2^-82, where the product of its scales would not hold fp32's bits, or spans more than fp32's exponents.  A block's sums are integers of up
// to 27 bits, which fp32 rounds once and adds (block scale x power of two x sum) over the blocks, one or two digits at a time.
//   A CTA owns a contiguous run of rows, taken up to 32 at a time (one or two MMA tiles, which share the activations), and a row's
// blocks in SEGMENTS of up to 128 (Q8_0: 64), 2 KB of every row.  A producer warp copies a segment (cp.async.bulk, a lane a row: the
// 16-byte pieces that cover it) into a ring of slots; the 16 other warps share its blocks, and their sums over all
// segments meet in shared memory.  Rows lie an odd multiple of 16 bytes apart in a slot, so that the eight rows of an access
// fall on different banks.  (Copies by the warps themselves, ten pieces of 16 bytes per row and turn with cp.async, took half the time.)
//   What bounds it is instruction issue (66 % of the slots of a launch by itself, Q4_0 3584 x 18944, 53 % of the ALU's; shared memory 26 %), and in front
// of the first rows the staging of the whole input by every CTA.  Blocks are taken in PAIRS, 9 (17) aligned
// words of a row: the scale of the first and two of its quants share word 0, its last two and the scale of the second word 4 (8).
// Lane t = 0 of a row completes its half word from there, so that no lane re-aligns what it loads: 2 (3) loads per
// block and row where re-aligned words took 3 (5).  The activations of even blocks are staged in that order of elements.
// B200, the kernel above -> this one, weights in no cache (the same matrix again and again): Q4_0 3584 x 18944 26.1 -> 15.0 us (25.8 -> 14.0), 3584 x 3584 11.0 -> 5.4,
// 18944 x 3584 23.9 -> 12.9; Q8_0 3584 x 18944 27.2 -> 18.5, 18944 x 3584 26.1 -> 15.3, 9000 x 18944 51.2 -> 40.8.  Four digits, which keep 30 bits below the largest, took
// 13.1, 4.8, 11.3, 17.6, 14.9 and 34.7, and lost what lies below: one large activation under a small weight took its block's other terms with it.  Where
// every block is plain (activations e^(8 N(0, 1))): Q4_0 3584 x 18944 34 us, Q8_0 38, slower than above; of 18944 columns N(0, 1) inputs have a plain
// block in one of 27 products, gated ones (silu(u) v) in every second, which takes no longer.  Error against 64 bits at 3584 x 18944 Q4_0 1.4e-7 -> 0.7e-7.
//   A row whose sum over digits is not finite (a scale that is not, sums beyond the range) is computed again in plain fp32.
constexpr int kMmaWarps = 16, kMmaRows = 32, kMmaSlots = 4;
constexpr int kMmaThreads = (kMmaWarps + 1) * 32;
__host__ __device__ constexpr int mma_seg(int fmt) { return fmt == FMT_Q8_0 ? 32 : 64; }       // pairs
// From row to row of a slot: whole pieces that cover a row's part of a segment of `per` pairs, an odd number of them.
__host__ __device__ constexpr int mma_stride(int fmt, int per) { return ((per * 2 * block_bytes(fmt) + 30) / 16 | 1) * 16; }
constexpr int kMmaDigits = 6;
__host__ __device__ constexpr int mma_digit_bytes(int nb) { return (nb * 32 + 127) / 128 * 128 + 32; }     // from digit to digit: four in turn on different banks
__host__ __device__ constexpr size_t mma_input_bytes(int nb) { return (size_t)kMmaDigits * mma_digit_bytes(nb) + ((size_t)nb * 4 + 15) / 16 * 16; }
constexpr size_t kMmaSums = (size_t)2 * kMmaWarps * kMmaRows * 4, kMmaBars = 2 * kMmaSlots * 8 + 16, kMmaFixed = kMmaSums + kMmaBars;

// Re-computes one row; every lane returns it.
template <int FMT>
__device__ __noinline__ float raw_row_plain(const float* __restrict__ act, const uint8_t* __restrict__ row, int nb) {
    constexpr int BB = block_bytes(FMT);
    float acc = 0.f;
    for (int b = threadIdx.x & 31; b < nb; b += 32) {
        const uint8_t* p = row + (size_t)b * BB;
        const float* x = act + (size_t)b * 32;
        const float d = half_bits_to_float(*reinterpret_cast<const unsigned short*>(p));
        float sum = 0.f;
        for (int i = 0; i < 32; i++) {
            const int q = FMT == FMT_Q8_0 ? (int)(int8_t)p[2 + i] : (i < 16 ? p[2 + i] & 15 : p[2 + i - 16] >> 4) - 8;
            sum = fmaf((float)q, x[i], sum);
        }
        acc = fmaf(d, sum, acc);
    }
    return warp_sum(acc);
}

// A row's block at `p` in shared memory, an even address, times its activations, of which lane i holds the i-th; in fp32.  Lanes are rows.
template <int FMT>
__device__ __noinline__ float mma_plain_block(uint32_t p, float x, float acc) {
    constexpr int QW = FMT == FMT_Q8_0 ? 8 : 4;
    auto word = [&](int i) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"((p & ~3u) + 4 * i));
        return v;
    };
    auto xi = [&](int i) { return __shfl_sync(MG_FULL_MASK, x, i); };
    auto x4 = [&](int i) { return make_float4(xi(4 * i), xi(4 * i + 1), xi(4 * i + 2), xi(4 * i + 3)); };
    const int sh = p & 2 ? 32 : 16;                         // quants start 2 bytes after the scale
    uint32_t lo = word(0);
    const float d = half_bits_to_float((unsigned short)(p & 2 ? lo >> 16 : lo & 0xffffu));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < QW; i++) {
        const uint32_t hi = word(i + 1), q = __funnelshift_rc(lo, hi, sh);
        if (FMT == FMT_Q8_0) sum = dot4_s8(q, x4(i), sum);
        else sum = dot4_u4(q >> 4 & 0x0f0f0f0fu, x4(4 + i), dot4_u4(q & 0x0f0f0f0fu, x4(i), sum));
        lo = hi;
    }
    return fmaf(d, sum, acc);
}

// `n` pairs of blocks for NT tiles of 16 rows.  at: this lane's rows g + 8 r, offset of the first pair in shared memory; digits,
// scales: of its first block.  A lane t gets columns 2 t and 2 t + 1 of a product, two digits that follow one another, high and low.  acc: even and odd
// blocks, so that fewer roundings follow one another.
template <int FMT, int NT>
__device__ __forceinline__ void mma_pairs(const uint8_t* smem, const uint32_t (&at)[2 * NT], int n, uint32_t digits, uint32_t scales, bool bvalid, int t,
                                          float (&acc)[2][4]) {
    constexpr int PB = 2 * block_bytes(FMT), QW = block_bytes(FMT) / 4 * 4;        // bytes of a pair; where the word that both blocks share lies
    const unsigned join = t == 0 ? 0x3254u : 0x3210u;
    auto word = [&](uint32_t p) { return *reinterpret_cast<const uint32_t*>(smem + p); };
#pragma unroll 2
    for (int k = 0; k < n; k++) {
        uint2 B[2];
        float s[2], d[2][2 * NT];
        uint32_t a[2][NT][4];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            B[j] = bvalid ? *reinterpret_cast<const uint2*>(smem + digits + (2 * k + j) * 32) : make_uint2(0u, 0u);
            s[j] = *reinterpret_cast<const float*>(smem + scales + (2 * k + j) * 4);
        }
#pragma unroll
        for (int r = 0; r < 2 * NT; r++) {
            const uint32_t p = at[r] + k * PB;
            const uint32_t both = word(p + QW);
            uint32_t(&e)[4] = a[0][r >> 1], (&o)[4] = a[1][r >> 1];
            d[0][r] = half_bits_to_float(*reinterpret_cast<const unsigned short*>(smem + p));
            d[1][r] = half_bits_to_float((unsigned short)(both >> 16));
            const uint32_t v0 = __byte_perm(word(p + 4 * t), both, join), v1 = word(p + QW + 4 + 4 * t);
            if (FMT == FMT_Q8_0) {
                e[r & 1] = v0; e[2 + (r & 1)] = word(p + 16 + 4 * t);
                o[r & 1] = v1; o[2 + (r & 1)] = word(p + QW + 20 + 4 * t);
            } else {
                e[r & 1] = ((v0 << 4) & 0xf0f0f0f0u) ^ 0x80808080u; e[2 + (r & 1)] = (v0 & 0xf0f0f0f0u) ^ 0x80808080u;
                o[r & 1] = ((v1 << 4) & 0xf0f0f0f0u) ^ 0x80808080u; o[2 + (r & 1)] = (v1 & 0xf0f0f0f0u) ^ 0x80808080u;
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < NT; i++) {
                const uint32_t(&o)[4] = a[j][i];
                int c[4];
                asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                    : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                    : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(B[j].x), "r"(B[j].y), "r"(0));
                acc[j][2 * i] = fmaf(d[j][2 * i] * s[j], __int2float_rn(c[0] * 256 + c[1]), acc[j][2 * i]);        // |c| <= 32 * 128 * 128
                acc[j][2 * i + 1] = fmaf(d[j][2 * i + 1] * s[j], __int2float_rn(c[2] * 256 + c[3]), acc[j][2 * i + 1]);
            }
    }
}

// An even number of blocks, and a matrix on a 16-byte boundary.  slot_rows: rows taken at a time; slots: of the ring.
template <int FMT>
__global__ void __launch_bounds__(kMmaThreads, 1) raw_block_matvec_mma_kernel(const float* __restrict__ act, const uint8_t* __restrict__ w, float* out, int N, int K,
                                                                       int slot_rows, int slots, int per) {
    constexpr int BB = block_bytes(FMT), SEG = mma_seg(FMT);
    extern __shared__ __align__(16) uint8_t mma_smem[];     // digits [digit][block][32], scales; sums [2][warp][row]; barriers; slots
    const int nb = K / 32, np = nb / 2, segs = (np + per - 1) / per, stride = mma_stride(FMT, per), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int digit_bytes = mma_digit_bytes(nb);
    const size_t rb = (size_t)nb * BB;
    float* part = reinterpret_cast<float*>(mma_smem + mma_input_bytes(nb));
    uint64_t* full = reinterpret_cast<uint64_t*>(mma_smem + mma_input_bytes(nb) + kMmaSums);
    uint64_t* empty = full + kMmaSlots;
    int* status = reinterpret_cast<int*>(empty + kMmaSlots), *inputs_off = status + 1;    // inputs_off: an activation is not finite
    unsigned* again = reinterpret_cast<unsigned*>(status + 2);     // [2] rows whose sum over digits is not finite
    const uint32_t ring = (uint32_t)(mma_input_bytes(nb) + kMmaFixed), slot_bytes = (uint32_t)slot_rows * stride;
    const int row_lo = (int)((long long)N * blockIdx.x / gridDim.x), row_hi = (int)((long long)N * (blockIdx.x + 1) / gridDim.x);
    if (threadIdx.x == 0) {
        for (int i = 0; i < slots; i++) { bar_init(full + i, 1); bar_init(empty + i, kMmaWarps); }
        *status = *inputs_off = 0;
        again[0] = again[1] = 0;
        bar_init_fence();
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();

    if (warp == kMmaWarps) {
        int s = 0, par = 1, n = 0;
        bool ok = true;
        for (int row0 = row_lo; ok && row0 < row_hi; row0 += slot_rows)
            for (int k = 0; k < segs; k++, n++) {
                if (n >= slots && !(ok = __all_sync(MG_FULL_MASK, bar_wait(empty + s, par, status)))) break;
                const int p0 = k * per, p1 = min(p0 + per, np);
                const uint8_t* src = w;
                uint8_t* to = mma_smem + ring + s * slot_bytes + lane * stride;
                unsigned bytes = 0;
                if (lane < min(slot_rows, row_hi - row0)) {
                    src += (size_t)(row0 + lane) * rb + (size_t)p0 * 2 * BB;
                    const unsigned lead = (unsigned)(reinterpret_cast<uintptr_t>(src) & 15u), need = lead + (unsigned)(p1 - p0) * 2 * BB;
                    src -= lead;
                    const size_t left = (size_t)(w + (size_t)N * rb - src);         // nothing behind the matrix is read
                    bytes = (unsigned)min((size_t)((need + 15u) & ~15u), left & ~(size_t)15);
                    for (unsigned i = bytes; i < need; i += 2) *reinterpret_cast<unsigned short*>(to + i) = *reinterpret_cast<const unsigned short*>(src + i);
                }
                const unsigned all = __reduce_add_sync(MG_FULL_MASK, bytes);
                __syncwarp();                               // the bytes that a lane stored itself are there before lane 0 arrives
                if (lane == 0) bar_expect(full + s, all);
                __syncwarp();
                if (bytes)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(to)), "l"(src), "r"(bytes),
                                 "r"(smem_addr(full + s)) : "memory");
                if (++s == slots) { s = 0; par ^= 1; }
            }
        // no copy may be in flight when the CTA leaves
        for (int i = max(0, n - slots); i < n; i++) bar_wait(full + i % slots, (i / slots) & 1, status);
        return;
    }

    // Activations.  A warp stages the blocks that it multiplies, with the rows it takes first, eight blocks at a time (Q8_0: of two segments): four
    // lanes share a block, lane q the elements that the MMA wants in words q and q + 4, in even blocks 4 q - 2 .. 4 q + 1 and so on (the first two
    // from the end of the block, or of its half, where q is 0).  The next ones are on the way meanwhile.
    constexpr int PART = FMT == FMT_Q8_0 ? 32 : 16, OWN = 2 * SEG / kMmaWarps, AHEAD = 8 / OWN;     // OWN: blocks of a segment; AHEAD: segments
    static_assert(OWN * AHEAD == 8 && AHEAD <= 2, "eight blocks");
    const int q = lane & 3, sub = lane / (4 * OWN);
    const bool odd = lane & 4, x8 = (reinterpret_cast<uintptr_t>(act) & 7) == 0;
    const int col[4] = {odd ? 4 * q : q ? 4 * q - 2 : PART - 2, odd ? 4 * q + 2 : 4 * q, odd ? 4 * q + 16 : q || PART == 32 ? 4 * q + 14 : 30, odd ? 4 * q + 18 : 4 * q + 16};
    float2 xs[4];                                           // elements col[i], col[i] + 1 of block xb (-1: none)
    int xb;
    auto share = [&](int k, int& lo) {                      // this warp's pairs of segment k: their number, the first
        const int p0 = k * per, here = min(per, np - p0);
        lo = here * warp / kMmaWarps;
        return here * (warp + 1) / kMmaWarps - lo;
    };
    auto load_x = [&](int k) {
        int lo;
        k += sub;
        const int blk = lane / 4 % OWN, n = k < segs ? share(k, lo) : 0;
        xb = blk < 2 * n ? (k * per + lo) * 2 + blk : -1;
        const float* x = act + (size_t)max(xb, 0) * 32;
#pragma unroll
        for (int i = 0; i < 4; i++)
            xs[i] = xb < 0 ? make_float2(0.f, 0.f) : x8 ? *reinterpret_cast<const float2*>(x + col[i]) : make_float2(x[col[i]], x[col[i] + 1]);
    };
    bool plains = false;                                    // does one of this warp's blocks go without digits?
    auto store_x = [&] {
        auto bits = [](float v) { return __float_as_uint(fabsf(v)); };
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) m = max(m, max(bits(xs[i].x), bits(xs[i].y)));
#pragma unroll
        for (int o = 1; o < 4; o *= 2) m = max(m, __shfl_xor_sync(MG_FULL_MASK, m, o));
        bool plain = m - 1u < (45u << 23) - 1u || m >= 255u << 23;
        const bool far = m >= 148u << 23;
        m = max(m >> 23, 45u);                              // exponent of the largest
        const float up = __uint_as_float((274u - m) << 23);
        // whole numbers by additions that leave no place behind the point; the constant's low bytes make those of signed digits, xor 128
        constexpr float kWhole = 12582912.0f + 32896.0f;
        const unsigned long long up2 = pack2(up, up), whole = pack2(kWhole, kWhole), minus = pack2(-1.0f, -1.0f), more = pack2(4194304.0f, 4194304.0f);
        uint32_t u[2][8], any = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned long long x = pack2(xs[i].x, xs[i].y), a = fma2(x, up2, whole), left = fma2(x, up2, fma2(a, minus, whole));      // exact, as what follows
            const unsigned long long b = fma2(left, more, whole), rest = fma2(left, more, fma2(b, minus, whole));
            u[0][2 * i] = (uint32_t)b; u[0][2 * i + 1] = (uint32_t)(b >> 32);
            u[1][2 * i] = (uint32_t)a; u[1][2 * i + 1] = (uint32_t)(a >> 32);
            any |= (uint32_t)rest | (uint32_t)(rest >> 32);
        }
        if (xb >= 0) {
            uint8_t* to = mma_smem + xb * 32 + 8 * q;
#pragma unroll
            for (int h = 0; h < 2; h++, to += 3 * digit_bytes) {
                uint32_t lo[2], mid[2], hi[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint32_t* a = u[h] + 4 * i;
                    const uint32_t u0 = __byte_perm(a[0], a[1], 0x5140), u1 = __byte_perm(a[2], a[3], 0x5140);     // bytes 0 and 1 of two
                    lo[i] = __byte_perm(u0, u1, 0x5410) ^ 0x80808080u;
                    mid[i] = __byte_perm(u0, u1, 0x7632) ^ 0x80808080u;
                    hi[i] = __byte_perm(__byte_perm(a[0], a[1], 0x0062), __byte_perm(a[2], a[3], 0x0062), 0x5410);     // each 64 more than the digit
                    hi[i] = ((hi[i] | 0x80808080u) - 0x40404040u) ^ 0x80808080u;
                }
                *reinterpret_cast<uint2*>(to) = make_uint2(mid[0], mid[1]);
                *reinterpret_cast<uint2*>(to + digit_bytes) = make_uint2(lo[0], lo[1]);
                *reinterpret_cast<uint2*>(to + 2 * digit_bytes) = make_uint2(hi[0], hi[1]);
            }
        }
        any &= 0x7fffffffu;
        if (__any_sync(MG_FULL_MASK, any || far || plain)) {
            // rests, and blocks beyond 2^21, where a product with `up` may leave fp32's exponents
            bool off = any != 0;
#pragma unroll
            for (int i = 0; i < 4; i++) off |= far && ((xs[i].x != 0.f && fabsf(xs[i].x * up) < 0x1p-126f) || (xs[i].y != 0.f && fabsf(xs[i].y * up) < 0x1p-126f));
            plain |= (__ballot_sync(MG_FULL_MASK, off) & 15u << (lane & 28)) != 0;          // the block's lanes
            plains |= __any_sync(MG_FULL_MASK, plain);
            if (m == 255) *inputs_off = 1;
        }
        if (xb >= 0 && q == 0) reinterpret_cast<float*>(mma_smem + kMmaDigits * digit_bytes)[xb] = plain ? 0.f : __uint_as_float((m - 20u) << 23);
        __syncwarp();
    };
    load_x(0);

    auto all_consumers = [] { asm volatile("bar.sync 1, %0;" ::"n"(kMmaWarps * 32) : "memory"); };
    const int g = lane >> 2, t = lane & 3;
    const int digit = g - (g > 2) - (g > 6);                // columns 2 and 6 are empty: a number's first digit has no lower one beside it
    const bool bvalid = (g & 3) != 2;
    const float weight = (t == 0 ? 0x1p-22f : t == 1 ? 0x1p-6f : t == 2 ? 1.0f : 65536.0f) * (FMT == FMT_Q8_0 ? 1.0f : 0.0625f);
    int s = 0, par = 0, buf = 0;
    for (int row0 = row_lo; row0 < row_hi; row0 += slot_rows, buf ^= 1) {
        const int rows = min(slot_rows, row_hi - row0);
        float acc[2][4] = {}, plain = 0.f;                  // plain: what row `lane` has in fp32
        for (int k = 0; k < segs; k++) {
            int lo;
            const int n = share(k, lo), p0 = k * per;
            const uint32_t first = (uint32_t)reinterpret_cast<uintptr_t>(w) + (uint32_t)((size_t)row0 * rb + (size_t)p0 * 2 * BB);  // its low bits
            const uint32_t from = ring + s * slot_bytes + lo * 2 * BB, digits = (p0 + lo) * 64 + digit * digit_bytes + t * 8,
                           sc = kMmaDigits * digit_bytes + (p0 + lo) * 8;
            // (rows that a tile has and the slot has not: its last one again, dropped)
            auto row_at = [&](int row) {
                const uint32_t r = min(row, slot_rows - 1);
                return from + r * stride + ((first + r * (uint32_t)rb) & 15u);
            };
            if (row0 == row_lo && k % AHEAD == 0) {
                store_x();
                if (k + AHEAD < segs) load_x(k + AHEAD);
            }
            unsigned off = 0;                               // blocks without digits, and their activations, a lane an element
            float x_off[OWN];
            if (plains) {
                off = __ballot_sync(MG_FULL_MASK, lane < 2 * n && *reinterpret_cast<const float*>(mma_smem + sc + 4 * lane) == 0.f);
#pragma unroll
                for (int b = 0; b < OWN; b++) x_off[b] = off >> b & 1 ? act[(size_t)((p0 + lo) * 2 + b) * 32 + lane] : 0.f;
            }
            bar_wait(full + s, par, status);
            if (rows > 16) {
                const uint32_t at[4] = {row_at(g), row_at(g + 8), row_at(g + 16), row_at(g + 24)};
                mma_pairs<FMT, 2>(mma_smem, at, n, digits, sc, bvalid, t, acc);
            } else {
                const uint32_t at[2] = {row_at(g), row_at(g + 8)};
                mma_pairs<FMT, 1>(mma_smem, at, n, digits, sc, bvalid, t, acc);
            }
            if (off) {
#pragma unroll
                for (int b = 0; b < OWN; b++)
                    if (off >> b & 1) plain = mma_plain_block<FMT>(smem_addr(mma_smem) + row_at(lane) + b * BB, x_off[b], plain);
            }
            __syncwarp();
            if (lane == 0) bar_arrive(empty + s);
            if (++s == slots) { s = 0; par ^= 1; }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float v = (acc[0][i] + acc[1][i]) * weight;
            v += __shfl_xor_sync(MG_FULL_MASK, v, 1);
            v += __shfl_xor_sync(MG_FULL_MASK, v, 2);
            if (t == 0) {
                part[(buf * kMmaWarps + warp) * kMmaRows + g + 8 * i] = v;
                if (!(fabsf(v) <= 3.402823466e38f)) atomicOr(again + buf, 1u << (g + 8 * i));
            }
        }
        if (plains) {
            __syncwarp();
            part[(buf * kMmaWarps + warp) * kMmaRows + lane] += plain;
        }
        all_consumers();                                    // (two buffers: a sum is read while the next rows are multiplied)
        if (warp == 0) {
            float u[kMmaWarps];
#pragma unroll
            for (int p = 0; p < kMmaWarps; p++) u[p] = part[(buf * kMmaWarps + p) * kMmaRows + lane];
#pragma unroll
            for (int h = kMmaWarps / 2; h > 0; h /= 2)
#pragma unroll
                for (int p = 0; p < h; p++) u[p] += u[p + h];
            float v = u[0];
            const bool off = lane < rows && ((again[buf] >> lane & 1) || (!(fabsf(v) <= 3.402823466e38f) && !*inputs_off));
            __syncwarp();
            if (lane == 0) again[buf] = 0;
            for (unsigned left = __ballot_sync(MG_FULL_MASK, off); left; left &= left - 1) {
                const int r = __ffs(left) - 1;
                const float sum = raw_row_plain<FMT>(act, w + (size_t)(row0 + r) * rb, nb);
                if (lane == r) v = sum;
            }
            if (*reinterpret_cast<volatile int*>(status)) v = __uint_as_float(0x7fc00000u);     // a copy never came
            if (lane < rows) out[row0 + lane] = v;
        }
    }
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
// 40960 817 / 112 us, 256 x 32768 99 / 7 us.  Elsewhere: 4864 x 896 Q8_0 4.4 us, 3584 x 36864 51.5, 600 x 18944 10.8 (what the integer kernel takes: there).
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

// A launch that may begin while the one before it ends (the kernels wait before they read).  raised: is the kernel's limit
// of shared memory up on a device?
template <typename... P, typename... A>
void launch_raw(void (*kern)(P...), std::atomic<bool>* raised, int dev, int grid, int threads, size_t smem, cudaStream_t stream, A... args) {
    if (smem > 48 * 1024 && !(dev < kMaxDevices && raised[dev].load(std::memory_order_relaxed))) {
        cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (dev < kMaxDevices) raised[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int FMT, int R, int V, int X>
void run_raw_matvec(const RawShape& p, int dev, const float* act, const uint8_t* w, float* out, int N, int K, cudaStream_t stream) {
    static std::atomic<bool> raised[kMaxDevices];
    launch_raw(raw_block_matvec_kernel<FMT, R, V, X>, raised, dev, p.grid, p.threads, p.smem, stream, act, w, out, N, K, p.ks);
}

// Rows a CTA of the integer kernel takes at a time, slots of its ring, and pairs of a segment; no rows: shared memory holds no two slots.  Two tiles of
// rows at a time (as even as may be) where that takes no more than a third more segments than there may be fewest, else one.  B200, us of Q8_0 / Q4_0, two
// tiles in so many segments, one tile: 9000 x 18944 40.8 in 12, 40.9 in 10 / 30.9 in 7, 29.0 in 5; 3584 x 24576 28.3 in 18, 28.7 in 12 / 21.8 in 10, 21.4 in 6;
// 2400 x 26624 24.4 in 17, 25.5 in 13 / 20.4 in 9, 21.8 in 7.
struct MmaShape {
    int rows, slots, per;
    size_t smem;
};
template <int FMT>
MmaShape mma_shape(int N, int K, int sms) {
    const int pairs = K / 64, most = cdiv(N, sms), least = cdiv(pairs, mma_seg(FMT));
    const size_t fixed = mma_input_bytes(K / 32) + kMmaFixed;
    for (int tiles = 2; tiles > 0; tiles--) {
        const int rows = cdiv(most, cdiv(most, 16 * tiles));
        for (int segs = least; 3 * segs <= 4 * least; segs++) {
            const int per = cdiv(pairs, segs);
            const size_t slot = (size_t)rows * mma_stride(FMT, per);
            for (int slots = kMmaSlots; slots >= 2; slots--)
                if (fixed + slots * slot <= kRawSmem) return {rows, slots, per, fixed + slots * slot};
        }
    }
    return {};
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
    const uint8_t* w = static_cast<const uint8_t*>(w_blocks);
    // The integer kernel, us of Q8_0 / Q4_0 on weights in no cache, the other -> this: 1088 columns 600 rows 3.43 -> 3.20 / 3.16 -> 3.22, 18944 rows 13.4 -> 9.2 / 12.6 ->
    // 9.4; 4864 columns 800 rows 4.4 -> 5.2 / 5.2 -> 4.9, 1200 rows 6.1 -> 5.4 / 8.0 -> 5.1; 8192
    // columns 600 rows 6.3 -> 6.0 / 7.8 -> 5.4; 18944 columns 800 rows 11.0 -> 11.6 / 14.7 -> 10.6, 1200 rows 17.6 -> 11.8 / 23.3 -> 10.6; 24576 columns 1200 rows 21.3
    // -> 14.3 / 20.0 -> 12.5.  Every CTA stages the whole input, so few rows do not pay for it.  Q8_0 of four to eight rows per SM: 3072 columns 4.4 to 5.1 -> 4.0 to 4.2,
    // 5120 columns 600 rows 4.3 -> 5.0, 1000 rows 6.1 -> 5.3, 6144 columns (the other kernel has one CTA per SM from 5472 on) 6.2 to 6.6 -> 5.3 to 5.6, 12288 columns
    // 8.5 to 11.1 -> 8.0 to 8.4 (at 1180 rows 7.9), 14336 columns 8.6 to 8.9 -> 9.4 to 9.7.
    const int r = N / sms;
    const bool enough = r >= 8 || (r >= 4 && (FMT == FMT_Q4_0 ? K <= 20480 : K <= 3072 || (K <= 12288 && (r >= 6 || K > 5440))));
    const bool ints = K > 1024 && K % 64 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && enough;
    const MmaShape q = ints ? mma_shape<FMT>(N, K, sms) : MmaShape{};
    if (q.rows > 0) {
        static std::atomic<bool> raised[kMaxDevices];
        launch_raw(raw_block_matvec_mma_kernel<FMT>, raised, dev, std::min(sms, N), kMmaThreads, q.smem, stream, act, w, out, N, K, q.rows, q.slots, q.per);
        return;
    }
    const RawShape p = raw_shape<FMT>(N, K, sms);
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
