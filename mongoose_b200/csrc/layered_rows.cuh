// Products of one token's vector with bf16 matrices.  The threads of a CTA (or a part of it, for narrow rows) share the
// columns of R rows at a time: a thread's vector values serve R rows, and the weights of a CTA's first rows, all of
// them where rows are few, are on the way before the kernel waits for its predecessor.  A row's sums over the warps
// meet in shared memory.  Vectors that need no norm are copied with cp.async, all of them in one trip to L2.
//
// What bounds a product is latency: waiting for the vector, norming it, one or two trips for weights (1 to 2 TB/s).
// A warp per row, or per four, read its vector from shared memory for every row and had fewer loads under way: 300 + 64
// tokens, six layers of 1.1B widths, B200: Mitotar 22.0 -> 19.1 ms, Kuzipel 25.0 -> 23.5 ms.  A ring of bulk copies that the
// eight warps of a CTA consumed slot by slot was slower than either (26.9 and 28.8 ms).
#pragma once

#include "layered_ops.cuh"

namespace mg {

constexpr int kRowThreads = 256;

// Threads that share a row of K columns, and rows a thread takes at a time: as many as leave every SM a CTA.
__host__ __device__ constexpr int row_group(int K) { return K <= 512 ? 64 : K <= 1024 ? 128 : 256; }
inline int rows_at_a_time(int K, long long rows, int sms) {
    int R = K <= 2048 ? 8 : 4;
    while (R > 1 && rows < (long long)R * (kRowThreads / row_group(K)) * sms) R /= 2;
    return R;
}

// AHEAD: chunks of 8 columns per thread and row that are fetched at once.
template <int EPI, int R, int AHEAD>
__device__ __forceinline__ void rows_body(const PhaseArgs& a, int bid, int nblocks, bool keep) {
    using C = Chunk<FMT_BF16>;
    extern __shared__ __align__(16) float smem[];
    __shared__ float part[2][kRowThreads / 32][R];
    float *xs = smem, *red = smem + a.K;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int group = row_group(a.K), groups = kRowThreads / group, t = threadIdx.x & (group - 1), mine = threadIdx.x / group * R;
    const int chunks = a.K / C::kWeights, rows = a.rows[0], per = R * groups;
    const uint4* W = reinterpret_cast<const uint4*>(a.w[0].qs);

    uint4 w[AHEAD][R];
    auto load = [&](int c0, int r0) {
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int c = c0 + i * group;
#pragma unroll
            for (int r = 0; r < R; r++) w[i][r] = c < chunks ? ld_stream16(W + (size_t)min(r0 + mine + r, rows - 1) * chunks + c) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    int r0 = bid * per;
    if (r0 < rows) load(t, r0);

    // the norms' weights on their way to this SM's L1, where they would cost a trip to L2 behind every sum
    const float* const vecs[] = {a.z_w[0], a.z_w[1], a.post_w, a.last_w, a.mix_mu};
#pragma unroll
    for (const float* v : vecs)
        if (v)
            for (int i = threadIdx.x * 32; i < a.k_valid; i += kRowThreads * 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(v + i));

    pdl_launch_dependents();
    pdl_wait();
    if (a.pro == PRO_X && !a.last_w && !a.cat && !(keep && a.h_store)) {
        const int n = a.k_valid;
        const bool vec = (reinterpret_cast<uintptr_t>(a.x_src) & 15) == 0;
        for (int i = threadIdx.x * 4; i < a.K; i += kRowThreads * 4) {
            if (vec && i + 4 <= n) {
                cp_async16(xs + i, a.x_src + i);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) xs[i + k] = i + k < n ? a.x_src[i + k] : 0.f;
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
    } else {
        stage_layered(a, xs, red, keep);
    }

    unsigned long long best = 0ull;
    for (int buf = 0; r0 < rows; buf ^= 1) {
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.f;
        for (int c0 = t;; ) {
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int c = c0 + i * group;
                if (c < chunks) {
                    const float4 x[2] = {*reinterpret_cast<const float4*>(xs + c * 8), *reinterpret_cast<const float4*>(xs + c * 8 + 4)};
#pragma unroll
                    for (int r = 0; r < R; r++) acc[r] += C::dot(w[i][r], x);
                }
            }
            c0 += AHEAD * group;
            if (c0 - t >= chunks) break;
            load(c0, r0);
        }
        const int next = r0 + nblocks * per;
        if (next < rows) load(t, next);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float v = warp_sum(acc[r]);
            if (lane == 0) part[buf][wid][r] = v;
        }
        __syncthreads();
        if ((int)threadIdx.x < per && r0 + (int)threadIdx.x < rows) {
            const int g = threadIdx.x / R, r = threadIdx.x - g * R, first = g * (group / 32);
            float v = 0.f;
            for (int q = 0; q < group / 32; q++) v += part[buf][first + q][r];
            const int row = r0 + threadIdx.x;
            if (EPI == EPI_LOGITS) {
                if (a.out) a.out[row] = v;
                const unsigned long long key = pack_best(v, (unsigned)(row + a.row_base));
                best = key > best ? key : best;
            } else {
                a.out[row] = EPI == EPI_GELU ? gelu_tanh(v) : v;
            }
        }
        r0 = next;
    }
    if (EPI == EPI_LOGITS) publish_best(a, best, reinterpret_cast<unsigned long long*>(red), nblocks);
}

template <int EPI, int R, int AHEAD>
__global__ void __launch_bounds__(kRowThreads, 2) rows_kernel(const PhaseArgs a) {
    rows_body<EPI, R, AHEAD>(a, blockIdx.x, gridDim.x, blockIdx.x == 0);
}

// Two independent matrices in one launch: the first `split` CTAs multiply a's, the others b's.
template <int R, int AHEAD>
__global__ void __launch_bounds__(kRowThreads, 2) rows_pair_kernel(const PhaseArgs a, const PhaseArgs b, int split) {
    const bool first = (int)blockIdx.x < split;
    rows_body<EPI_STORE, R, AHEAD>(first ? a : b, first ? blockIdx.x : blockIdx.x - split, first ? split : gridDim.x - split,
                                   first ? blockIdx.x == 0 : (int)blockIdx.x == split);
}

// Part p's CTAs multiply its matrix by the mix with its own mu.
template <int R, int AHEAD>
__global__ void __launch_bounds__(kRowThreads, 2) rows_parts_kernel(const PhaseArgs a, const PhaseParts parts) {
    int p = 0;
#pragma unroll
    for (int i = 1; i < kMaxParts; i++)
        if (i < parts.n && (int)blockIdx.x >= parts.first[i]) p = i;
    PhaseArgs b = a;
    b.w[0] = parts.w[p]; b.rows[0] = parts.rows[p]; b.mix_mu = parts.mu[p]; b.out = parts.out[p];
    rows_body<EPI_STORE, R, AHEAD>(b, blockIdx.x - parts.first[p], parts.first[p + 1] - parts.first[p], blockIdx.x == 0);
}

}  // namespace mg
