// One token of a layer-described model: products, and the mixer step, in
// which the attention branch (split over keys) and the matrix-memory branch run side by side.
#include <algorithm>
#include <type_traits>

#include "layered_ops.cuh"
#include "layered_rows.cuh"

namespace mg {

namespace {

constexpr int kStepThreads = 512;
constexpr int kStateRows = 16;      // rows of the state a warp holds at a time

// One token of the matrix memory: CTA (head, slice of 32 value columns); lanes over columns, warps over
// the rows of the state.  Every slice forms the head's normaliser; slice 0 stores it into the other
// parity slot, so no slice reads what another writes.
__device__ __forceinline__ void mem_step(const MixerStep& a, int cta, float* smem) {
    const MatMem& M = a.mem;
    const int head = cta / a.vslices, slice = cta % a.vslices;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float* red = smem;                      // 40
    float* part = smem + 40;                // nw * 32
    float* ks = part + nw * 32;             // dim
    float* qs = ks + M.dim;                 // dim
    const int pos = a.st->pos;
    const bool fresh = pos == 0;
    const float* row = a.proj;
    const int v = slice * 32 + lane;
    float* S = M.S + (size_t)head * M.dim * M.vdim + v;
    // the state was left by the last token: it is on its way before the predecessor has finished
    float s0[kStateRows];
    auto load_rows = [&](int d0) {
#pragma unroll
        for (int i = 0; i < kStateRows; i++) {
            const int d = d0 + wid + i * nw;
            s0[i] = !fresh && v < M.vdim && d < M.dim ? S[(size_t)d * M.vdim] : 0.f;
        }
    };
    load_rows(0);
    const int cur = pos & 1;
    const float m0 = fresh ? 0.f : M.m[cur * M.heads + head];
    const int d_own = threadIdx.x;
    const float n_own = fresh || d_own >= M.dim ? 0.f : M.nrm[((size_t)cur * M.heads + head) * M.dim + d_own];
    pdl_wait();
    const float vv = v < M.vdim ? row[a.c.mv + head * M.vdim + v] : 0.f;
    const float ig = soft_cap(row[a.c.mi + head] + M.i_bias[head], M.cap);
    const float fg = log_sigmoid(soft_cap(row[a.c.mf + head] + M.f_bias[head], M.cap));
    const float m1 = fmaxf(fg + m0, ig);
    const float keep = expf(fg + m0 - m1), add = expf(ig - m1);
    const float qscale = 1.0f / sqrtf((float)M.dim);
    float nq = 0.f;
    for (int d = threadIdx.x; d < M.dim; d += blockDim.x) {
        const float k = row[a.c.mk + head * M.dim + d], q = row[a.c.mq + head * M.dim + d] * qscale;
        ks[d] = k * add;
        qs[d] = q;
        const float n0 = d == d_own ? n_own : fresh ? 0.f : M.nrm[((size_t)cur * M.heads + head) * M.dim + d];
        const float n1 = keep * n0 + add * k;
        if (slice == 0) M.nrm[((size_t)(cur ^ 1) * M.heads + head) * M.dim + d] = n1;
        nq = fmaf(n1, q, nq);
    }
    nq = block_sum(nq, red);                // its barriers publish ks and qs
    if (slice == 0 && threadIdx.x == 0) M.m[(cur ^ 1) * M.heads + head] = m1;
    float acc = 0.f;
    for (int d0 = 0; d0 < M.dim; d0 += kStateRows * nw) {
        if (d0 > 0) load_rows(d0);
#pragma unroll
        for (int i = 0; i < kStateRows; i++) {
            const int d = d0 + wid + i * nw;
            if (v < M.vdim && d < M.dim) {
                const float s1 = fmaf(ks[d], vv, keep * s0[i]);
                S[(size_t)d * M.vdim] = s1;
                acc = fmaf(s1, qs[d], acc);
            }
        }
    }
    part[wid * 32 + lane] = acc;
    __syncthreads();
    if (wid == 0 && v < M.vdim) {
        float o = 0.f;
        for (int w = 0; w < nw; w++) o += part[w * 32 + lane];
        a.mem_o[head * M.vdim + v] = o / (fmaxf(fabsf(nq), expf(-m1)) + 1e-6f);
    }
}

// Shared memory of the attention part: AttnSmem, and behind it
//   rnew [kv_heads], knew [kv_heads][dim_s] the new key as it is stored (read back
//   from the cache where shared memory has no room for it).
inline size_t step_extra(const GateAttn& A) { return ((size_t)pad_to(A.kv_heads, 4) + 3) * 4; }
inline size_t step_key(const GateAttn& A, size_t kt_bytes) { return (size_t)A.kv_heads * A.dim_s * kt_bytes; }

// What bounds the step is the latency of one tile of keys: loads that follow one another, each phase behind a barrier, on the CTAs of
// a few keys each.  So four lanes share a score and a mixed weight, sixteen a query's norm, keys are dealt four by four, and
// everything that no predecessor leaves (cached keys, tables, the norms' weights, addresses) is there before the wait; the new key
// reaches the CTA that ends with it through shared memory, not through the cache.  B200, 1.1B widths, 320 positions, us from the
// wait to the end of this kernel: 9.2 with 256 threads, a thread per score, eight lanes per norm and tiles of eight keys, 4.3 now;
// 300 + 64 tokens of six layers 18.20 -> 16.92 ms.  Runs of 4 / 8 keys per CTA, us per token of the kernel as it is: four layers of 1.1B widths at 20
// positions 162.4 / 161.6, 300 169.6 / 165.6 (a lane per score), 1200 171.9 / 171.4, 4000 192.8 / 194.1; 0.5B 143.0 / 141.8, 143.3 / 147.4, 147.9 / 145.8, 160.9 / 161.0;
// two of 7B widths at 300 220.9 / 220.6, 4000 245.9 / 246.7.
//   Many keys per CTA (the memory leaves 84 CTAs at 1.1B widths) are bound by instructions instead: a tile holds the range, up to 16 keys, and from
// 192 scores on a lane has one for itself.  us per token, tiles of eight and four lanes per score -> now: six layers of 1.1B widths at 300, 700, 1200, 2000 and 4500
// positions 238.5, 249.8, 278.9, 308.2, 370.5 -> 239.3, 240.7, 243.1, 255.2, 276.0; two of 7B widths at 300, 2000 and 4500 221.3, 242.2, 266.9 -> 221.1, 231.4, 248.8;
// four of 0.5B at 330, 2000 and 7000 144.3, 154.8, 209.2 -> 143.8, 145.5, 182.7.  (A thread per score on 256 threads, tiles of eight: four layers of 1.1B 182.3 at
// 300, 211.1 at 2000, where four lanes per score took 214.7.)  Tiles of 32 take 251.2 at 2000 and 171.2 at 7000, and 240.4 at 300, where nothing but the shared memory differs.
// From 256 or 128 scores on: 243.7 or 240.4 at 700, else the same.
constexpr int kStepTile = 16, kStepShared = 192;        // keys of a tile; scores of one that four lanes each share
template <typename KT, int EP>
__global__ void __launch_bounds__(kStepThreads) mixer_step_kernel(const MixerStep a) {
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    if ((int)blockIdx.x < a.n_mem) {
        mem_step(a, blockIdx.x, smem);
        return;
    }
    constexpr int CN = Chunk16<KT>::n;
    const GateAttn& A = a.at;
    const int H = A.heads, DS = A.dim_s, KV = A.kv_heads, group = H / KV, chunks = DS / CN;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = kStepThreads / 32;
    const AttnSmem<KT> sm(A, 1, a.tile, smem);
    const int row = KV * sm.ks;
    // tables and the norms' weights are on the way before the position is known
    const int pos = a.st->pos, len = pos + 1;
    for (int h = wid; h < H; h += nw)
        for (int g = lane; g < H; g += 32) cp_async4(sm.talk + h * sm.ts + g, A.talk + h * H + g);
    for (int i = tid; i < H; i += kStepThreads) { cp_async4(sm.bias + i, A.head_bias + i); cp_async4(sm.slope + i, A.slopes + i); }
    const int part16 = lane & 15;
    float qk[8];                                    // of the first 128 elements
#pragma unroll
    for (int i = 0; i < 8; i++) qk[i] = part16 + 16 * i < A.dim ? A.q_norm[part16 + 16 * i] * A.k_norm[part16 + 16 * i] : 0.f;
    int head_of[EP], key_of[EP];                    // this thread's output elements
#pragma unroll
    for (int e = 0; e < EP; e++) {
        const int el = 2 * (tid + e * kStepThreads), h = el / DS;
        head_of[e] = el < H * DS ? h : -1;
        key_of[e] = h / group * sm.ks + el - h * DS;
    }
    const int split = blockIdx.x - a.n_mem;
    int j0, j1;
    const int active = key_split(len, a.splits, a.grain, split, &j0, &j1);
    if (split >= active || pos >= A.max_seq) {
        cp_async_commit();
        cp_async_wait<0>();
        return;
    }
    int tile = a.grain;                             // a power of two
    while (tile < j1 - j0 && tile < a.tile) tile *= 2;
    const int tsh = 31 - __clz(tile);
    float* rnew = sm.slope + A.heads;
    KT* knew = a.key_copy ? reinterpret_cast<KT*>((reinterpret_cast<uintptr_t>(rnew + A.kv_heads) + 15) & ~(uintptr_t)15)
                          : static_cast<KT*>(A.cache) + (size_t)pos * A.kv_heads * A.dim_s;

    // cached keys of a tile, rows behind them zero
    const int pieces = chunks, step = kStepThreads / pieces, first = tid / pieces, piece = tid - first * pieces;
    auto load_tile = [&](int buf, int j) {
        const int rows = tile * KV, valid = max(0, min(rows, (min(j1, pos) - j) * KV));
        KT* dst = sm.k + (size_t)buf * a.tile * row + piece * CN;
        const KT* src = static_cast<const KT*>(A.cache) + (size_t)j * KV * DS + piece * CN;
        if (first < step)
            for (int r = first; r < rows; r += step) {
                if (r < valid) cp_async16(dst + r * sm.ks, src + (size_t)r * DS);
                else *reinterpret_cast<uint4*>(dst + r * sm.ks) = make_uint4(0u, 0u, 0u, 0u);
            }
        for (int i = tid; i < valid; i += kStepThreads) cp_async4(sm.r + buf * a.tile * KV + i, A.cache_r + (size_t)j * KV + i);
        cp_async_commit();
    };
    load_tile(0, j0);
    const float temp = query_temp(A, pos) * A.scale;
    pdl_wait();

    // this token's query, sixteen lanes per head, and its key where this CTA's range ends with it
    {
        const int sub = part16;
        const unsigned mask = 0xffffu << (lane & 16);
        for (int h = tid >> 4; h < H; h += kStepThreads / 16) {
            const float* p = a.proj + a.c.q + h * A.dim;
            float v[8], ss = 0.f;                   // the first 128 values are loaded at once
#pragma unroll
            for (int i = 0; i < 8; i++) {
                v[i] = sub + 16 * i < A.dim ? p[sub + 16 * i] : 0.f;
                ss = fmaf(v[i], v[i], ss);
            }
            for (int d = sub + 128; d < A.dim; d += 16) ss = fmaf(p[d], p[d], ss);
#pragma unroll
            for (int o = 1; o < 16; o *= 2) ss += __shfl_xor_sync(mask, ss, o);
            const float r = temp / sqrtf(ss / (float)A.dim + A.eps);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int d = sub + 16 * i;
                if (d < DS) sm.q[h * sm.qs + d] = v[i] * r * qk[i];
            }
            for (int d = sub + 128; d < DS; d += 16) sm.q[h * sm.qs + d] = d < A.dim ? p[d] * r * A.q_norm[d] * A.k_norm[d] : 0.f;
        }
    }
    if (j1 == len)
        for (int c = nw - 1 - wid; c < KV; c += nw) store_key<KT>(A, a.proj + a.c.k + c * A.dim, pos, c, lane, a.key_copy ? knew + c * DS : nullptr, rnew + c);

    float2 acc[EP];
#pragma unroll
    for (int e = 0; e < EP; e++) acc[e] = make_float2(0.f, 0.f);
    const unsigned quad = 0xfu << (lane & 28);
    int buf = 0;
    for (int j = j0; j < j1; j += tile, buf ^= 1) {
        if (j + tile < j1) load_tile(buf ^ 1, j + tile);
        else cp_async_commit();
        cp_async_wait<1>();
        KT* K = sm.k + (size_t)buf * a.tile * row;
        float* R = sm.r + buf * a.tile * KV;
        if (j1 == len && pos < j + tile) {          // the new key is this CTA's, and in this tile (the rows of the copies end before it)
            __syncthreads();
            KT* to = K + (size_t)(pos - j) * row;
            for (int i = tid; i < KV * DS; i += kStepThreads) to[i / DS * sm.ks + i % DS] = knew[i];
            for (int i = tid; i < KV; i += kStepThreads) R[(pos - j) * KV + i] = rnew[i];
        }
        __syncthreads();
        const int keys = min(tile, j1 - j);
        // every head and key: four lanes for each, lanes over the tile's rows, or one, lanes over heads
        auto each = [&](auto lanes, auto unit) {
            if constexpr (lanes == 4) {
                for (int u = tid >> 2; u < H << tsh; u += kStepThreads / 4) unit(u >> tsh, u & (tile - 1));
            } else {
                const int p_step = kStepThreads / H, h_step = kStepThreads - p_step * H;
                for (int p = tid / H, h = tid % H; p < keys;) {
                    unit(h, p);
                    p += p_step;
                    h += h_step;
                    if (h >= H) { h -= H; p++; }
                }
            }
        };
        auto weights = [&](auto lanes) {
            constexpr int LANES = lanes;
            const int sub = LANES == 4 ? lane & 3 : 0;
            auto total = [&](float v) {
                if (LANES == 4) {
                    v += __shfl_xor_sync(quad, v, 1);
                    v += __shfl_xor_sync(quad, v, 2);
                }
                return v;
            };
            each(lanes, [&](int h, int p) {
                const int c = h / group;
                const KT* kp = K + p * row + c * sm.ks;
                const float* qp = sm.q + h * sm.qs;
                float d0 = 0.f, d1 = 0.f;
#pragma unroll 2
                for (int ch = sub; ch < chunks; ch += LANES) {
                    float kk[CN];
                    Chunk16<KT>::load(kp + ch * CN, kk);
#pragma unroll
                    for (int i = 0; i < CN; i += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(qp + ch * CN + i);
                        d0 = fmaf(kk[i], v.x, d0);
                        d1 = fmaf(kk[i + 1], v.y, d1);
                        d0 = fmaf(kk[i + 2], v.z, d0);
                        d1 = fmaf(kk[i + 3], v.w, d1);
                    }
                }
                d0 = total(d0 + d1);
                if (sub == 0) {
                    const float z = d0 * (p < keys ? R[p * KV + c] : 0.f) - sm.slope[h] * (float)(pos - (j + p)) + sm.bias[h];
                    sm.w[h * sm.ws + p] = p < keys ? sigmoid(z) : 0.f;
                }
            });
            __syncthreads();
            each(lanes, [&](int h, int p) {
                const float* t = sm.talk + h * sm.ts;
                float v = 0.f;
#pragma unroll 8
                for (int g = sub; g < H; g += LANES) v = fmaf(t[g], sm.w[g * sm.ws + p], v);
                v = total(v);
                if (sub == 0) sm.mix[h * sm.ws + p] = v;
            });
        };
        if (H << tsh <= kStepShared) weights(std::integral_constant<int, 4>{});
        else weights(std::integral_constant<int, 1>{});
        __syncthreads();
#pragma unroll
        for (int e = 0; e < EP; e++)
            if (head_of[e] >= 0) {
#pragma unroll 4
                for (int p = 0; p < keys; p++) {
                    const float2 kv = pair_f32(K + p * row + key_of[e]);
                    const float m = sm.mix[head_of[e] * sm.ws + p];
                    acc[e].x = fmaf(m, kv.x, acc[e].x);
                    acc[e].y = fmaf(m, kv.y, acc[e].y);
                }
            }
        if (j + tile < j1) __syncthreads();         // w, mix and this buffer are used again
    }
#pragma unroll
    for (int e = 0; e < EP; e++)
        if (head_of[e] >= 0) *reinterpret_cast<float2*>(a.part + (size_t)split * H * DS + 2 * (tid + e * kStepThreads)) = acc[e];
}

constexpr int kJoinCols = 16, kJoinParts = 16;      // outputs per CTA, threads that share one output's splits

// Joins the key splits, and norms and gates the memory's outputs (one CTA per memory head).
__global__ void __launch_bounds__(kJoinCols * kJoinParts) mixer_join_kernel(const MixerStep a) {
    __shared__ __align__(16) float red[8];
    pdl_launch_dependents();
    int j0, j1;
    const int active = key_split(a.st->pos + 1, a.splits, a.grain, 0, &j0, &j1);
    pdl_wait();
    const MatMem& M = a.mem;
    const int nm = a.n_mem ? M.heads : 0;
    if ((int)blockIdx.x < nm) {
        const int head = blockIdx.x;
        const float* o = a.mem_o + head * M.vdim;
        float ss = 0.f;
        for (int v = threadIdx.x; v < M.vdim; v += blockDim.x) ss = fmaf(o[v], o[v], ss);
        float total[1] = {ss};
        sums8(total, red);
        const float r = 1.0f / sqrtf(total[0] / (float)M.vdim + M.eps);
        for (int v = threadIdx.x; v < M.vdim; v += blockDim.x) {
            const int c = head * M.vdim + v;
            a.mem_y[c] = o[v] * r * M.norm[c] * sigmoid(a.proj[a.c.mg + c]);
        }
        return;
    }
    const GateAttn& A = a.at;
    const int col = threadIdx.x % kJoinCols, grp = threadIdx.x / kJoinCols;
    const int e = (blockIdx.x - nm) * kJoinCols + col;
    const bool ok = e < A.heads * A.dim;
    const int src = ok ? e / A.dim * A.dim_s + e % A.dim : 0;
    const size_t stride = (size_t)A.heads * A.dim_s;
    float v = 0.f;
    if (ok) {
#pragma unroll 8
        for (int s = grp; s < active; s += kJoinParts) v += a.part[s * stride + src];
    }
    __shared__ float sum[kJoinParts][kJoinCols];
    sum[grp][col] = v;
    __syncthreads();
    if (grp == 0 && ok) {
#pragma unroll
        for (int g = 1; g < kJoinParts; g++) v += sum[g][col];
        a.attn_out[e] = v;
    }
}

__global__ void __launch_bounds__(256) resolve_kernel(const ResolveArgs a) {
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    pdl_wait();
    stage_layered(a.p, smem, smem + a.p.K, false);
    for (int i = threadIdx.x; i < a.p.k_valid; i += blockDim.x) a.out[i] = smem[i];
}

template <typename KT>
cudaError_t step_for(const MixerStep& a, size_t smem, bool pdl, cudaStream_t s) {
    const int pairs = (a.at.heads * a.at.dim_s / 2 + kStepThreads - 1) / kStepThreads;
    const int grid = a.n_mem + a.splits;
    auto run = [&](auto kern) {
        cudaError_t c = allow_smem(kern, std::max(smem, kModelSmem));
        return c != cudaSuccess ? c : launch_pdl(kern, grid, kStepThreads, smem, pdl, s, a);
    };
    if (pairs <= 1) return run(mixer_step_kernel<KT, 1>);
    if (pairs <= 2) return run(mixer_step_kernel<KT, 2>);
    if (pairs <= 4) return run(mixer_step_kernel<KT, 4>);
    if (pairs <= 8) return run(mixer_step_kernel<KT, 8>);
    return cudaErrorInvalidValue;
}

}  // namespace

namespace {

template <typename F>
cudaError_t by_rows(int R, int K, F f) {
    auto go = [&](auto r, auto ahead) { return f(r, ahead); };
    using std::integral_constant;
    if (K <= 2048)
        return R == 8 ? go(integral_constant<int, 8>{}, integral_constant<int, 1>{}) : R == 4 ? go(integral_constant<int, 4>{}, integral_constant<int, 1>{})
             : R == 2 ? go(integral_constant<int, 2>{}, integral_constant<int, 1>{}) : go(integral_constant<int, 1>{}, integral_constant<int, 1>{});
    return R == 4 ? go(integral_constant<int, 4>{}, integral_constant<int, 3>{}) : R == 2 ? go(integral_constant<int, 2>{}, integral_constant<int, 3>{})
                  : go(integral_constant<int, 1>{}, integral_constant<int, 3>{});
}
inline size_t rows_smem(int K) { return ((size_t)K + 72) * sizeof(float); }
inline int rows_grid(int K, int rows, int R, int most) {
    const int per = R * (kRowThreads / row_group(K));
    return std::max(1, std::min((rows + per - 1) / per, most));
}

}  // namespace

cudaError_t rows_attrs() {
    for (int k : {2048, 4096})
        for (int R : {1, 2, 4, 8}) {
            const cudaError_t c = by_rows(R, k, [&](auto r, auto ahead) {
                constexpr int RR = decltype(r)::value, A = decltype(ahead)::value;
                for (auto* f : {rows_kernel<EPI_STORE, RR, A>, rows_kernel<EPI_GELU, RR, A>, rows_kernel<EPI_LOGITS, RR, A>})
                    if (cudaError_t e = allow_smem(f, rows_smem(kMaxRow))) return e;
                if (cudaError_t e = allow_smem(rows_pair_kernel<RR, A>, rows_smem(kMaxRow))) return e;
                return allow_smem(rows_parts_kernel<RR, A>, rows_smem(kMaxRow));
            });
            if (c != cudaSuccess) return c;
        }
    return cudaSuccess;
}

cudaError_t launch_rows(const PhaseArgs& a, int epi, int sms, bool pdl, cudaStream_t s) {
    const int R = rows_at_a_time(a.K, a.rows[0], sms);
    return by_rows(R, a.K, [&](auto r, auto ahead) {
        constexpr int RR = decltype(r)::value, A = decltype(ahead)::value;
        auto kern = epi == EPI_GELU ? rows_kernel<EPI_GELU, RR, A> : epi == EPI_LOGITS ? rows_kernel<EPI_LOGITS, RR, A> : rows_kernel<EPI_STORE, RR, A>;
        return launch_pdl(kern, rows_grid(a.K, a.rows[0], R, 2 * sms), kRowThreads, rows_smem(a.K), pdl, s, a);
    });
}

cudaError_t launch_rows_pair(const PhaseArgs& a, const PhaseArgs& b, int sms, bool pdl, cudaStream_t s) {
    const int K = std::max(a.K, b.K);
    const int R = rows_at_a_time(K, a.rows[0] + b.rows[0], sms);
    // CTAs in proportion to the bytes
    const long long wa = (long long)a.rows[0] * a.K, wb = (long long)b.rows[0] * b.K;
    const int most = (int)std::max(1ll, std::min(2ll * sms - 1, (wa * 2 * sms + (wa + wb) / 2) / (wa + wb)));
    const int ga = rows_grid(a.K, a.rows[0], R, most), gb = rows_grid(b.K, b.rows[0], R, 2 * sms - most);
    return by_rows(R, K, [&](auto r, auto ahead) {
        return launch_pdl(rows_pair_kernel<decltype(r)::value, decltype(ahead)::value>, ga + gb, kRowThreads, rows_smem(K), pdl, s, a, b, ga);
    });
}

cudaError_t launch_rows_parts(const PhaseArgs& a, PhaseParts& p, int sms, bool pdl, cudaStream_t s) {
    long long all = 0;
    for (int k = 0; k < p.n; k++) all += p.rows[k];
    const int R = rows_at_a_time(a.K, all, sms);
    for (int k = 0; k < p.n; k++) p.first[k + 1] = p.first[k] + rows_grid(a.K, p.rows[k], R, std::max(1, (int)(2ll * sms * p.rows[k] / all)));
    return by_rows(R, a.K, [&](auto r, auto ahead) {
        return launch_pdl(rows_parts_kernel<decltype(r)::value, decltype(ahead)::value>, p.first[p.n], kRowThreads, rows_smem(a.K), pdl, s, a, p);
    });
}

size_t mixer_step_smem(const GateAttn& at, const MatMem& mem, bool f32_cache, int* tile) {
    const size_t need_mem = (40 + kStepThreads + 2 * (size_t)mem.dim) * sizeof(float);
    size_t need = attn_smem(at, 1, f32_cache ? 4 : 2, kStepTile, tile);
    if (need == 0) return 0;
    need += step_extra(at);
    if (const size_t key = step_key(at, f32_cache ? 4 : 2); need + key <= kModelSmem) need += key;
    return need > need_mem ? need : need_mem;
}

cudaError_t launch_mixer_step(const MixerStep& a, bool f32_cache, bool pdl, cudaStream_t s) {
    MixerStep b = a;
    int tile;
    const size_t smem = mixer_step_smem(a.at, a.mem, f32_cache, &tile), kt = f32_cache ? 4 : 2;
    b.key_copy = smem >= attn_smem(a.at, 1, (int)kt, kStepTile, &tile) + step_extra(a.at) + step_key(a.at, kt);
    return f32_cache ? step_for<float>(b, smem, pdl, s) : step_for<__nv_bfloat16>(b, smem, pdl, s);
}

cudaError_t launch_mixer_join(const MixerStep& a, bool pdl, cudaStream_t s) {
    const int nm = a.n_mem ? a.mem.heads : 0;
    return launch_pdl(mixer_join_kernel, nm + (a.at.heads * a.at.dim + kJoinCols - 1) / kJoinCols, kJoinCols * kJoinParts, 0, pdl, s, a);
}

cudaError_t launch_resolve(const ResolveArgs& a, bool pdl, cudaStream_t s) {
    const size_t smem = ((size_t)a.p.K + 72) * sizeof(float);
    cudaError_t c = allow_smem(resolve_kernel, kModelSmem);
    return c != cudaSuccess ? c : launch_pdl(resolve_kernel, 1, 256, smem, pdl, s, a);
}

}  // namespace mg
