// Portions of a prompt of a layer-described model: row-wise kernels, attention on
// the CUDA cores (32-bit mode and head counts the tensor-core kernel does not take), and the matrix
// memory in chunked form: every chunk's contribution in parallel, one pass over the chunks, then every
// chunk's outputs in parallel.
#include <type_traits>

#include "layered_ops.cuh"

namespace mg {

namespace {

template <typename AT>
__global__ void __launch_bounds__(256) embed_rows_kernel(WeightView embed, int ld_embed, const float* pos_tab, const int* tokens,
                                                         int pos0, int width, float* x, AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, token = tokens[r];
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float v = embed_value(embed, FMT_BF16, ld_embed, token, i) + (pos_tab ? pos_tab[(size_t)(pos0 + r) * width + i] : 0.f);
        x[(size_t)r * width + i] = v;
        from_f32(v, act + (size_t)r * ld_act + i);
    }
}

// One warp per (token, query head or key head).
template <typename AT>
__global__ void __launch_bounds__(256) qk_rows_kernel(GateAttn A, const float* proj, int ldp, int q_col, int k_col, int pos0, int n,
                                                      AT* qh) {
    pdl_launch_dependents();
    pdl_wait();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int per = A.heads + A.kv_heads, t = w / per, h = w - t * per;
    if (t >= n) return;
    const float* row = proj + (size_t)t * ldp;
    if (h < A.heads)
        norm_query(A, row + q_col + h * A.dim, query_temp(A, pos0 + t), qh + ((size_t)t * A.heads + h) * A.dim_s, lane);
    else
        store_key<AT>(A, row + k_col + (h - A.heads) * A.dim, pos0 + t, h - A.heads, lane);
}

// The same with four values per load, sixteen lanes per (token, head): sizes and columns that are multiples of four, heads of up
// to 64 C values.  A prompt of 2048 tokens, 36 heads of 64: 25 us with a warp per head and a value per load.
template <typename AT, int C>
__global__ void __launch_bounds__(256) qk_quads_kernel(GateAttn A, const float* proj, int ldp, int q_col, int k_col, int pos0, int n, AT* qh) {
    pdl_launch_dependents();
    pdl_wait();
    const int u = (blockIdx.x * 256 + threadIdx.x) >> 4, l = threadIdx.x & 15;
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    const int per = A.heads + A.kv_heads, t = u / per, h = u - t * per;
    if (t >= n) return;
    const bool query = h < A.heads;
    const float* src = proj + (size_t)t * ldp + (query ? q_col + h * A.dim : k_col + (h - A.heads) * A.dim);
    float v[C][4], w[C][4], ss = 0.f;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int d = 4 * (l + 16 * c);
#pragma unroll
        for (int i = 0; i < 4; i++) { v[c][i] = 0.f; w[c][i] = 0.f; }
        if (d < A.dim) {
            load_values<4>(src + d, v[c]);
            if (query) {
                float k[4];
                load_values<4>(A.q_norm + d, w[c]);
                load_values<4>(A.k_norm + d, k);
#pragma unroll
                for (int i = 0; i < 4; i++) w[c][i] *= k[i];
            }
        }
        if (!query) {               // a key's 1 / rms is that of the row as stored
#pragma unroll
            for (int i = 0; i < 4; i++) {
                AT r;
                from_f32(v[c][i], &r);
                v[c][i] = to_f32(r);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) ss = fmaf(v[c][i], v[c][i], ss);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(mask, ss, o);
    const float rms = sqrtf(ss / (float)A.dim + A.eps);
    AT* dst = query ? qh + ((size_t)t * A.heads + h) * A.dim_s : static_cast<AT*>(A.cache) + ((size_t)(pos0 + t) * A.kv_heads + h - A.heads) * A.dim_s;
    const float r = query ? query_temp(A, pos0 + t) * A.scale / rms : 1.f;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int d = 4 * (l + 16 * c);
        if (query) {
#pragma unroll
            for (int i = 0; i < 4; i++) v[c][i] *= r * w[c][i];
        }
        if (d < A.dim_s) store_values<4>(v[c], dst + d);
    }
    if (!query && l == 0) A.cache_r[(size_t)(pos0 + t) * A.kv_heads + h - A.heads] = 1.0f / rms;
}

template <typename KT, int NQ, int EP>
__global__ void __launch_bounds__(kAttnThreads) gate_attn_rows_kernel(GateAttn A, const KT* qh, int pos0, int n, int tile, KT* out,
                                                                      int ld_out) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const AttnSmem<KT> sm(A, NQ, tile, smem);
    const int t0 = (gridDim.x - 1 - blockIdx.x) * NQ;      // the longest rows first
    const int row = A.heads * A.dim_s;
    for (int i = threadIdx.x; i < NQ * row; i += kAttnThreads)
        sm.q[i / A.dim_s * sm.qs + i % A.dim_s] = t0 + i / row < n ? to_f32(qh[(size_t)t0 * row + i]) : 0.f;
    sm.load_tables(A);
    __syncthreads();
    const int last = min(t0 + NQ, n) - 1;
    float acc[NQ][EP][2] = {};
    attend<KT, NQ, EP>(A, sm, pos0 + t0, 0, pos0 + last + 1, tile, acc);
#pragma unroll
    for (int e = 0; e < EP; e++) {
        const int el = 2 * (threadIdx.x + e * kAttnThreads);
        if (el >= row) continue;
        const int h = el / A.dim_s, d = el - h * A.dim_s;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            if (t0 + q > last) continue;
            KT* o = out + (size_t)(t0 + q) * ld_out + h * A.dim + d;
            if (d < A.dim) from_f32(acc[q][e][0], o);
            if (d + 1 < A.dim) from_f32(acc[q][e][1], o + 1);
        }
    }
}

template <typename AT>
__global__ void __launch_bounds__(256) post_rows_kernel(float* x, const float* z0, const float* z1, const float* w0, const float* w1,
                                                        const float* post_w, float eps, int width, AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float y[];
    __shared__ float red[40];
    const size_t r = blockIdx.x;
    const float inv = 1.0f / (float)width;
    const float *a = z0 + r * width, *b = z1 ? z1 + r * width : nullptr;
    float ra = 1.f, rb = 0.f, ss = 0.f;
    if (b) {
        float s0 = 0.f, s1 = 0.f;
        for (int i = threadIdx.x; i < width; i += blockDim.x) { s0 = fmaf(a[i], a[i], s0); s1 = fmaf(b[i], b[i], s1); }
        ra = 0.5f / sqrtf(block_sum(s0, red) * inv + eps);
        rb = 0.5f / sqrtf(block_sum(s1, red) * inv + eps);
    }
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float v = b ? a[i] * ra * w0[i] + b[i] * rb * w1[i] : a[i];
        y[i] = v;
        ss = fmaf(v, v, ss);
    }
    const float rr = 1.0f / sqrtf(block_sum(ss, red) * inv + eps);
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float v = x[r * width + i] + y[i] * rr * (1.0f + post_w[i]);
        x[r * width + i] = v;
        from_f32(v, act + r * ld_act + i);
    }
}

// The same for widths that are multiples of four, up to 1024 C: a row stays in registers from its one load to its store, and
// the weights are under way while it is summed.  2048 rows of 2048, two branches: 21 us with loads value by value, twice.
template <typename AT, int C>
__global__ void __launch_bounds__(256) post_quads_kernel(float* x, const float* z0, const float* z1, const float* w0, const float* w1,
                                                         const float* post_w, float eps, int width, AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[72];
    const size_t r = blockIdx.x;
    const float inv = 1.0f / (float)width;
    float a[C][4], b[C][4], y[C][4], p[C][4], u[C][4], w[C][4];
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int i = 4 * (threadIdx.x + 256 * c);
#pragma unroll
        for (int q = 0; q < 4; q++) { a[c][q] = b[c][q] = y[c][q] = p[c][q] = u[c][q] = w[c][q] = 0.f; }
        if (i < width) {
            load_values<4>(z0 + r * width + i, a[c]);
            if (z1) {
                load_values<4>(z1 + r * width + i, b[c]);
                load_values<4>(w0 + i, u[c]);
                load_values<4>(w1 + i, w[c]);
            }
            load_values<4>(x + r * width + i, y[c]);
            load_values<4>(post_w + i, p[c]);
        }
    }
    if (z1) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int q = 0; q < 4; q++) { s0 = fmaf(a[c][q], a[c][q], s0); s1 = fmaf(b[c][q], b[c][q], s1); }
        const float2 t = block_sum2(s0, s1, red);
        const float ra = 0.5f / sqrtf(t.x * inv + eps), rb = 0.5f / sqrtf(t.y * inv + eps);
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[c][q] = a[c][q] * ra * u[c][q] + b[c][q] * rb * w[c][q];
    }
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int q = 0; q < 4; q++) ss = fmaf(a[c][q], a[c][q], ss);
    const float rr = 1.0f / sqrtf(block_sum(ss, red) * inv + eps);
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int i = 4 * (threadIdx.x + 256 * c);
        if (i >= width) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) y[c][q] += a[c][q] * rr * (1.0f + p[c][q]);
        store_values<4>(y[c], x + r * width + i);
        store_values<4>(y[c], act + r * ld_act + i);
    }
}

// Mean and 1 / sqrt(spread + eps) of row y for a norm of the given kind; a thread reads V values at a time, those
// it would write in a loop of the same shape.
template <int V>
__device__ __forceinline__ float2 row_norm(const float* y, int kind, float eps, int width, float* red) {
    const float inv = 1.0f / (float)width;
    float s = 0.f;
    for (int i = threadIdx.x * V; i < width; i += blockDim.x * V) {
        float v[V];
        load_values<V>(y + i, v);
#pragma unroll
        for (int q = 0; q < V; q++) s += kind == NORM_LAYER ? v[q] : v[q] * v[q];
    }
    s = block_sum(s, red) * inv;
    if (kind != NORM_LAYER) return make_float2(0.f, 1.0f / sqrtf(s + eps));
    float d = 0.f;
    for (int i = threadIdx.x * V; i < width; i += blockDim.x * V) {
        float v[V];
        load_values<V>(y + i, v);
#pragma unroll
        for (int q = 0; q < V; q++) d = fmaf(v[q] - s, v[q] - s, d);
    }
    return make_float2(s, 1.0f / sqrtf(block_sum(d, red) * inv + eps));
}

template <typename AT>
__global__ void __launch_bounds__(256) last_norm_rows_kernel(const float* x, const int* rows, const float* w, int kind, float eps, int width,
                                                             AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[40];
    const float* a = x + (size_t)rows[blockIdx.x] * width;
    const float2 n = row_norm<1>(a, kind, eps, width, red);
    const float one = kind == NORM_RMS_AROUND_ZERO ? 1.0f : 0.0f;
    for (int i = threadIdx.x; i < width; i += blockDim.x) from_f32((a[i] - n.x) * n.y * (one + w[i]), act + (size_t)blockIdx.x * ld_act + i);
}

template <typename AT, int V>
__global__ void __launch_bounds__(256) prenorm_rows_kernel(const PrenormRows a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float y[];
    __shared__ float red[40];
    const int W = a.width, step = 256 * V;
    const size_t r = blockIdx.x;
    float* x = a.x + r * W;
    AT* act = static_cast<AT*>(a.act) + r * a.ld_act;
    for (int i = threadIdx.x * V; i < W; i += step) {
        float v[V];
        load_values<V>(x + i, v);
        if (a.z) {
            float z[V], ls[V];
            load_values<V>(a.z + r * W + i, z);
            load_values<V>(a.ls + i, ls);
#pragma unroll
            for (int q = 0; q < V; q++) v[q] += a.mult * (ls[q] * z[q]);
            store_values<V>(v, x + i);
        }
        if (a.norm_w) store_values<V>(v, y + i);
        else if (a.act) store_values<V>(v, act + i);
        if (a.cat) {
            load_values<V>(a.cat + r * W + i, v);
            store_values<V>(v, act + W + i);
        }
    }
    if (!a.norm_w) return;
    const float2 n = row_norm<V>(y, a.kind, a.eps, W, red);
    const float one = a.kind == NORM_RMS_AROUND_ZERO ? 1.0f : 0.0f;
    for (int i = threadIdx.x * V; i < W; i += step) {
        float v[V], w[V];
        load_values<V>(y + i, v);
        load_values<V>(a.norm_w + i, w);
#pragma unroll
        for (int q = 0; q < V; q++) v[q] = (v[q] - n.x) * n.y * (one + w[q]);
        if (a.h) store_values<V>(v, a.h + r * W + i);
        else store_values<V>(v, act + i);
    }
}

// ---------------------------------------------------------------------
// Matrix memory in chunks of kMemChunk tokens.
// ---------------------------------------------------------------------

// One CTA per head, one warp per chunk: gates, the log-forget sum inside each chunk, and the running maximum
// m_t = max(f_t + m_{t-1}, i_t) as a scan of the maps m -> max(m + f, i): within halves of a chunk by
// shuffles, across the chunks through shared memory.
constexpr int kGateWarps = 32;

__global__ void __launch_bounds__(kGateWarps * 32) mem_gates_kernel(MatMem M, int i_col, int f_col, const float* proj, int ldp, int pos0,
                                                                    int n, MemRows w) {
    pdl_launch_dependents();
    pdl_wait();
    static_assert(kMemChunk == 64, "a warp holds a chunk as two tokens per lane");
    __shared__ double sum_f[kGateWarps];
    __shared__ float top_i[kGateWarps], m_end;
    const int h = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float m = pos0 == 0 ? 0.f : M.m[(pos0 & 1) * M.heads + h];      // before the chunks of this pass
    if (threadIdx.x == 0) w.m0[h] = m;
    const float ib = M.i_bias[h], fb = M.f_bias[h];
    for (int c0 = 0; c0 * kMemChunk < n; c0 += kGateWarps) {
        const int t0 = (c0 + warp) * kMemChunk;
        float ig[2], mi[2];
        double b[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int t = t0 + 32 * k + lane;
            ig[k] = -INFINITY;                      // tokens past n change nothing: f = 0, i = -inf
            float fg = 0.f;
            if (t < n) {
                ig[k] = soft_cap(proj[(size_t)t * ldp + i_col + h] + ib, M.cap);
                fg = log_sigmoid(soft_cap(proj[(size_t)t * ldp + f_col + h] + fb, M.cap));
            }
            b[k] = (double)fg;
            mi[k] = ig[k];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double pb = __shfl_up_sync(MG_FULL_MASK, b[k], o);
                const float pm = __shfl_up_sync(MG_FULL_MASK, mi[k], o);
                if (lane >= o) { mi[k] = fmaxf((float)((double)pm + b[k]), mi[k]); b[k] += pb; }
            }
        }
        const double b0 = __shfl_sync(MG_FULL_MASK, b[0], 31);
        const float i0 = __shfl_sync(MG_FULL_MASK, mi[0], 31);
        mi[1] = fmaxf((float)((double)i0 + b[1]), mi[1]);
        b[1] += b0;
        __syncthreads();                            // the last pass's sums have been read
        if (lane == 31) { sum_f[warp] = b[1]; top_i[warp] = mi[1]; }
        __syncthreads();
        float before = m;
        for (int c = 0; c < warp; c++) before = fmaxf((float)((double)before + sum_f[c]), top_i[c]);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int t = t0 + 32 * k + lane;
            const float mt = fmaxf((float)((double)before + b[k]), mi[k]);
            if (t < n) {
                w.b[(size_t)h * n + t] = b[k];
                w.ig[(size_t)h * n + t] = ig[k];
                w.mm[(size_t)h * n + t] = mt;
            }
            if (k == 1 && lane == 31) {
                if (t0 < n) w.g[(size_t)h * ((n + kMemChunk - 1) / kMemChunk) + c0 + warp] = expf((float)b[1] + before - mt);
                if (warp == kGateWarps - 1) m_end = mt;
            }
        }
        __syncthreads();
        m = m_end;
    }
    if (threadIdx.x == 0) M.m[((pos0 + n) & 1) * M.heads + h] = m;
}

// Running maximum before token t0 of the portion (the state's own slot may be overwritten by now).
__device__ __forceinline__ float mem_before(const MemRows& w, int h, int n, int t0) {
    return t0 > 0 ? w.mm[(size_t)h * n + t0 - 1] : w.m0[h];
}

// U[chunk][head] = sum over the chunk of exp(b_T - b_s + i_s - m_T) k_s v_s^T, a 64 x 64 tile per CTA.
__global__ void __launch_bounds__(256) mem_chunk_kernel(MatMem M, int k_col, int v_col, const float* proj, int ldp, int n, int vtiles,
                                                        MemRows w) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float Ks[kMemChunk][68], Vs[kMemChunk][68];
    const int ch = blockIdx.x, h = blockIdx.y, d0 = blockIdx.z / vtiles * 64, v0 = blockIdx.z % vtiles * 64;
    const int t0 = ch * kMemChunk, T = min(kMemChunk, n - t0);
    const double bT = w.b[(size_t)h * n + t0 + T - 1];
    const float mT = w.mm[(size_t)h * n + t0 + T - 1];
    // every load at once; a token's factor is formed by one thread, not by each that holds one of its values
    __shared__ float fs[kMemChunk];
    constexpr int kLoads = kMemChunk * 64 / 256;
    const int c = threadIdx.x & 63, s0 = threadIdx.x >> 6;
    float k[kLoads], v[kLoads];
#pragma unroll
    for (int r = 0; r < kLoads; r++) {
        const int s = s0 + 4 * r;
        const float* row = proj + (size_t)(t0 + s) * ldp;
        k[r] = s < T && d0 + c < M.dim ? row[k_col + h * M.dim + d0 + c] : 0.f;
        v[r] = s < T && v0 + c < M.vdim ? row[v_col + h * M.vdim + v0 + c] : 0.f;
    }
    if (threadIdx.x < kMemChunk) {
        const int s = threadIdx.x;
        fs[s] = s < T ? expf((float)(bT - w.b[(size_t)h * n + t0 + s]) + w.ig[(size_t)h * n + t0 + s] - mT) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kLoads; r++) {
        const int s = s0 + 4 * r;
        Ks[s][c] = s < T && d0 + c < M.dim ? k[r] * fs[s] : 0.f;
        Vs[s][c] = v[r];
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4] = {}, nk[4] = {};
#pragma unroll 8
    for (int s = 0; s < kMemChunk; s++) {
        const float4 a = *reinterpret_cast<const float4*>(&Ks[s][ty * 4]), b = *reinterpret_cast<const float4*>(&Vs[s][tx * 4]);
        const float aa[4] = {a.x, a.y, a.z, a.w}, bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            nk[i] += aa[i];
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(aa[i], bb[j], acc[i][j]);
        }
    }
    float* U = w.U + ((size_t)ch * M.heads + h) * M.dim * M.vdim;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = d0 + ty * 4 + i;
        if (d >= M.dim) continue;
        if (v0 == 0 && tx == 0) w.nU[((size_t)ch * M.heads + h) * M.dim + d] = nk[i];
        float* to = U + (size_t)d * M.vdim + v0 + tx * 4;
        if ((M.vdim & 3) == 0) {
            if (v0 + tx * 4 < M.vdim) *reinterpret_cast<float4*>(to) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (v0 + tx * 4 + j < M.vdim) to[j] = acc[i][j];
    }
}

// Pass over the chunks: U becomes the state BEFORE each chunk, and the state after the last is stored.
__global__ void __launch_bounds__(256) mem_scan_kernel(MatMem M, int pos0, int n, int chunks, MemRows w) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t per = (size_t)M.dim * M.vdim, all = M.heads * per, nall = (size_t)M.heads * M.dim;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= all + nall) return;
    const bool is_n = e >= all;
    const size_t i = is_n ? e - all : e;
    const int h = (int)(i / (is_n ? (size_t)M.dim : per));
    float* U = is_n ? w.nU + i : w.U + i;
    const size_t stride = is_n ? nall : all;
    float s = 0.f;
    if (pos0 > 0) s = is_n ? M.nrm[(pos0 & 1) * nall + i] : M.S[i];
    const float* g = w.g + (size_t)h * chunks;
    for (int c0 = 0; c0 < chunks; c0 += 8) {        // eight chunks' loads in flight
        float u[8], gg[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            u[i] = c0 + i < chunks ? U[(c0 + i) * stride] : 0.f;
            gg[i] = c0 + i < chunks ? g[c0 + i] : 1.f;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (c0 + i < chunks) U[(c0 + i) * stride] = s;
            s = fmaf(gg[i], s, u[i]);
        }
    }
    if (is_n) M.nrm[((pos0 + n) & 1) * nall + i] = s;
    else M.S[i] = s;
}

// Outputs of one chunk and head, 64 value columns per CTA.
__global__ void __launch_bounds__(256) mem_out_kernel(MatMem M, int q_col, int k_col, int v_col, const float* proj, int ldp,
                                                      int n, MemRows w) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float Qs[32][68], Ks[32][68], Ss[32][68];
    __shared__ __align__(16) float P[kMemChunk][68];            // [s][t]
    __shared__ float nq_s[kMemChunk], ns[32];
    __shared__ double bs[kMemChunk];
    __shared__ float is[kMemChunk], ms[kMemChunk];
    float (*Vs)[68] = reinterpret_cast<float (*)[68]>(&Qs[0][0]);   // 64 rows over Qs and Ks once they are consumed
    static_assert(sizeof(Qs) + sizeof(Ks) == 64 * 68 * 4, "the value tile reuses the query and key tiles");
    const int ch = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 64;
    const int t0 = ch * kMemChunk, T = min(kMemChunk, n - t0);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (threadIdx.x < kMemChunk) {
        const int t = threadIdx.x;
        bs[t] = t < T ? w.b[(size_t)h * n + t0 + t] : 0.0;
        is[t] = t < T ? w.ig[(size_t)h * n + t0 + t] : -INFINITY;
        ms[t] = t < T ? w.mm[(size_t)h * n + t0 + t] : 0.f;
    }
    const float mprev = mem_before(w, h, n, t0);
    const float qscale = 1.0f / sqrtf((float)M.dim);
    const float* U = w.U + ((size_t)ch * M.heads + h) * M.dim * M.vdim;
    const float* nU = w.nU + ((size_t)ch * M.heads + h) * M.dim;
    float pa[4][4] = {}, oa[4][4] = {};         // rows t = ty*4.., columns s or v = tx*4..
    float nq = 0.f;                             // thread t < 64: n_prev . q_t
    // the next 32 columns are under way while these are multiplied
    float q[8], k[8], u[8], nn = 0.f;
    auto load = [&](int k0) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = threadIdx.x + 256 * r, t = i >> 5, d = i & 31, sd = i >> 6, sv = i & 63;
            const float* row = proj + (size_t)(t0 + t) * ldp + h * M.dim + k0 + d;
            const bool in = t < T && k0 + d < M.dim;
            q[r] = in ? row[q_col] : 0.f;
            k[r] = in ? row[k_col] : 0.f;
            u[r] = k0 + sd < M.dim && v0 + sv < M.vdim ? U[(size_t)(k0 + sd) * M.vdim + v0 + sv] : 0.f;
        }
        if (threadIdx.x < 32) nn = k0 + threadIdx.x < M.dim ? nU[k0 + threadIdx.x] : 0.f;
    };
    load(0);
    for (int k0 = 0; k0 < M.dim; k0 += 32) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = threadIdx.x + 256 * r;
            Qs[i & 31][i >> 5] = q[r] * qscale;
            Ks[i & 31][i >> 5] = k[r];
            Ss[i >> 6][i & 63] = u[r];
        }
        if (threadIdx.x < 32) ns[threadIdx.x] = nn;
        __syncthreads();
        if (k0 + 32 < M.dim) load(k0 + 32);
        if (threadIdx.x < kMemChunk) {
#pragma unroll 8
            for (int d = 0; d < 32; d++) nq = fmaf(ns[d], Qs[d][threadIdx.x], nq);
        }
#pragma unroll 8
        for (int d = 0; d < 32; d++) {
            const float4 a = *reinterpret_cast<const float4*>(&Qs[d][ty * 4]), b = *reinterpret_cast<const float4*>(&Ks[d][tx * 4]),
                         c = *reinterpret_cast<const float4*>(&Ss[d][tx * 4]);
            const float aa[4] = {a.x, a.y, a.z, a.w}, bb[4] = {b.x, b.y, b.z, b.w}, cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    pa[i][j] = fmaf(aa[i], bb[j], pa[i][j]);
                    oa[i][j] = fmaf(aa[i], cc[j], oa[i][j]);
                }
        }
    }
    __syncthreads();
    float val[kMemChunk * 64 / 256];
#pragma unroll
    for (int r = 0; r < kMemChunk * 64 / 256; r++) {
        const int s = (threadIdx.x >> 6) + 4 * r, c = threadIdx.x & 63;
        val[r] = s < T && v0 + c < M.vdim ? proj[(size_t)(t0 + s) * ldp + v_col + h * M.vdim + v0 + c] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = ty * 4 + i;
        const float inter = t < T ? expf((float)bs[t] + mprev - ms[t]) : 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = tx * 4 + j;
            P[s][t] = s <= t && t < T ? pa[i][j] * expf((float)(bs[t] - bs[s]) + is[s] - ms[t]) : 0.f;
            oa[i][j] *= inter;
        }
    }
#pragma unroll
    for (int r = 0; r < kMemChunk * 64 / 256; r++) Vs[(threadIdx.x >> 6) + 4 * r][threadIdx.x & 63] = val[r];
    __syncthreads();
    if (threadIdx.x < kMemChunk) {
        const int t = threadIdx.x;
        float d = nq * (t < T ? expf((float)bs[t] + mprev - ms[t]) : 0.f);
        for (int s = 0; s < kMemChunk; s++) d += P[s][t];
        nq_s[t] = 1.0f / (fmaxf(fabsf(d), expf(-ms[t])) + 1e-6f);
    }
#pragma unroll 8
    for (int s = 0; s < kMemChunk; s++) {
        const float4 a = *reinterpret_cast<const float4*>(&P[s][ty * 4]), b = *reinterpret_cast<const float4*>(&Vs[s][tx * 4]);
        const float aa[4] = {a.x, a.y, a.z, a.w}, bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) oa[i][j] = fmaf(aa[i], bb[j], oa[i][j]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = ty * 4 + i;
        if (t >= T) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int v = v0 + tx * 4 + j;
            if (v < M.vdim) w.o[(size_t)(t0 + t) * M.heads * M.vdim + h * M.vdim + v] = oa[i][j] * nq_s[t];
        }
    }
}

// One warp per (token, head): unit rms, norm weight, output gate.
template <typename AT>
__global__ void __launch_bounds__(256) head_norm_rows_kernel(int heads, int vdim, float eps, const float* norm, const float* gate, int ldg,
                                                             int gate_kind, int n, const float* o, AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    const int wq = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int t = wq / heads, h = wq - t * heads;
    if (t >= n) return;
    const float* p = o + ((size_t)t * heads + h) * vdim;
    float ss = 0.f;
    for (int v = lane; v < vdim; v += 32) ss = fmaf(p[v], p[v], ss);
    const float r = 1.0f / sqrtf(warp_sum(ss) / (float)vdim + eps);
    for (int v = lane; v < vdim; v += 32) {
        const int c = h * vdim + v;
        const float g = gate[(size_t)t * ldg + c];
        from_f32(p[v] * r * norm[c] * (gate_kind == GATE_SILU ? silu(g) : sigmoid(g)), act + (size_t)t * ld_act + c);
    }
}

// The same with a quad of values per lane and `lanes` lanes (a power of two) per head: head sizes that are whole
// quads, up to 128.
template <typename AT>
__global__ void __launch_bounds__(256) head_norm_quads_kernel(int heads, int vdim, int lanes, float eps, const float* norm, const float* gate,
                                                              int ldg, int gate_kind, int n, const float* o, AT* act, int ld_act) {
    pdl_launch_dependents();
    pdl_wait();
    const int unit = (blockIdx.x * 256 + threadIdx.x) / lanes, sub = threadIdx.x & (lanes - 1);
    const int t = unit / heads, h = unit - t * heads, c = h * vdim + sub * 4;
    const bool in = t < n && sub * 4 < vdim;
    float v[4] = {}, g[4], w[4];
    if (in) {
        load_values<4>(o + (size_t)t * heads * vdim + c, v);
        load_values<4>(gate + (size_t)t * ldg + c, g);
        load_values<4>(norm + c, w);
    }
    float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
    for (int m = lanes / 2; m > 0; m >>= 1) ss += __shfl_xor_sync(MG_FULL_MASK, ss, m);
    const float r = 1.0f / sqrtf(ss / (float)vdim + eps);
    if (!in) return;
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] *= r * w[q] * (gate_kind == GATE_SILU ? silu(g[q]) : sigmoid(g[q]));
    store_values<4>(v, act + (size_t)t * ld_act + c);
}

template <typename KT, int NQ>
cudaError_t attn_rows_for(const GateAttn& at, const void* qh, int pos0, int n, void* out, int ld_out, bool pdl, cudaStream_t s) {
    int tile;
    const size_t smem = attn_smem(at, NQ, sizeof(KT), 32, &tile);
    if (!smem) return cudaErrorInvalidValue;
    auto run = [&](auto kern) {
        cudaError_t c = allow_smem(kern, kModelSmem);
        if (c != cudaSuccess) return c;
        launch_pdl(kern, (n + NQ - 1) / NQ, kAttnThreads, smem, pdl, s, at, (const KT*)qh, pos0, n, tile, (KT*)out, ld_out);
        return cudaGetLastError();
    };
    switch (attn_pairs(at)) {
        case 1: return run(gate_attn_rows_kernel<KT, NQ, 1>);
        case 2: return run(gate_attn_rows_kernel<KT, NQ, 2>);
        case 4: return run(gate_attn_rows_kernel<KT, NQ, 4>);
        case 8: return run(gate_attn_rows_kernel<KT, NQ, 8>);
        case 16: return run(gate_attn_rows_kernel<KT, NQ, 16>);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_embed_rows(const WeightView& embed, int ld_embed, const float* pos_tab, const int* tokens, int pos0, int n,
                              int width, float* x, void* act, int ld_act, bool f32, bool pdl, cudaStream_t s) {
    if (f32) launch_pdl(embed_rows_kernel<float>, n, 256, 0, pdl, s, embed, ld_embed, pos_tab, tokens, pos0, width, x, (float*)act, ld_act);
    else launch_pdl(embed_rows_kernel<__nv_bfloat16>, n, 256, 0, pdl, s, embed, ld_embed, pos_tab, tokens, pos0, width, x, (__nv_bfloat16*)act, ld_act);
    return cudaGetLastError();
}

cudaError_t launch_qk_rows(const GateAttn& at, const float* proj, int ldp, int q_col, int k_col, int pos0, int n, void* qh, bool f32,
                           bool pdl, cudaStream_t s) {
    if (((at.dim | ldp | q_col | k_col) & 3) == 0 && at.dim <= 256) {
        auto quads = [&](auto* q) {
            using AT = std::remove_pointer_t<decltype(q)>;
            const int grid = (n * (at.heads + at.kv_heads) + 15) / 16;
            if (at.dim <= 64) launch_pdl(qk_quads_kernel<AT, 1>, grid, 256, 0, pdl, s, at, proj, ldp, q_col, k_col, pos0, n, q);
            else if (at.dim <= 128) launch_pdl(qk_quads_kernel<AT, 2>, grid, 256, 0, pdl, s, at, proj, ldp, q_col, k_col, pos0, n, q);
            else launch_pdl(qk_quads_kernel<AT, 4>, grid, 256, 0, pdl, s, at, proj, ldp, q_col, k_col, pos0, n, q);
            return cudaGetLastError();
        };
        return f32 ? quads((float*)qh) : quads((__nv_bfloat16*)qh);
    }
    const int grid = (n * (at.heads + at.kv_heads) + 7) / 8;
    if (f32) launch_pdl(qk_rows_kernel<float>, grid, 256, 0, pdl, s, at, proj, ldp, q_col, k_col, pos0, n, (float*)qh);
    else launch_pdl(qk_rows_kernel<__nv_bfloat16>, grid, 256, 0, pdl, s, at, proj, ldp, q_col, k_col, pos0, n, (__nv_bfloat16*)qh);
    return cudaGetLastError();
}

size_t gate_attn_rows_smem(const GateAttn& at, bool f32, int* tile) { return attn_smem(at, 1, f32 ? 4 : 2, 32, tile); }

cudaError_t launch_gate_attn_rows(const GateAttn& at, const void* qh, int pos0, int n, void* out, int ld_out, bool f32, bool pdl, cudaStream_t s) {
    int tile;
    const bool four = attn_pairs(at) <= 8 && attn_smem(at, 4, f32 ? 4 : 2, 32, &tile) > 0;
    if (f32) return four ? attn_rows_for<float, 4>(at, qh, pos0, n, out, ld_out, pdl, s) : attn_rows_for<float, 1>(at, qh, pos0, n, out, ld_out, pdl, s);
    return four ? attn_rows_for<__nv_bfloat16, 4>(at, qh, pos0, n, out, ld_out, pdl, s)
                : attn_rows_for<__nv_bfloat16, 1>(at, qh, pos0, n, out, ld_out, pdl, s);
}

cudaError_t launch_post_rows(float* x, const float* z0, const float* z1, const float* w0, const float* w1, const float* post_w, float eps,
                             int n, int width, void* act, int ld_act, bool f32, bool pdl, cudaStream_t s) {
    if ((width & 3) == 0 && width <= 4096) {
        auto quads = [&](auto* o) {
            using AT = std::remove_pointer_t<decltype(o)>;
            if (width <= 1024) launch_pdl(post_quads_kernel<AT, 1>, n, 256, 0, pdl, s, x, z0, z1, w0, w1, post_w, eps, width, o, ld_act);
            else if (width <= 2048) launch_pdl(post_quads_kernel<AT, 2>, n, 256, 0, pdl, s, x, z0, z1, w0, w1, post_w, eps, width, o, ld_act);
            else launch_pdl(post_quads_kernel<AT, 4>, n, 256, 0, pdl, s, x, z0, z1, w0, w1, post_w, eps, width, o, ld_act);
            return cudaGetLastError();
        };
        return f32 ? quads((float*)act) : quads((__nv_bfloat16*)act);
    }
    const size_t smem = (size_t)width * sizeof(float);
    if (f32) launch_pdl(post_rows_kernel<float>, n, 256, smem, pdl, s, x, z0, z1, w0, w1, post_w, eps, width, (float*)act, ld_act);
    else launch_pdl(post_rows_kernel<__nv_bfloat16>, n, 256, smem, pdl, s, x, z0, z1, w0, w1, post_w, eps, width, (__nv_bfloat16*)act, ld_act);
    return cudaGetLastError();
}

cudaError_t launch_last_norm_rows(const float* x, const int* rows, const float* w, int kind, float eps, int n, int width, void* act,
                                  int ld_act, bool f32, bool pdl, cudaStream_t s) {
    if (f32) launch_pdl(last_norm_rows_kernel<float>, n, 256, 0, pdl, s, x, rows, w, kind, eps, width, (float*)act, ld_act);
    else launch_pdl(last_norm_rows_kernel<__nv_bfloat16>, n, 256, 0, pdl, s, x, rows, w, kind, eps, width, (__nv_bfloat16*)act, ld_act);
    return cudaGetLastError();
}

cudaError_t launch_prenorm_rows(const PrenormRows& a, bool f32, bool pdl, cudaStream_t s) {
    const size_t smem = (size_t)a.width * sizeof(float);
    const bool quads = a.width % 4 == 0;
    if (f32 && quads) launch_pdl(prenorm_rows_kernel<float, 4>, a.n, 256, smem, pdl, s, a);
    else if (f32) launch_pdl(prenorm_rows_kernel<float, 1>, a.n, 256, smem, pdl, s, a);
    else if (quads) launch_pdl(prenorm_rows_kernel<__nv_bfloat16, 4>, a.n, 256, smem, pdl, s, a);
    else launch_pdl(prenorm_rows_kernel<__nv_bfloat16, 1>, a.n, 256, smem, pdl, s, a);
    return cudaGetLastError();
}

template <typename AT>
static cudaError_t head_norm_for(int heads, int vdim, float eps, const float* norm, const float* gate, int ldg, int gate_kind, int n, const float* o,
                                 AT* act, int ld_act, bool pdl, cudaStream_t s) {
    const bool quads = vdim % 4 == 0 && vdim <= 128 && ldg % 4 == 0 && (reinterpret_cast<uintptr_t>(gate) & 15) == 0;
    int lanes = 1;
    while (lanes * 4 < vdim) lanes *= 2;
    if (quads)
        launch_pdl(head_norm_quads_kernel<AT>, (int)(((long long)n * heads * lanes + 255) / 256), 256, 0, pdl, s, heads, vdim, lanes, eps, norm, gate, ldg, gate_kind, n, o, act, ld_act);
    else
        launch_pdl(head_norm_rows_kernel<AT>, (n * heads + 7) / 8, 256, 0, pdl, s, heads, vdim, eps, norm, gate, ldg, gate_kind, n, o, act, ld_act);
    return cudaGetLastError();
}

cudaError_t launch_head_norm_rows(int heads, int vdim, float eps, const float* norm, const float* gate, int ldg, int gate_kind, int n,
                                  const float* o, void* act, int ld_act, bool f32, bool pdl, cudaStream_t s) {
    return f32 ? head_norm_for(heads, vdim, eps, norm, gate, ldg, gate_kind, n, o, (float*)act, ld_act, pdl, s)
               : head_norm_for(heads, vdim, eps, norm, gate, ldg, gate_kind, n, o, (__nv_bfloat16*)act, ld_act, pdl, s);
}

cudaError_t launch_mem_rows(const MatMem& mem, const ProjCols& c, const float* proj, int ldp, int pos0, int n, const MemRows& w, void* act,
                            int ld_act, bool f32, bool pdl, cudaStream_t s) {
    const int chunks = (n + kMemChunk - 1) / kMemChunk, dt = (mem.dim + 63) / 64, vt = (mem.vdim + 63) / 64;
    launch_pdl(mem_gates_kernel, mem.heads, kGateWarps * 32, 0, pdl, s, mem, c.mi, c.mf, proj, ldp, pos0, n, w);
    launch_pdl(mem_chunk_kernel, dim3(chunks, mem.heads, dt * vt), 256, 0, pdl, s, mem, c.mk, c.mv, proj, ldp, n, vt, w);
    const size_t elems = (size_t)mem.heads * mem.dim * (mem.vdim + 1);
    launch_pdl(mem_scan_kernel, (unsigned)((elems + 255) / 256), 256, 0, pdl, s, mem, pos0, n, chunks, w);
    launch_pdl(mem_out_kernel, dim3(chunks, mem.heads, vt), 256, 0, pdl, s, mem, c.mq, c.mk, c.mv, proj, ldp, n, w);
    return launch_head_norm_rows(mem.heads, mem.vdim, mem.eps, mem.norm, proj + c.mg, ldp, GATE_SIGMOID, n, w.o, act, ld_act, f32, pdl, s);
}

}  // namespace mg
