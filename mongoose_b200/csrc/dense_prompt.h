// Prompts of the fixed seven-matrix decode block in batches of tokens (dense_prompt.cu): what the
// engine's host code launches.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "decode_kernels.cuh"

namespace mg {

constexpr int kPromptMaxWidth = 28672;      // a row of the residual in shared memory

// fp32 rows [token][width] as three bf16 parts whose sum is the value: part p of token t starts at p * part + t * width.
struct SplitRows {
    __nv_bfloat16* p;
    long long part;
    int width;
};

// Sums of a product whose columns of K were cut into `n` pieces: piece s of token t starts at s * stride + t * ld.
struct PieceSums {
    const float* p;
    int n, ld;
    long long stride;
};

// out[token][col[m] + row] = sum over k of x[token][k] W_m[row][k], per piece of K (grid z).
struct PromptGemm {
    CUtensorMap x;              // [3 parts][tokens][K] in boxes of 64 columns x (64 or 32) tokens
    int n_tile;                 // tokens per tile: 64 or 32
    WeightView w[3];            // matrices that share the input; tiles tile_end[m-1] .. tile_end[m]-1 belong to matrix m
    int rows[3], col[3], tile_end[3];
    int fmt, K, tokens;
    int steps;                  // steps of 64 columns per piece
    int pieces;
    float* out;
    int ld;
    long long stride;
    int* status;
};

struct PromptNorm {             // x += sums (or x = embedding row); out = x / rms(x) * w
    float* x;
    PieceSums add;              // n == 0: none
    const int* tokens;          // not NULL: x = embedding row of tokens[t]
    WeightView embed;
    int embed_fmt;
    const float* w;
    float eps;
    SplitRows out;
};

struct PromptRope {             // bias, rotation, cache append
    PieceSums qkv;
    const float* bias[3];
    const float *cos_tab, *sin_tab;
    int q_dim, kv_dim, head_dim, pos0;
    int first;                  // first column present in the sums (q_dim: keys and values only)
    float* q;                   // [token][q_dim]
    __half *kc, *vc;            // this layer's cache
};

struct PromptAttn {
    const float* q;
    const __half *kc, *vc;
    int n_heads, n_kv_heads, kv_dim, pos0, tokens;
    SplitRows out;
};

cudaError_t prompt_kernel_attrs();        // once per device
cudaError_t launch_prompt_gemm(const PromptGemm& g, cudaStream_t s);
cudaError_t launch_prompt_norm(const PromptNorm& a, int tokens, cudaStream_t s);
cudaError_t launch_prompt_rope(const PromptRope& a, int tokens, cudaStream_t s);
cudaError_t launch_prompt_attn(const PromptAttn& a, int head_dim, cudaStream_t s);
cudaError_t launch_prompt_swiglu(const PieceSums& gu, const SplitRows& out, int tokens, cudaStream_t s);

}  // namespace mg
