// Prompts of the fixed seven-matrix decode block in batches of tokens: workspace and launches.  Included by engine.cu.
#pragma once

namespace {

// Fewer tokens than this go through the decode path one by one.  Measured on B200, batched against one by one: 4 tokens 452
// against 624 us (six layers of 0.5B widths), 638 against 776 us (six of 1.1B), 295 against 1052 us (two of 7B);
// 3 tokens would gain nothing on the narrow ones, whose batches of up to 32 tokens cost what their launches cost.
constexpr int kPromptMin = 4;
// 512 tokens: 2.2 ms for six layers of 1.1B widths (101 ms one by one), 1.8 ms for two of 7B (134 ms).
constexpr int kPromptBatch = 512;

// Places of the workspace's buffers from `block` on (NULL: none is set); returns its size.
size_t dense_prompt_carve(const mg_engine* e, DensePrompt& p, uint8_t* block) {
    const mg_config& c = e->cfg;
    const size_t cap = std::min(kPromptBatch, (c.max_seq + 63) & ~63), widest = std::max(2 * c.ffn_dim, c.dim + 2 * c.kv_dim);
    size_t at = 0;
    auto carve = [&](auto** b, size_t count) {
        if (block) *b = reinterpret_cast<std::remove_reference_t<decltype(*b)>>(block + at);
        at += (count * sizeof(**b) + 255) & ~(size_t)255;
    };
    carve(&p.tokens, e->out_cap); carve(&p.x, cap * c.dim); carve(&p.q, cap * c.dim);
    // a product is cut along K only while its tiles of 128 x 64 leave SMs idle
    carve(&p.sums, std::max(cap * widest, (size_t)e->num_sms * 128 * 64));
    carve(&p.act, 3 * cap * c.dim); carve(&p.mid, 3 * cap * c.ffn_dim); carve(&p.status, 1);
    return at;
}

void dense_prompt_free(mg_engine* e) {
    if (e->prompt.block) ARENA_FREE(e, e->prompt.block);
    e->dev_bytes -= e->prompt.bytes;
    e->prompt = DensePrompt{};
}

// The workspace, for engines that batch prompts: one GPU and every layer.  Made with the engine, and looked at again when it is built
// and knows its share of the model: one that turned out to be a stage or a tensor-parallel rank gives it back to its arena. Where
// there is no memory for it, prompts are fed token by token.  (An allocation of its own, beside the arena, moves the words that the persistent
// kernel's CTAs exchange: steps took 0.3 to 0.8 % longer.)
int dense_prompt_build(mg_engine* e) {
    DensePrompt& p = e->prompt;
    const mg_config& c = e->cfg;
    const bool wanted = c.dim <= kPromptMaxWidth && e->sh.size == 1 && e->own_ls == 0 && e->own_le == c.n_layers;
    if (wanted == (p.cap > 0)) return MG_OK;
    dense_prompt_free(e);
    if (!wanted) return MG_OK;
    const size_t bytes = dense_prompt_carve(e, p, nullptr);
    p.block = static_cast<uint8_t*>(e->arena.alloc(bytes));
    if (!p.block) return MG_OK;
    p.bytes = bytes;
    e->dev_bytes += bytes;
    dense_prompt_carve(e, p, p.block);
    const int cap = std::min(kPromptBatch, (c.max_seq + 63) & ~63);
    MG_CUDA(e, cudaMemset(p.status, 0, 4));
    for (int i = 0; i < 2; i++)
        if (!make_tile_map(&p.act_map[i], p.act, c.dim, cap, 3, c.dim, (long long)cap * c.dim, i ? 32 : 64) ||
            !make_tile_map(&p.mid_map[i], p.mid, c.ffn_dim, cap, 3, c.ffn_dim, (long long)cap * c.ffn_dim, i ? 32 : 64))
            return fail(e, MG_ERR_CUDA, "prompt: tensor maps cannot be encoded");
    p.cap = cap;
    return MG_OK;
}

bool dense_prompt_takes(const mg_engine* e, int n) { return e->prompt.cap && n >= kPromptMin; }

// x W^T for up to three matrices on one input, into p.sums.
int dense_prompt_gemm(mg_engine* e, const CUtensorMap maps[2], int K, int n, const int* slots, int n_mats, PieceSums* out) {
    DensePrompt& p = e->prompt;
    PromptGemm g{};
    const int small = n <= 32;
    g.x = maps[small];
    g.n_tile = small ? 32 : 64;
    g.fmt = e->cfg.layer_fmt; g.K = K; g.tokens = n;
    int tiles = 0, cols = 0;
    for (int m = 0; m < 3; m++) {
        if (m < n_mats) {
            const DevMatrix& w = e->mats[slots[m]];
            g.w[m] = w.view(); g.rows[m] = w.rows; g.col[m] = cols;
            tiles += (w.rows + 127) / 128;
            cols += w.rows;
        }
        g.tile_end[m] = tiles;
    }
    const int steps = (K + 63) / 64, ctas = tiles * ((n + g.n_tile - 1) / g.n_tile);
    const int cut = std::max(1, std::min(e->num_sms / ctas, steps / 3));
    g.steps = (steps + cut - 1) / cut;
    g.pieces = (steps + g.steps - 1) / g.steps;
    g.out = p.sums; g.ld = cols; g.stride = (long long)n * cols; g.status = p.status;
    MG_CUDA(e, dense_kernels()->prompt_gemm(g, e->stream));
    *out = PieceSums{p.sums, g.pieces, cols, g.stride};
    return MG_OK;
}

// Caches of every layer for tokens at positions pos .. pos + n - 1.  The last layer's output feeds nothing but the
// token's own logits, which are not asked for here: of it only keys and values are formed.
int dense_prompt(mg_engine* e, const int* tokens, int n, int pos) {
    DensePrompt& p = e->prompt;
    const mg_config& c = e->cfg;
    const DenseKernels* k = dense_kernels();
    const int L = c.n_layers;
    cudaStream_t s = e->stream;
    MG_CUDA(e, cudaStreamSynchronize(s));
    p.ran = true;
    for (int i = 0; i < n; i++) e->pin_i[8 + i] = tokens[i];
    MG_CUDA(e, cudaMemcpyAsync(p.tokens, e->pin_i + 8, (size_t)n * 4, cudaMemcpyHostToDevice, s));
    const SplitRows act{p.act, (long long)p.cap * c.dim, c.dim}, mid{p.mid, (long long)p.cap * c.ffn_dim, c.ffn_dim};
    for (int at = 0; at < n; at += p.cap) {
        const int m = std::min(p.cap, n - at);
        PieceSums sums{};
        int rc;
        for (int l = 0; l < L; l++) {
            const int b = l * 12;
            const bool last = l == L - 1;
            const size_t kvoff = (size_t)l * c.max_seq * c.kv_dim;
            PromptNorm norm{};
            norm.x = p.x; norm.eps = c.rms_eps; norm.out = act;
            norm.w = e->vecs[b];
            if (l == 0) {
                norm.tokens = p.tokens + at;
                norm.embed = e->mats[L * 12 + 1].view();
                norm.embed_fmt = c.head_fmt;
            } else {
                norm.add = sums;
            }
            MG_CUDA(e, k->prompt_norm(norm, m, s));
            const int qkv[3] = {b + 1, b + 2, b + 3}, wo = b + 7, gu[2] = {b + 9, b + 10}, down = b + 11;
            if ((rc = dense_prompt_gemm(e, p.act_map, c.dim, m, qkv + last, 3 - last, &sums))) return rc;
            PromptRope rope{};
            rope.qkv = sums;
            for (int i = 0; i < 3; i++) rope.bias[i] = e->vecs[b + 4 + i];
            rope.cos_tab = e->cos_tab; rope.sin_tab = e->sin_tab;
            rope.q_dim = c.dim; rope.kv_dim = c.kv_dim; rope.head_dim = c.head_dim; rope.pos0 = pos + at;
            rope.first = last ? c.dim : 0;
            rope.q = p.q; rope.kc = e->kc + kvoff; rope.vc = e->vc + kvoff;
            MG_CUDA(e, k->prompt_rope(rope, m, s));
            e->launches += 3;
            if (last) break;
            PromptAttn attn{p.q, rope.kc, rope.vc, c.n_heads, c.n_kv_heads, c.kv_dim, pos + at, m, act};
            MG_CUDA(e, k->prompt_attn(attn, c.head_dim, s));
            if ((rc = dense_prompt_gemm(e, p.act_map, c.dim, m, &wo, 1, &sums))) return rc;
            norm.tokens = nullptr;
            norm.add = sums;
            norm.w = e->vecs[b + 8];
            MG_CUDA(e, k->prompt_norm(norm, m, s));
            if ((rc = dense_prompt_gemm(e, p.act_map, c.dim, m, gu, 2, &sums))) return rc;
            MG_CUDA(e, k->prompt_swiglu(sums, mid, m, s));
            if ((rc = dense_prompt_gemm(e, p.mid_map, c.ffn_dim, m, &down, 1, &sums))) return rc;
            e->launches += 6;
        }
    }
    return MG_OK;
}

}  // namespace
