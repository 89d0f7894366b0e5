// A layer's launches in one call, for steps of few tokens: their kernels take less time than the host takes to launch them one binding after
// the other.  A step of eight tokens, 2,304 to 4,096 tokens into their requests, through an attention layer of width 2048 keeps the GPU busy for 33 us
// and took 55 with a call, an allocation and a set of checks per kernel; 37 so.  A token through a feed-forward of width 1024: 9.2 us of
// kernels, 15.6 before, 11.9 so.  Nothing is kept between calls: the intermediate results lie in `work`, which the caller allocates
// for the call.  The kernels and their arguments are those of the calls one by one.
#include "common.cuh"

extern "C" {
int lb_gemm_skinny(const void* x, const void* w, void* out, int tokens, int k, int n, int epilogue, int activation, void* state, const float* conv_weight, const float* conv_bias,
                   const int* token_segment, const int* segment_start, const int* segment_length, const int* segment_slot, int segments, int taps, int num_slots, int prefetch,
                   int* status, cudaStream_t stream, float limit, const float* bias, int x_stride);
int lb_qk_norm_rope_write(const void* qkv, void* q_out, void* k_pages, void* v_pages, const float* q_weight, const float* k_weight, float eps, float scale_offset,
                          const float* inv_freq, int rotary_dim, const int* positions, const int* token_segment, const int* block_table, int tokens, int num_heads,
                          int num_groups, int head_dim, int page_size, int num_pages, int max_blocks, int write_kv, int dtype, int* status, cudaStream_t stream,
                          int value_dim, const float* bias, float* row_inv, float turn_scale, int row_stride, int value_groups, float temperature, int temperature_every, int requests);
int lb_attention_decode(const void* q, const void* k_pages, const void* v_pages, void* out, float* scratch, const int* positions, const int* token_segment,
                        const int* block_table, const int* token_list, int tokens, int num_heads, int num_groups, int head_dim, int page_size, int num_pages, int max_blocks,
                        float scale, int window, int splits, int blocks_per_split, int fresh_keys, int* status, cudaStream_t stream, int keep_first, int value_dim,
                        int value_groups, int two_maps, int out_float);
}

namespace lb {

static int skinny_product(const void* x, const void* w, void* out, int tokens, int k, int n, int epilogue, int activation, float limit, cudaStream_t stream) {
    return lb_gemm_skinny(x, w, out, tokens, k, n, epilogue, activation, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0, 0, 1, nullptr, stream, limit, nullptr, k);
}

// What lb_gemm_skinny refuses, asked before a step's first launch: a step runs as a whole or not at all.
static bool skinny_takes(const void* x, const void* w, int tokens, int k, int n) {
    return tokens >= 1 && tokens <= 16 && k >= 32 && k % 32 == 0 && n >= 8 && n % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

constexpr int kSkinnyIdentity = 2;   // the activation's code
constexpr int kSkinnyGated = 3;      // the epilogue's

}  // namespace lb

extern "C" {

// out [tokens, out_width] = (up * act(gate)) @ down.T for [up ; gate] = x @ up_gate.T; epilogue 0 stores bfloat16, 2 adds to a 32-bit `out`.
// work: tokens * hidden bfloat16 values.  Returns 0, a CUDA error code or -2, with nothing launched, for sizes or an alignment the products do not take.
int lb_gated_mlp_step(const void* x, const void* up_gate, const void* down, void* out, void* work, long long work_bytes, int tokens, int width, int hidden, int out_width,
                      int activation, float limit, int epilogue, cudaStream_t stream) {
    if (work_bytes < static_cast<long long>(tokens) * hidden * 2 || (epilogue != 0 && epilogue != 2) || !lb::skinny_takes(x, up_gate, tokens, width, hidden) ||
        !lb::skinny_takes(work, down, tokens, hidden, out_width))
        return -2;
    const int code = lb::skinny_product(x, up_gate, work, tokens, width, hidden, lb::kSkinnyGated, activation, limit, stream);
    return code != 0 ? code : lb::skinny_product(work, down, out, tokens, hidden, out_width, epilogue, lb::kSkinnyIdentity, 0.0f, stream);
}

// An attention layer whose tokens all attend alone: x @ qkv_weight.T, the rewrite of q, k and v, the split-key attention (with the merge of its
// splits) and the out-projection.  epilogue as above; work: the product's rows, the queries, the heads' outputs (bfloat16, each from a multiple
// of 256 bytes on), then the attention's scratch (tokens * heads * splits * (head_dim + 2) floats).  Returns -2, with nothing launched, for
// what one of the four would refuse.
int lb_attention_step(const void* x, const void* qkv_weight, const void* out_weight, void* out, void* work, long long work_bytes, int tokens, int width, int qkv_width, int out_width,
                      int epilogue, void* k_pages, void* v_pages, const float* q_norm, const float* k_norm, float eps, float scale_offset, const float* inv_freq, int rotary_dim,
                      const int* positions, const int* token_segment, const int* block_table, int num_heads, int num_groups, int head_dim, int page_size, int num_pages,
                      int max_blocks, int write_kv, float turn_scale, float temperature, int temperature_every, float scale, int window, int keep_first, int splits,
                      int blocks_per_split, int fresh_keys, int* status, cudaStream_t stream) {
    if (num_groups < 1 || num_heads % num_groups != 0 || head_dim < 16 || head_dim > 128 || head_dim % 16 != 0 || page_size % 16 != 0 || rotary_dim < 0 || rotary_dim > head_dim ||
        rotary_dim % 2 != 0 || temperature_every < 0 || splits < 1 || blocks_per_split < 1 || fresh_keys < -1 || keep_first < 0 || !(scale > 0.0f) ||
        (epilogue != 0 && epilogue != 2) || qkv_width < num_heads * head_dim + (write_kv ? 2 * num_groups * head_dim : 0) ||
        !lb::skinny_takes(x, qkv_weight, tokens, width, qkv_width) || !lb::skinny_takes(work, out_weight, tokens, num_heads * head_dim, out_width))
        return -2;
    auto rounded = [](long long bytes) { return (bytes + 255) / 256 * 256; };
    const int heads_width = num_heads * head_dim;
    const long long queries_at = rounded(2LL * tokens * qkv_width), mixed_at = queries_at + rounded(2LL * tokens * heads_width), scratch_at = mixed_at + rounded(2LL * tokens * heads_width);
    if (work_bytes < scratch_at + 4LL * tokens * num_heads * splits * (head_dim + 2)) return -2;
    char* memory = static_cast<char*>(work);
    void *queries = memory + queries_at, *mixed = memory + mixed_at;
    int code = lb::skinny_product(x, qkv_weight, work, tokens, width, qkv_width, 0, lb::kSkinnyIdentity, 0.0f, stream);
    if (code != 0) return code;
    code = lb_qk_norm_rope_write(work, queries, k_pages, v_pages, q_norm, k_norm, eps, scale_offset, inv_freq, rotary_dim, positions, token_segment, block_table, tokens, num_heads,
                                 num_groups, head_dim, page_size, num_pages, max_blocks, write_kv, lb::kBFloat16, status, stream, head_dim, nullptr, nullptr, turn_scale, qkv_width,
                                 num_groups, temperature, temperature_every, tokens);
    if (code != 0) return code;
    code = lb_attention_decode(queries, k_pages, v_pages, mixed, reinterpret_cast<float*>(memory + scratch_at), positions, token_segment, block_table, nullptr, tokens, num_heads,
                               num_groups, head_dim, page_size, num_pages, max_blocks, scale, window, splits, blocks_per_split, fresh_keys, status, stream, keep_first, head_dim,
                               num_groups, 0, 0);
    if (code != 0) return code;
    return lb::skinny_product(mixed, out_weight, out, tokens, heads_width, out_width, epilogue, lb::kSkinnyIdentity, 0.0f, stream);
}

}  // extern "C"
