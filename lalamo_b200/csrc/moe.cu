// Routed feed-forward: a router that scores experts (sigmoid or softmax), restricts the choice to the best
// groups of neighbouring experts, and picks the `top` largest; gated experts evaluated per (token, chosen
// expert) with the expert's weights streamed once per pair; and the weighted sum of the experts' outputs.
// Router, scores and the weighted sum are 32-bit.
#include "common.cuh"

namespace lb {

// The lane-wise best (largest value, lowest index among equals) over a warp; every lane gets it.
__device__ __forceinline__ void warp_argmax(float& value, int& index) {
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        const float other_value = __shfl_xor_sync(0xffffffffu, value, offset);
        const int other_index = __shfl_xor_sync(0xffffffffu, index, offset);
        if (other_value > value || (other_value == value && other_index < index)) {
            value = other_value;
            index = other_index;
        }
    }
}

// A block takes TT tokens: its warps share out the experts' logits (EPW experts at a time, for all of the block's tokens, so that a
// router row is loaded once for TT tokens), then the tokens.  Every lane adds the same products in the same order whatever TT
// and EPW are, so a token's logits do not depend on the step it is in.
//   z[e] = x . router[e] (+ bias[e])  (32-bit);   s[e] = sigmoid(z[e])   (score_kind 0),  softmax(z)[e]   (score_kind 1)  or  z[e]  (score_kind 2)
//   experts form `group_count` equal groups of neighbours; a group's score is the sum of its two largest s (of its
//   only one, in groups of one), or with `group_top` 1 its largest s; experts outside the best `group_keep` groups cannot be chosen;
//   chosen[t, :] = the `top` eligible experts of largest s, in that order; weights[t, :] = their s (divided by their
//   sum if `renormalize` is 1; the softmax over just the chosen s if it is 2), times `weight_scale`.
//   `choice_bias` (may be null): experts (and groups) are ranked by s[e] + choice_bias[e]; the weights stay the s themselves.
//   `extra` further rows of `router` after the experts' are gates of something every token runs: extra_out[t, x] =
//   sigmoid(x_t . router[experts + x]), 32-bit like the scores.
// Shared memory per token: s[experts], candidates[experts], group score[group_count], and the token's row in 32-bit where it is staged.
// Few tokens are bound by the latency of the router's loads (hence 16 warps of one expert each, all of a row's loads on their way at
// once), many by the loads themselves (hence 8 tokens a load).  Measured, 16 experts and rows of
// 2,048: 8 tokens 9.6 us (20.6 with four warps a token, four experts each), 2,048 tokens 20.7 us (48.5 with one token a warp).
template <typename T, int TT, int EPW>
__global__ void __launch_bounds__(TT == 1 ? 512 : 256)
moe_route_kernel(const T* __restrict__ x, const float* __restrict__ router, int* __restrict__ chosen, float* __restrict__ weights,
                 int tokens, int width, int experts, int top, int group_count, int group_keep, int score_kind, int renormalize,
                 float weight_scale, int row_floats, int group_floats, const float* __restrict__ bias,
                 const float* __restrict__ choice_bias, int extra, float* __restrict__ extra_out, int group_top) {
    extern __shared__ __align__(16) float shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int token0 = blockIdx.x * TT, tokens_here = min(TT, tokens - token0);
    const int logits = experts + extra;   // rows of the router
    const int pitch = experts + logits + group_floats;   // floats of a token's scratch, a multiple of 4
    float* rows_s = shared + TT * pitch;   // row_floats = width (a multiple of 4) a token if the rows are staged, else 0
    if (row_floats > 0) {
        // the tokens' rows once into shared memory (32-bit, four elements a thread and turn), then EPW experts' rows at a time, 16
        // bytes a lane and turn
        const T* rows = x + static_cast<size_t>(token0) * width;
#pragma unroll 8
        for (int d = 4 * threadIdx.x; d < tokens_here * width; d += 4 * blockDim.x) {
            if constexpr (sizeof(T) == 4) {
                *reinterpret_cast<float4*>(rows_s + d) = *reinterpret_cast<const float4*>(rows + d);
            } else {
                const uint2 raw = *reinterpret_cast<const uint2*>(rows + d);
                const float2 low = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(raw.x)), high = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(raw.y));
                *reinterpret_cast<float4*>(rows_s + d) = make_float4(low.x, low.y, high.x, high.y);
            }
        }
        __syncthreads();
        for (int e0 = EPW * warp; e0 < logits; e0 += EPW * warps) {
            float dots[TT][EPW];
#pragma unroll
            for (int t = 0; t < TT; ++t)
#pragma unroll
                for (int r = 0; r < EPW; ++r) dots[t][r] = 0.0f;
#pragma unroll (16 / EPW)
            for (int c = 4 * lane; c < width; c += 128) {   // sixteen loads of the router's rows on their way at a time
                float4 w[EPW];
#pragma unroll
                for (int r = 0; r < EPW; ++r) w[r] = *reinterpret_cast<const float4*>(router + static_cast<size_t>(e0 + r < logits ? e0 + r : e0) * width + c);
#pragma unroll
                for (int t = 0; t < TT; ++t) {
                    const float4 xv = *reinterpret_cast<const float4*>(rows_s + (t < tokens_here ? t : 0) * row_floats + c);
#pragma unroll
                    for (int r = 0; r < EPW; ++r) {
                        dots[t][r] += xv.x * w[r].x;
                        dots[t][r] += xv.y * w[r].y;
                        dots[t][r] += xv.z * w[r].z;
                        dots[t][r] += xv.w * w[r].w;
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < TT; ++t) {
#pragma unroll
                for (int r = 0; r < EPW; ++r) {
                    const float dot = warp_sum(dots[t][r]);
                    if (lane == 0 && e0 + r < logits) shared[t * pitch + e0 + r] = dot;
                }
            }
        }
    } else {
        for (int t = 0; t < tokens_here; ++t) {
            const T* row = x + static_cast<size_t>(token0 + t) * width;
            for (int e = warp; e < logits; e += warps) {
                const float* w = router + static_cast<size_t>(e) * width;
                float dot = 0.0f;
                for (int d = lane; d < width; d += 32) dot += to_float(row[d]) * w[d];
                dot = warp_sum(dot);
                if (lane == 0) shared[t * pitch + e] = dot;
            }
        }
    }
    __syncthreads();
    for (int t = warp; t < tokens_here; t += warps) {
        const int token = token0 + t;
        float* scores = shared + t * pitch;
        float* candidates = scores + logits;
        float* group_score = candidates + experts;   // group_floats >= group_count of them
        for (int x = lane; x < extra; x += 32) extra_out[static_cast<size_t>(token) * extra + x] = 1.0f / (1.0f + expf(-scores[experts + x]));
        if (bias != nullptr) {
            for (int e = lane; e < experts; e += 32) scores[e] += bias[e];
            __syncwarp();
        }
        if (score_kind == 2) {
            // the logits themselves rank the experts
        } else if (score_kind == 1) {
            float largest = -INFINITY;
            for (int e = lane; e < experts; e += 32) largest = fmaxf(largest, scores[e]);
            largest = warp_max(largest);
            float total = 0.0f;
            for (int e = lane; e < experts; e += 32) total += expf(scores[e] - largest);
            total = warp_sum(total);
            for (int e = lane; e < experts; e += 32) scores[e] = expf(scores[e] - largest) / total;
        } else {
            for (int e = lane; e < experts; e += 32) scores[e] = 1.0f / (1.0f + expf(-scores[e]));
        }
        __syncwarp();
        const int members = experts / group_count;
        for (int group = lane; group < group_count; group += 32) {
            float first = -INFINITY, second = -INFINITY;
            for (int m = 0; m < members; ++m) {
                const float s = scores[group * members + m] + (choice_bias != nullptr ? choice_bias[group * members + m] : 0.0f);
                if (s > first) {
                    second = first;
                    first = s;
                } else if (s > second) {
                    second = s;
                }
            }
            group_score[group] = members >= 2 && group_top != 1 ? first + second : first;
        }
        for (int e = lane; e < experts; e += 32) candidates[e] = -INFINITY;
        __syncwarp();
        for (int round = 0; round < group_keep; ++round) {
            float best = -INFINITY;
            int best_group = 0x7fffffff;
            for (int group = lane; group < group_count; group += 32) {
                const float s = group_score[group];
                if (s > best) {   // ascending scan: the lowest index among equals stays
                    best = s;
                    best_group = group;
                }
            }
            warp_argmax(best, best_group);
            if (best_group == 0x7fffffff) break;
            for (int m = lane; m < members; m += 32)
                candidates[best_group * members + m] = scores[best_group * members + m] + (choice_bias != nullptr ? choice_bias[best_group * members + m] : 0.0f);
            if (lane == 0) group_score[best_group] = -INFINITY;
            __syncwarp();
        }
        float total = 0.0f;
        for (int round = 0; round < top; ++round) {
            float best = -INFINITY;
            int best_expert = 0x7fffffff;
            for (int e = lane; e < experts; e += 32) {
                const float s = candidates[e];
                if (s > best) {
                    best = s;
                    best_expert = e;
                }
            }
            warp_argmax(best, best_expert);
            if (best_expert == 0x7fffffff) best_expert = 0, best = 0.0f;   // fewer eligible experts than `top`: a weight of zero
            else if (choice_bias != nullptr) best = scores[best_expert];   // ranked with the bias, weighed without it
            total += best;
            if (lane == 0) {
                chosen[static_cast<size_t>(token) * top + round] = best_expert;
                weights[static_cast<size_t>(token) * top + round] = best;
                if (best_expert < experts) candidates[best_expert] = -INFINITY;
            }
            __syncwarp();
        }
        if (lane == 0 && renormalize == 2) {
            // the softmax over the chosen scores only (the first chosen is the largest)
            float* mine = weights + static_cast<size_t>(token) * top;
            const float largest = mine[0];
            float sum = 0.0f;
            for (int round = 0; round < top; ++round) {
                mine[round] = expf(mine[round] - largest);
                sum += mine[round];
            }
            for (int round = 0; round < top; ++round) mine[round] = mine[round] / sum * weight_scale;
        } else if (lane == 0) {
            const float factor = (renormalize && total > 0.0f ? 1.0f / total : 1.0f) * weight_scale;
            if (factor != 1.0f)
                for (int round = 0; round < top; ++round) weights[static_cast<size_t>(token) * top + round] *= factor;
        }
    }
}

__device__ __forceinline__ float moe_activate(float v, int activation) {
    if (activation == 0) return v / (1.0f + expf(-v));                                   // silu
    if (activation == 1) return 0.5f * v * (1.0f + erff(v * 0.70710678118654752440f));    // gelu (exact)
    return v;
}

// Where a pair's weight multiplies its expert's input (expert(w x) instead of w expert(x)), the two sums are multiplied by it in 32-bit,
// which is the same since both are linear in the input: `pair_weight` of the kernels below (null: inputs as they are).

// The hidden value of a gated expert from its two 32-bit sums, as a value of T.
template <typename T>
__device__ __forceinline__ float moe_hidden(float gate, float up, int activation, float limit) {
    if (activation == kSigmoidLimit) return round_to<T>(sigmoid_limit_gate(gate, up, limit));
    return round_to<T>(round_to<T>(moe_activate(round_to<T>(gate), activation)) * round_to<T>(up));
}

// The hidden value of an expert without a gate, act(W_up x), from its 32-bit sum: activated in 32-bit, rounded once.
template <typename T>
__device__ __forceinline__ float moe_plain_hidden(float up, int activation) {
    return round_to<T>(moe_activate(up, activation));
}

// One block per (token, chosen expert) pair p (`gate` null: experts without a gate, hidden = act(W_up[e] x)): hidden = act(W_gate[e] x) * (W_up[e] x), rounded to T; out[p] = W_down[e] hidden
// in 32-bit.  A warp per output row, lanes along the row, sums in lane order then over the warp.
//   gate, up [experts, ff, width];  down [experts, width, ff];  out [pairs, width] (32-bit)
template <typename T>
__global__ void moe_expert_stream_kernel(const T* __restrict__ x, const T* __restrict__ gate, const T* __restrict__ up, const T* __restrict__ down,
                                         const int* __restrict__ chosen, float* __restrict__ out, int top, int width, int ff, int experts,
                                         int activation, float limit, const float* __restrict__ pair_weight) {
    extern __shared__ float shared[];
    float* x_s = shared;           // width
    float* hidden = shared + width;   // ff
    const int pair = blockIdx.x;
    const int token = pair / top;
    const int expert = chosen[pair];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    float* dst = out + static_cast<size_t>(pair) * width;
    if (expert < 0 || expert >= experts) {
        for (int d = threadIdx.x; d < width; d += blockDim.x) dst[d] = 0.0f;
        return;
    }
    for (int d = threadIdx.x; d < width; d += blockDim.x) x_s[d] = to_float(x[static_cast<size_t>(token) * width + d]);
    __syncthreads();
    const float factor = pair_weight != nullptr ? pair_weight[pair] : 1.0f;
    const T* up_rows = up + static_cast<size_t>(expert) * ff * width;
    const T* gate_rows = gate != nullptr ? gate + static_cast<size_t>(expert) * ff * width : up_rows;
    for (int f = warp; f < ff; f += warps) {
        const T* g_row = gate_rows + static_cast<size_t>(f) * width;
        const T* u_row = up_rows + static_cast<size_t>(f) * width;
        float g = 0.0f, u = 0.0f;
        for (int d = lane; d < width; d += 32) {
            if (gate != nullptr) g += x_s[d] * to_float(g_row[d]);
            u += x_s[d] * to_float(u_row[d]);
        }
        g = warp_sum(g) * factor;
        u = warp_sum(u) * factor;
        if (lane == 0) hidden[f] = gate != nullptr ? moe_hidden<T>(g, u, activation, limit) : moe_plain_hidden<T>(u, activation);
    }
    __syncthreads();
    const T* down_rows = down + static_cast<size_t>(expert) * width * ff;
    for (int r = warp; r < width; r += warps) {
        const T* d_row = down_rows + static_cast<size_t>(r) * ff;
        float sum = 0.0f;
        for (int f = lane; f < ff; f += 32) sum += hidden[f] * to_float(d_row[f]);
        sum = warp_sum(sum);
        if (lane == 0) dst[r] = sum;
    }
}

// out[t, :] = T(sum_k weights[t, k] * expert_out[t * top + k, :]), added in the order of k (`weights` null: the plain sum).
template <typename T>
__global__ void moe_combine_kernel(const float* __restrict__ expert_out, const float* __restrict__ weights, const int* __restrict__ chosen, int experts,
                                   T* __restrict__ out, int top, int width) {
    const int token = blockIdx.x;
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float sum = 0.0f;
        for (int k = 0; k < top; ++k) {
            const int expert = chosen[static_cast<size_t>(token) * top + k];
            if (expert < 0 || expert >= experts) continue;   // no expert: nothing was computed for the pair
            sum += (weights != nullptr ? weights[static_cast<size_t>(token) * top + k] : 1.0f) * expert_out[(static_cast<size_t>(token) * top + k) * width + d];
        }
        out[static_cast<size_t>(token) * width + d] = from_float<T>(sum);
    }
}

// The same for widths that come in fours and up to eight experts a token, which stay in registers: four columns a thread and turn, the pairs' loads
// of a turn all on their way at once.  Bound by the pairs' rows: 2,048 tokens of four rows of 2,048 take 14.7 us (18.5 a column at a time), 8 tokens
// 3.3 (6.1).
constexpr int kCombineTop = 8;
template <typename T>
__global__ void __launch_bounds__(256)
moe_combine_wide_kernel(const float* __restrict__ expert_out, const float* __restrict__ weights, const int* __restrict__ chosen, int experts, T* __restrict__ out, int top,
                        int width) {
    wait_for_previous_kernel();
    allow_next_kernel();
    const int token = blockIdx.x;
    const size_t pair0 = static_cast<size_t>(token) * top;
    float weight[kCombineTop];
    bool real[kCombineTop];
#pragma unroll
    for (int k = 0; k < kCombineTop; ++k) {
        const int expert = k < top ? chosen[pair0 + k] : -1;
        real[k] = expert >= 0 && expert < experts;   // no expert: nothing was computed for the pair
        weight[k] = real[k] && weights != nullptr ? weights[pair0 + k] : 1.0f;
    }
    for (int d = 4 * threadIdx.x; d < width; d += 4 * blockDim.x) {
        float4 rows[kCombineTop];
#pragma unroll
        for (int k = 0; k < kCombineTop; ++k)
            if (real[k]) rows[k] = *reinterpret_cast<const float4*>(expert_out + (pair0 + k) * width + d);
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < kCombineTop; ++k) {
            if (real[k]) {
                sum.x += weight[k] * rows[k].x;
                sum.y += weight[k] * rows[k].y;
                sum.z += weight[k] * rows[k].z;
                sum.w += weight[k] * rows[k].w;
            }
        }
        T* destination = out + static_cast<size_t>(token) * width + d;
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(destination) = sum;
        } else {
            const __nv_bfloat162 low = __floats2bfloat162_rn(sum.x, sum.y), high = __floats2bfloat162_rn(sum.z, sum.w);
            *reinterpret_cast<uint2*>(destination) = make_uint2(*reinterpret_cast<const uint32_t*>(&low), *reinterpret_cast<const uint32_t*>(&high));
        }
    }
}

// residual[t, :] += sum_k weights[t, k] * expert_out[t * top + k, :] + every_gate[t] * every[t, :] on the 32-bit residual stream:
// the routed experts' weighted sum (in the order of k) and what every token runs besides (`every`, may be null; `every_gate`
// one 32-bit number per token, null: 1), added in 32-bit without a rounding in between.
template <typename T>
__global__ void moe_combine_add_kernel(const float* __restrict__ expert_out, const float* __restrict__ weights, const int* __restrict__ chosen, int experts,
                                       const T* __restrict__ every, const float* __restrict__ every_gate, int gate_stride, float* __restrict__ residual,
                                       int top, int width) {
    const int token = blockIdx.x;
    const float gate = every_gate != nullptr ? every_gate[static_cast<size_t>(token) * gate_stride] : 1.0f;
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float sum = 0.0f;
        for (int k = 0; k < top; ++k) {
            const int expert = chosen[static_cast<size_t>(token) * top + k];
            if (expert < 0 || expert >= experts) continue;
            sum += (weights != nullptr ? weights[static_cast<size_t>(token) * top + k] : 1.0f) * expert_out[(static_cast<size_t>(token) * top + k) * width + d];
        }
        if (every != nullptr) sum += gate * to_float(every[static_cast<size_t>(token) * width + d]);
        residual[static_cast<size_t>(token) * width + d] += sum;
    }
}

// ---------------------------------------------------------------- few tokens: 16-byte loads, many blocks
// The same two products with the rows of an expert's matrices shared out over blocks: grid (pairs, row slices),
// four warps, a warp takes eight rows, four at a time, a lane 16 bytes of each row per turn (so eight loads of a
// lane are on their way at once).  Needs rows of 16-byte multiples.
constexpr int kStreamRowsPerWarp = 8, kStreamWarps = 4, kStreamRowsPerBlock = kStreamRowsPerWarp * kStreamWarps;

template <typename T, int V>
__device__ __forceinline__ void load_vector(const T* address, float (&values)[V]) {
    if constexpr (sizeof(T) == 2) {
        const uint4 raw = *reinterpret_cast<const uint4*>(address);
        const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 two = __bfloat1622float2(pairs[i]);
            values[2 * i] = two.x;
            values[2 * i + 1] = two.y;
        }
    } else {
        const float4 raw = *reinterpret_cast<const float4*>(address);
        values[0] = raw.x, values[1] = raw.y, values[2] = raw.z, values[3] = raw.w;
    }
}

// sums[r] = x_s . rows[r], r < 4 (rows that do not exist are given as the first row and ignored by the caller)
template <typename T>
__device__ __forceinline__ void four_dots(const float* __restrict__ x_s, const T* const (&rows)[4], int length, int lane, float (&sums)[4]) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int r = 0; r < 4; ++r) sums[r] = 0.0f;
    for (int c = lane * V; c < length; c += 32 * V) {
        float w[4][V];
#pragma unroll
        for (int r = 0; r < 4; ++r) load_vector<T, V>(rows[r] + c, w[r]);
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const float xv = x_s[c + i];
#pragma unroll
            for (int r = 0; r < 4; ++r) sums[r] += xv * w[r][i];
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) sums[r] = warp_sum(sums[r]);
}

// hidden[pair, f] = T(act(gate[e][f] . x) * (up[e][f] . x)) for the block's slice of f (`gate` null: T(act(up[e][f] . x))).
template <typename T>
__global__ void __launch_bounds__(32 * kStreamWarps)
moe_gate_up_stream_kernel(const T* __restrict__ x, const T* __restrict__ gate, const T* __restrict__ up, const int* __restrict__ chosen,
                          T* __restrict__ hidden, int top, int width, int ff, int experts, int activation, float limit,
                          const float* __restrict__ pair_weight) {
    extern __shared__ float x_s[];   // width
    const int pair = blockIdx.x, token = pair / top, expert = chosen[pair];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.y * kStreamRowsPerBlock + warp * kStreamRowsPerWarp;
    if (expert < 0 || expert >= experts) {
        for (int f = first + lane; f < min(ff, first + kStreamRowsPerWarp); f += 32) hidden[static_cast<size_t>(pair) * ff + f] = from_float<T>(0.0f);
        return;
    }
    for (int d = threadIdx.x; d < width; d += blockDim.x) x_s[d] = to_float(x[static_cast<size_t>(token) * width + d]);
    __syncthreads();
    const float factor = pair_weight != nullptr ? pair_weight[pair] : 1.0f;
    const T* up_rows = up + static_cast<size_t>(expert) * ff * width;
    const T* gate_rows = gate != nullptr ? gate + static_cast<size_t>(expert) * ff * width : up_rows;
    for (int f0 = first; f0 < min(ff, first + kStreamRowsPerWarp); f0 += 4) {
        const T* g_rows[4];
        const T* u_rows[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int f = f0 + r < ff ? f0 + r : f0;
            g_rows[r] = gate_rows + static_cast<size_t>(f) * width;
            u_rows[r] = up_rows + static_cast<size_t>(f) * width;
        }
        float g[4] = {0.0f, 0.0f, 0.0f, 0.0f}, u[4];
        if (gate != nullptr) four_dots<T>(x_s, g_rows, width, lane, g);
        four_dots<T>(x_s, u_rows, width, lane, u);
        if (lane < 4 && f0 + lane < ff) {
            const float gv = (lane == 0 ? g[0] : lane == 1 ? g[1] : lane == 2 ? g[2] : g[3]) * factor;
            const float uv = (lane == 0 ? u[0] : lane == 1 ? u[1] : lane == 2 ? u[2] : u[3]) * factor;
            hidden[static_cast<size_t>(pair) * ff + f0 + lane] = from_float<T>(gate != nullptr ? moe_hidden<T>(gv, uv, activation, limit) : moe_plain_hidden<T>(uv, activation));
        }
    }
}

// out[pair, r] = down[e][r] . hidden[pair] for the block's slice of r (32-bit).
template <typename T>
__global__ void __launch_bounds__(32 * kStreamWarps)
moe_down_stream_kernel(const T* __restrict__ hidden, const T* __restrict__ down, const int* __restrict__ chosen, float* __restrict__ out, int width,
                       int ff, int experts) {
    extern __shared__ float h_s[];   // ff
    const int pair = blockIdx.x, expert = chosen[pair];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.y * kStreamRowsPerBlock + warp * kStreamRowsPerWarp;
    float* dst = out + static_cast<size_t>(pair) * width;
    if (expert < 0 || expert >= experts) {
        for (int r = first + lane; r < min(width, first + kStreamRowsPerWarp); r += 32) dst[r] = 0.0f;
        return;
    }
    for (int f = threadIdx.x; f < ff; f += blockDim.x) h_s[f] = to_float(hidden[static_cast<size_t>(pair) * ff + f]);
    __syncthreads();
    const T* down_rows = down + static_cast<size_t>(expert) * width * ff;
    for (int r0 = first; r0 < min(width, first + kStreamRowsPerWarp); r0 += 4) {
        const T* rows[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) rows[r] = down_rows + static_cast<size_t>(r0 + r < width ? r0 + r : r0) * ff;
        float sums[4];
        four_dots<T>(h_s, rows, ff, lane, sums);
        if (lane < 4 && r0 + lane < width) dst[r0 + lane] = lane == 0 ? sums[0] : lane == 1 ? sums[1] : lane == 2 ? sums[2] : sums[3];
    }
}

}  // namespace lb

extern "C" {

int lb_moe_route(const void* x, const float* router, int* chosen, float* weights, int tokens, int width, int experts, int top, int group_count,
                 int group_keep, int score_kind, int renormalize, float weight_scale, int dtype, cudaStream_t stream, const float* bias,
                 const float* choice_bias, int extra, float* extra_out, int group_top) {
    // `router` has experts + extra rows; extra_out [tokens, extra] (see the kernel).
    if (tokens == 0) return 0;
    if (experts < 1 || top < 1 || top > experts || group_count < 1 || experts % group_count != 0 || group_keep < 1 || group_keep > group_count) return -2;
    if (extra < 0 || (extra > 0 && extra_out == nullptr) || group_top < 1 || group_top > 2) return -2;
    // A token's scratch: scores, candidates, group scores (padded so that the staged row starts on 16 bytes), and the row.
    const int scratch = (2 * experts + extra + group_count + 3) / 4 * 4;
    if (4 * static_cast<size_t>(scratch) * sizeof(float) > 48 * 1024) return -2;
    int row_floats = width % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (dtype == lb::kBFloat16 ? 8 : 16) == 0 ? width : 0;   // rows that start on 16 bytes (8, in bfloat16) are staged and read 16 bytes a lane
    if (4 * static_cast<size_t>(scratch + row_floats) * sizeof(float) > 160 * 1024) row_floats = 0;   // by the sizes alone, not by the tokens (see the kernel)
    const int padded_groups = scratch - 2 * experts - extra;   // the kernel lays the three arrays out by these counts
    // Tokens a block: one while that leaves the multiprocessors no more than two blocks each, then 2, 4, 8 (four times as many fit).
    const int sms = lb::multiprocessor_count();
    int per_block = tokens <= 2 * sms ? 1 : tokens <= 4 * sms ? 2 : tokens <= 8 * sms ? 4 : 8;
    if (per_block == 8 && 8 * static_cast<size_t>(scratch + row_floats) * sizeof(float) > 160 * 1024) per_block = 4;
    const size_t shared = per_block * static_cast<size_t>(scratch + row_floats) * sizeof(float);
    LB_DISPATCH_DTYPE(dtype, {
        auto kernel = per_block == 1 ? lb::moe_route_kernel<T, 1, 1> : per_block == 2 ? lb::moe_route_kernel<T, 2, 2> : per_block == 4 ? lb::moe_route_kernel<T, 4, 2> : lb::moe_route_kernel<T, 8, 2>;
        if (shared > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
        kernel<<<(tokens + per_block - 1) / per_block, per_block == 1 ? 512 : 256, shared, stream>>>(
            static_cast<const T*>(x), router, chosen, weights, tokens, width, experts, top, group_count, group_keep, score_kind, renormalize, weight_scale,
            row_floats, padded_groups, bias, choice_bias, extra, extra_out, group_top);
    })
    return LB_LAUNCH_RESULT();
}

int lb_moe_expert_stream(const void* x, const void* gate, const void* up, const void* down, const int* chosen, float* out, int pairs, int top,
                         int width, int ff, int experts, int activation, int dtype, cudaStream_t stream, float limit, const float* pair_weight) {
    if (pairs == 0) return 0;
    const size_t shared = (static_cast<size_t>(width) + ff) * sizeof(float);
    if (shared > 200 * 1024) return -2;
    LB_DISPATCH_DTYPE(dtype, {
        auto kernel = lb::moe_expert_stream_kernel<T>;
        if (shared > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
        kernel<<<pairs, 256, shared, stream>>>(static_cast<const T*>(x), static_cast<const T*>(gate), static_cast<const T*>(up), static_cast<const T*>(down),
                                               chosen, out, top, width, ff, experts, activation, limit, pair_weight);
    })
    return LB_LAUNCH_RESULT();
}

int lb_moe_combine(const float* expert_out, const float* weights, const int* chosen, int experts, void* out, int tokens, int top, int width, int dtype,
                   cudaStream_t stream) {
    if (tokens == 0) return 0;
    if (width % 4 == 0 && top <= lb::kCombineTop && reinterpret_cast<uintptr_t>(expert_out) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0) {
        LB_DISPATCH_DTYPE(dtype, {
            return static_cast<int>(lb::launch_overlapped(lb::moe_combine_wide_kernel<T>, dim3(tokens), dim3(256), 0, stream, expert_out, weights, chosen, experts, static_cast<T*>(out), top,
                                                          width));
        })
    }
    LB_DISPATCH_DTYPE(dtype, {
        lb::moe_combine_kernel<T><<<tokens, 256, 0, stream>>>(expert_out, weights, chosen, experts, static_cast<T*>(out), top, width);
    })
    return LB_LAUNCH_RESULT();
}

int lb_moe_combine_add(const float* expert_out, const float* weights, const int* chosen, int experts, const void* every, const float* every_gate,
                       int gate_stride, float* residual, int tokens, int top, int width, int dtype, cudaStream_t stream) {
    if (tokens == 0) return 0;
    LB_DISPATCH_DTYPE(dtype, {
        lb::moe_combine_add_kernel<T><<<tokens, 256, 0, stream>>>(expert_out, weights, chosen, experts, static_cast<const T*>(every), every_gate, gate_stride,
                                                                   residual, top, width);
    })
    return LB_LAUNCH_RESULT();
}

// The two products of the few-token path: `hidden` [pairs, ff] in the activation type, `out` [pairs, width] in 32-bit.
// Rows of 16-byte multiples only (width and ff multiples of 8 for bfloat16, of 4 for float32): -2 otherwise.
int lb_moe_expert_stream_wide(const void* x, const void* gate, const void* up, const void* down, const int* chosen, void* hidden, float* out, int pairs,
                              int top, int width, int ff, int experts, int activation, int dtype, cudaStream_t stream, float limit, const float* pair_weight) {
    if (pairs == 0) return 0;
    const int vector = dtype == lb::kBFloat16 ? 8 : 4;
    if (width % vector != 0 || ff % vector != 0 || width * sizeof(float) > 160 * 1024 || ff * sizeof(float) > 160 * 1024) return -2;
    const dim3 up_grid(pairs, (ff + lb::kStreamRowsPerBlock - 1) / lb::kStreamRowsPerBlock), down_grid(pairs, (width + lb::kStreamRowsPerBlock - 1) / lb::kStreamRowsPerBlock);
    LB_DISPATCH_DTYPE(dtype, {
        auto first = lb::moe_gate_up_stream_kernel<T>;
        auto second = lb::moe_down_stream_kernel<T>;
        if (width * sizeof(float) > 48 * 1024) cudaFuncSetAttribute(first, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(width * sizeof(float)));
        if (ff * sizeof(float) > 48 * 1024) cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ff * sizeof(float)));
        first<<<up_grid, 32 * lb::kStreamWarps, width * sizeof(float), stream>>>(static_cast<const T*>(x), static_cast<const T*>(gate), static_cast<const T*>(up), chosen,
                                                                                static_cast<T*>(hidden), top, width, ff, experts, activation, limit,
                                                                                pair_weight);
        second<<<down_grid, 32 * lb::kStreamWarps, ff * sizeof(float), stream>>>(static_cast<const T*>(hidden), static_cast<const T*>(down), chosen, out, width, ff, experts);
    })
    return LB_LAUNCH_RESULT();
}

}  // extern "C"
