// The gated delta rule with one decay per head and key channel, over ragged portions of requests:
//
//   S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
//
// with S a [key_dim, value_dim] matrix per request and head, kept in 32-bit in the request's state
// slot.  Four kernels: `prepare` (short causal convolutions with silu over q, k and v, unit q and k,
// beta and the decays, all in 32-bit), `conv_state` (the convolutions' last inputs into the slot),
// `scan` (the recurrence, token by token; long portions go through recurrent_blocks.cu instead) and `output` (per-head RMS norm
// times a sigmoid gate).  The order of every sum in these kernels is the same however the request was cut into steps and whatever else is in
// the batch.  Long portions' blocks add up in an order of their own: there a result depends on the cutting, to rounding.
#include "common.cuh"

#include <type_traits>

namespace lb {

constexpr int kPrepareMaxPerLane = 16;   // key_dim <= 512

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplusf_(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// The convolution's input of channel `ch` at relative time `rel` of the token's portion (negative: from the state,
// whose rows hold relative times -(taps-1) .. -1).
template <typename T>
__device__ __forceinline__ float conv_input(const T* __restrict__ proj, int proj_width, const T* __restrict__ state_rows, int channels,
                                            int start, int rel, int taps, int ch) {
    if (rel >= 0) return to_float(proj[static_cast<size_t>(start + rel) * proj_width + ch]);
    const int row = taps - 1 + rel;
    return row >= 0 ? to_float(state_rows[static_cast<size_t>(row) * channels + ch]) : 0.0f;
}

// y = silu(sum_j w[ch, taps-1-j] * input(t - j)), lags in the order j = 0, 1, ...  (Loading up to eight taps into
// registers before the first is used, under predicates, took 89 us where this loop takes 48.)
template <typename T>
__device__ __forceinline__ float conv_silu(const T* __restrict__ proj, int proj_width, const T* __restrict__ state_rows, int channels,
                                           const float* __restrict__ weight, int start, int rel, int taps, int ch) {
    float acc = 0.0f;
    for (int j = 0; j < taps; ++j)
        acc += weight[static_cast<size_t>(ch) * taps + (taps - 1 - j)] * conv_input(proj, proj_width, state_rows, channels, start, rel - j, taps, ch);
    return acc * sigmoidf_(acc);
}

// grid (tokens, slices of a token's units), a warp per unit: the `groups` query heads, the `groups` key heads, the
// `heads` value heads, and per head its decays and beta.
//   proj [tokens, proj_width]: q (groups x dk) | k (groups x dk) | v (heads x dv) | b (heads) | unused
//   ag   [tokens, ag_width]:   a (heads x dk) | ...
//   q_out, k_out [tokens, groups, dk], v_out [tokens, heads, dv], beta_out [tokens, heads], g_out [tokens, heads, dk]: 32-bit
template <typename T, bool UPDATE>
__global__ void gdr_prepare_kernel(const T* __restrict__ proj, int proj_width, const T* __restrict__ ag, int ag_width,
                                   std::conditional_t<UPDATE, T*, const T* __restrict__> conv_state, const float* __restrict__ conv_weight,
                                   const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                   float* __restrict__ q_out, float* __restrict__ k_out, float* __restrict__ v_out,
                                   float* __restrict__ beta_out, float* __restrict__ g_out,
                                   const int* __restrict__ token_segment, const int* __restrict__ segment_start,
                                   const int* __restrict__ segment_slot, int heads, int groups, int dk, int dv, int taps,
                                   int num_slots, float unit_eps, float q_scale, int* status, int decay_per_head) {
    wait_for_previous_kernel();
    allow_next_kernel();
    // decay_per_head: `ag` holds one decay logit per head (heads columns) and dt_bias one element per head; the head's
    // decay is written to all of its key channels.
    // UPDATE: every portion of the step is one token, and the lane that convolves a channel (the only reader of that
    // channel's rows in the slot) also shifts the rows and appends the token's input; no state kernel runs after this one.
    // (Otherwise the state is read-only here, and says so: the loads were a third slower without it.)
    const int token = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int segment = token_segment[token];
    const int start = segment_start[segment];
    const int slot = segment_slot[segment];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0) report_error(status, kBadSlot);
        return;
    }
    const int channels = 2 * groups * dk + heads * dv;
    auto state_rows = conv_state + static_cast<size_t>(slot) * (taps > 1 ? taps - 1 : 0) * channels;
    const int rel = token - start;
    auto shift_state = [&](int ch) {
        if constexpr (UPDATE) {
            if (taps <= 1) return;
            for (int i = 0; i + 2 < taps; ++i) state_rows[static_cast<size_t>(i) * channels + ch] = state_rows[static_cast<size_t>(i + 1) * channels + ch];
            state_rows[static_cast<size_t>(taps - 2) * channels + ch] = proj[static_cast<size_t>(token) * proj_width + ch];
        }
    };
    const int units = 2 * groups + 2 * heads;
    for (int unit = blockIdx.y * warps + warp; unit < units; unit += gridDim.y * warps) {
        if (unit < 2 * groups) {
            // a query or key head: convolution, silu, unit length (and the query's scale)
            const bool is_query = unit < groups;
            const int head = is_query ? unit : unit - groups;
            const int ch0 = unit * dk;   // q channels come first, then k
            float values[kPrepareMaxPerLane];
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < kPrepareMaxPerLane; ++i) {
                const int c = lane + 32 * i;
                values[i] = 0.0f;
                if (c < dk) {
                    values[i] = conv_silu(proj, proj_width, state_rows, channels, conv_weight, start, rel, taps, ch0 + c);
                    sum += values[i] * values[i];
                    shift_state(ch0 + c);
                }
            }
            sum = warp_sum(sum);
            const float inv = rsqrtf(sum + unit_eps) * (is_query ? q_scale : 1.0f);
            float* dst = (is_query ? q_out : k_out) + (static_cast<size_t>(token) * groups + head) * dk;
#pragma unroll
            for (int i = 0; i < kPrepareMaxPerLane; ++i) {
                const int c = lane + 32 * i;
                if (c < dk) dst[c] = values[i] * inv;
            }
        } else if (unit < 2 * groups + heads) {
            const int head = unit - 2 * groups;
            const int ch0 = 2 * groups * dk + head * dv;
            float* dst = v_out + (static_cast<size_t>(token) * heads + head) * dv;
            for (int c = lane; c < dv; c += 32) {
                dst[c] = conv_silu(proj, proj_width, state_rows, channels, conv_weight, start, rel, taps, ch0 + c);
                shift_state(ch0 + c);
            }
        } else {
            const int head = unit - 2 * groups - heads;
            const float rate = expf(a_log[head]);
            const T* a_row = ag + static_cast<size_t>(token) * ag_width + static_cast<size_t>(head) * dk;
            float* dst = g_out + (static_cast<size_t>(token) * heads + head) * dk;
            if (decay_per_head) {
                const float decay = expf(-rate * softplusf_(to_float(ag[static_cast<size_t>(token) * ag_width + head]) + dt_bias[head]));
                for (int c = lane; c < dk; c += 32) dst[c] = decay;
            } else {
                for (int c = lane; c < dk; c += 32) dst[c] = expf(-rate * softplusf_(to_float(a_row[c]) + dt_bias[head * dk + c]));
            }
            if (lane == 0) beta_out[static_cast<size_t>(token) * heads + head] = sigmoidf_(to_float(proj[static_cast<size_t>(token) * proj_width + channels + head]));
        }
    }
}

// The same for portions of several tokens, four taps and heads of up to 128 channels that come in fours: a piece of L lanes (L a power of two,
// four neighbouring channels a lane) walks over kPrepareRun neighbouring rows of one unit with the convolution's last inputs and the taps' weights
// in registers, so that an input is read once and not once a tap.  The squares of a unit norm are added up as the kernel above adds them (channels
// 32 apart, then over the warp), by way of shared memory, so that a token's numbers are the same bits whatever else is in its step.
// grid (groups of tokens, units), four warps.
// What bounds it: the 32-bit rows it writes (16 KB a token at 8 heads of 128 x 128).  Measured at
// those sizes and 2,048 tokens: 25.4 us, 67 us with a lane per channel that reads its taps' inputs each for itself.
constexpr int kPrepareRun = 8, kPrepareTaps = 4;

template <typename T>
__device__ __forceinline__ void load_four(const T* source, float (&values)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(source);
        values[0] = x.x, values[1] = x.y, values[2] = x.z, values[3] = x.w;
    } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(source);
        const float2 low = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(raw.x)), high = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(raw.y));
        values[0] = low.x, values[1] = low.y, values[2] = high.x, values[3] = high.y;
    }
}

template <typename T>
__global__ void __launch_bounds__(128)
gdr_prepare_run_kernel(const T* __restrict__ proj, int proj_width, const T* __restrict__ ag, int ag_width, const T* __restrict__ conv_state,
                       const float* __restrict__ conv_weight, const float* __restrict__ a_log, const float* __restrict__ dt_bias, float* __restrict__ q_out,
                       float* __restrict__ k_out, float* __restrict__ v_out, float* __restrict__ beta_out, float* __restrict__ g_out,
                       const int* __restrict__ token_segment, const int* __restrict__ segment_start, const int* __restrict__ segment_slot, int tokens, int heads, int groups,
                       int dk, int dv, int num_slots, float unit_eps, float q_scale, int* status, int decay_per_head) {
    wait_for_previous_kernel();
    allow_next_kernel();
    constexpr int TAPS = kPrepareTaps;
    __shared__ __align__(16) float rows_s[4][128];   // a warp's rows of queries or keys, its pieces' side by side
    const int unit = blockIdx.y, warp = threadIdx.x >> 5;
    const bool is_value = unit >= 2 * groups && unit < 2 * groups + heads, is_decay = unit >= 2 * groups + heads;
    const int width = is_value ? dv : dk;
    int lanes = 1;   // L
    while (4 * lanes < width) lanes <<= 1;
    const int piece = (threadIdx.x & 31) / lanes, lane = (threadIdx.x & 31) % lanes, pieces = 32 / lanes;
    const int first = (static_cast<int>(blockIdx.x) * 4 + warp) * pieces * kPrepareRun + piece * kPrepareRun;
    if (first - piece * kPrepareRun >= tokens) return;   // the whole warp
    const int channels = 2 * groups * dk + heads * dv, c = 4 * lane;
    const bool live = c < width;
    if (is_decay) {
        const int head = unit - 2 * groups - heads;
        const float rate = expf(a_log[head]);
        float bias[4] = {};
        if (live) {
#pragma unroll
            for (int e = 0; e < 4; ++e) bias[e] = dt_bias[decay_per_head ? head : head * dk + c + e];
        }
        for (int token = first; token < min(tokens, first + kPrepareRun); ++token) {
            const T* row = ag + static_cast<size_t>(token) * ag_width;
            float z[4], decay[4];
            if (decay_per_head) {
                z[0] = z[1] = z[2] = z[3] = to_float(row[head]);
            } else if (live) {
                load_four(row + head * dk + c, z);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) decay[e] = decay_per_head && e > 0 ? decay[0] : expf(-rate * softplusf_(z[e] + bias[e]));
            if (live) *reinterpret_cast<float4*>(g_out + (static_cast<size_t>(token) * heads + head) * dk + c) = make_float4(decay[0], decay[1], decay[2], decay[3]);
            if (lane == 0) beta_out[static_cast<size_t>(token) * heads + head] = sigmoidf_(to_float(proj[static_cast<size_t>(token) * proj_width + channels + head]));
        }
        return;
    }
    const int ch0 = is_value ? 2 * groups * dk + (unit - 2 * groups) * dv : unit * dk;   // q channels come first, then k, then v
    float weight[4][TAPS], before[TAPS - 1][4];   // before[j]: the input of j + 1 tokens ago
    if (live) {
#pragma unroll
        for (int e = 0; e < 4; ++e) load_four<float>(conv_weight + static_cast<size_t>(ch0 + c + e) * TAPS, weight[e]);
    }
    int segment = -1;
    for (int token = first; token < first + kPrepareRun; ++token) {
        const bool real = token < tokens;   // (the lanes of a piece agree; the warp's pieces meet in the sums below)
        const int now = real ? token_segment[token] : segment;
        bool good = real;
        if (real && (now != segment || token == first)) {
            segment = now;
            const int start = segment_start[segment], slot = segment_slot[segment];
            if (slot < 0 || slot >= num_slots) {
                if (lane == 0) report_error(status, kBadSlot);
                segment = -1;   // asked again for the next token
                good = false;
            } else if (live) {
                const T* state_rows = conv_state + static_cast<size_t>(slot) * (TAPS - 1) * channels;
#pragma unroll
                for (int j = 0; j < TAPS - 1; ++j) {
                    const int rel = token - start - 1 - j;
                    if (rel >= 0) load_four(proj + static_cast<size_t>(start + rel) * proj_width + ch0 + c, before[j]);
                    else load_four(state_rows + static_cast<size_t>(TAPS - 1 + rel) * channels + ch0 + c, before[j]);
                }
            }
        }
        float values[4] = {};
        if (good && live) {
            float input[4];
            load_four(proj + static_cast<size_t>(token) * proj_width + ch0 + c, input);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float acc = weight[e][TAPS - 1] * input[e];   // as conv_silu: left to itself the compiler fuses the first product, not the second
#pragma unroll
                for (int j = 1; j < TAPS; ++j) acc = fmaf(weight[e][TAPS - 1 - j], before[j - 1][e], acc);
                values[e] = acc * sigmoidf_(acc);
            }
#pragma unroll
            for (int j = TAPS - 2; j > 0; --j)
#pragma unroll
                for (int e = 0; e < 4; ++e) before[j][e] = before[j - 1][e];
#pragma unroll
            for (int e = 0; e < 4; ++e) before[0][e] = input[e];
        }
        if (is_value) {
            if (good && live) *reinterpret_cast<float4*>(v_out + (static_cast<size_t>(token) * heads + unit - 2 * groups) * dv + c) = make_float4(values[0], values[1], values[2], values[3]);
        } else {
            // unit length (and the query's scale)
            const int warp_lane = threadIdx.x & 31;
            float sum = 0.0f;
            __syncwarp();   // the token before's rows have been read
            *reinterpret_cast<float4*>(&rows_s[warp][4 * warp_lane]) = make_float4(values[0], values[1], values[2], values[3]);
            __syncwarp();
            for (int other = 0; other < pieces; ++other) {
                float squares = 0.0f;
                for (int channel = warp_lane; channel < width; channel += 32) {
                    const float value = rows_s[warp][4 * lanes * other + channel];
                    squares += value * value;
                }
                squares = warp_sum(squares);
                if (other == piece) sum = squares;
            }
            const bool is_query = unit < groups;
            const float inv = rsqrtf(sum + unit_eps) * (is_query ? q_scale : 1.0f);
            float* destination = (is_query ? q_out : k_out) + (static_cast<size_t>(token) * groups + (is_query ? unit : unit - groups)) * dk + c;
            if (good && live) *reinterpret_cast<float4*>(destination) = make_float4(values[0] * inv, values[1] * inv, values[2] * inv, values[3] * inv);
        }
    }
}

// grid (portions, channel slices): the slot's rows become the last taps-1 inputs of [old rows ; the portion's inputs].
// A thread walks a channel's rows upwards; row i is written after row length + i (> i) was read.
template <typename T>
__global__ void gdr_conv_state_kernel(const T* __restrict__ proj, int proj_width, T* __restrict__ conv_state, const int* __restrict__ segment_start,
                                      const int* __restrict__ segment_length, const int* __restrict__ segment_slot, int channels, int taps,
                                      int num_slots) {
    wait_for_previous_kernel();
    allow_next_kernel();
    const int segment = blockIdx.x;
    const int slot = segment_slot[segment];
    if (slot < 0 || slot >= num_slots) return;   // reported by the kernel before
    const int start = segment_start[segment], length = segment_length[segment];
    T* rows = conv_state + static_cast<size_t>(slot) * (taps - 1) * channels;
    for (int ch = blockIdx.y * blockDim.x + threadIdx.x; ch < channels; ch += gridDim.y * blockDim.x) {
        for (int i = 0; i < taps - 1; ++i) {
            const int rel = length - (taps - 1) + i;
            rows[static_cast<size_t>(i) * channels + ch] =
                rel >= 0 ? proj[static_cast<size_t>(start + rel) * proj_width + ch] : rows[static_cast<size_t>(taps - 1 + rel) * channels + ch];
        }
    }
}

// The recurrence.  grid (portions, heads, ceil(dv / 8)); a block holds 8 columns of S, a thread R = 8 rows of one
// column in registers.  A column's DKP rows (key_dim rounded up, padded rows stay zero) are spread over SPLIT = DKP / 8
// neighbouring lanes; lane `part` holds the rows ((i / 4) * SPLIT + part) * 4 + i % 4, so that the lanes of a column read
// neighbouring 16-byte pieces of k, q and g from shared memory.  A token's step is one chain of dependent instructions
// (decay, dot, the lanes' sums, write, read-out, the lanes' sums) that a warp issues in order, and a multiprocessor's
// schedulers hold one warp each here, which issues about one instruction in three cycles: so the kernel is as fast as a
// warp's instructions per token are few, hence many small blocks (a sequence of 2,048 tokens at 8 heads of 64 x 128
// runs on 128 blocks of two warps).  Measured at those sizes: 32 rows x 1 column a lane 304 ns a token, 8 rows x 4
// columns 382 ns, 8 rows x 1 column 273 ns.  Tokens come in batches through two stages of shared memory: the next
// batch's k, q, g, v and beta are on their way (cp.async) while this one is worked on.  Every sum runs in a fixed order.
constexpr int kScanCols = 8, kScanThreadCols = 1, kScanThreadRows = 8;

template <int DKP>
struct ScanShared {
    static constexpr int kBatch = 8;   // small stages: many blocks fit a multiprocessor, whose warps hide each other's waits
    static constexpr int kStageFloats = kBatch * (3 * DKP + kScanCols + 4);   // k, q, g rows, v columns, beta (padded to 16 bytes)
    static constexpr size_t kBytes = 2 * kStageFloats * sizeof(float);
};

__device__ __forceinline__ void scan_copy_4(float* shared_destination, const float* global_source) {
    const uint32_t destination = static_cast<uint32_t>(__cvta_generic_to_shared(shared_destination));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(destination), "l"(global_source) : "memory");
}
__device__ __forceinline__ void scan_copy_16(float* shared_destination, const float* global_source) {
    const uint32_t destination = static_cast<uint32_t>(__cvta_generic_to_shared(shared_destination));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(destination), "l"(global_source) : "memory");
}

// DELTA false: the plain linear recurrence S <- diag(g_t) S + k_t v_t^T, o_t = S^T q_t (no correction by what the state
// already holds under k_t, no beta): the same state layout, stages and read-out with a shorter chain per token.
template <int DKP, int SPLIT, bool DELTA>
__global__ void __launch_bounds__((kScanCols / kScanThreadCols) * SPLIT)
gdr_scan_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ g, const float* __restrict__ v,
                const float* __restrict__ beta, float* __restrict__ state, float* __restrict__ out, const int* __restrict__ segment_start,
                const int* __restrict__ segment_length, const int* __restrict__ segment_slot, int heads, int groups, int dk, int dv,
                int num_slots, int* status, const int* __restrict__ segment_list) {
    wait_for_previous_kernel();
    allow_next_kernel();
    // segment_list (may be null): the portions this launch runs.
    constexpr int R = kScanThreadRows, C = kScanThreadCols;
    static_assert(DKP == R * SPLIT && SPLIT <= 32, "a column's rows lie in one warp");
    using Shared = ScanShared<DKP>;
    constexpr int kBatch = Shared::kBatch;
    extern __shared__ __align__(16) float scan_memory[];
    const int segment = segment_list ? segment_list[blockIdx.x] : static_cast<int>(blockIdx.x);
    const int head = blockIdx.y, col0 = blockIdx.z * kScanCols;
    const int tid = threadIdx.x, column_group = tid / SPLIT, part = tid % SPLIT;
    const int group = head / (heads / groups);
    const int slot = segment_slot[segment];
    if (slot < 0 || slot >= num_slots) {
        if (tid == 0) report_error(status, kBadSlot);
        return;
    }
    const int start = segment_start[segment], length = segment_length[segment];
    const int column = col0 + C * column_group;   // the thread's first column
    auto k_of = [&](int stage) { return scan_memory + stage * Shared::kStageFloats; };
    auto q_of = [&](int stage) { return k_of(stage) + kBatch * DKP; };
    auto g_of = [&](int stage) { return k_of(stage) + 2 * kBatch * DKP; };
    auto v_of = [&](int stage) { return k_of(stage) + 3 * kBatch * DKP; };
    auto beta_of = [&](int stage) { return v_of(stage) + kBatch * kScanCols; };
    // The state's loads are on their way before anything else: a block of one token waits for little else.  64 tokens that decode, 8 heads: of 128 x 128
    // 60 us and with the delta rule 58 (67 and 65 with the padding and the inputs' copies before them), of 64 x 128 20 us (27).
    float* S_base = state + (static_cast<size_t>(slot) * heads + head) * dk * dv;
    float S[C][R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = ((i >> 2) * SPLIT + part) * 4 + (i & 3);
#pragma unroll
        for (int c = 0; c < C; ++c) S[c][i] = (row < dk && column + c < dv) ? S_base[static_cast<size_t>(row) * dv + column + c] : 0.0f;
    }
    // The padding (rows of S past key_dim, columns past value_dim), where there is any, is written once: the copies never touch it.
    for (int index = tid; dk < DKP && index < 2 * kBatch * DKP; index += blockDim.x) {
        const int stage = index / (kBatch * DKP), rest = index - stage * kBatch * DKP;
        if (rest % DKP >= dk) {
            k_of(stage)[rest] = 0.0f;
            q_of(stage)[rest] = 0.0f;
            g_of(stage)[rest] = 1.0f;
        }
    }
    for (int index = tid; col0 + kScanCols > dv && index < 2 * kBatch * kScanCols; index += blockDim.x) {
        const int stage = index / (kBatch * kScanCols), rest = index - stage * kBatch * kScanCols;
        if (col0 + rest % kScanCols >= dv) v_of(stage)[rest] = 0.0f;
    }
    const bool wide = dk % 4 == 0;   // rows of 16-byte multiples (the buffers are 16-byte aligned)
    auto fetch = [&](int stage, int t0) {
        const int n = min(kBatch, length - t0);
        if (wide) {
            const int pieces = dk / 4;
            for (int index = tid; index < n * pieces; index += blockDim.x) {
                const int tt = index / pieces, c = 4 * (index - tt * pieces);
                const size_t token = static_cast<size_t>(start + t0 + tt);
                scan_copy_16(k_of(stage) + tt * DKP + c, k + (token * groups + group) * dk + c);
                scan_copy_16(q_of(stage) + tt * DKP + c, q + (token * groups + group) * dk + c);
                scan_copy_16(g_of(stage) + tt * DKP + c, g + (token * heads + head) * dk + c);
            }
        } else {
            for (int index = tid; index < n * dk; index += blockDim.x) {
                const int tt = index / dk, c = index - tt * dk;
                const size_t token = static_cast<size_t>(start + t0 + tt);
                scan_copy_4(k_of(stage) + tt * DKP + c, k + (token * groups + group) * dk + c);
                scan_copy_4(q_of(stage) + tt * DKP + c, q + (token * groups + group) * dk + c);
                scan_copy_4(g_of(stage) + tt * DKP + c, g + (token * heads + head) * dk + c);
            }
        }
        const int columns = min(kScanCols, dv - col0);
        for (int index = tid; index < n * columns; index += blockDim.x) {
            const int tt = index / columns, c = index - tt * columns;
            scan_copy_4(v_of(stage) + tt * kScanCols + c, v + (static_cast<size_t>(start + t0 + tt) * heads + head) * dv + col0 + c);
        }
        if constexpr (DELTA)
            for (int tt = tid; tt < n; tt += blockDim.x) scan_copy_4(beta_of(stage) + tt, beta + static_cast<size_t>(start + t0 + tt) * heads + head);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(0, 0);
    int stage = 0;
    for (int t0 = 0; t0 < length; t0 += kBatch, stage ^= 1) {
        const int n = min(kBatch, length - t0);
        if (t0 + kBatch < length) {
            fetch(stage ^ 1, t0 + kBatch);   // that stage was used up in the turn before (the barrier at its end)
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float* beta_s = beta_of(stage);
        for (int tt = 0; tt < n; ++tt) {
            const float4* k4 = reinterpret_cast<const float4*>(k_of(stage) + tt * DKP);
            const float4* q4 = reinterpret_cast<const float4*>(q_of(stage) + tt * DKP);
            const float4* g4 = reinterpret_cast<const float4*>(g_of(stage) + tt * DKP);
            float values[C];
#pragma unroll
            for (int c = 0; c < C; ++c) values[c] = v_of(stage)[tt * kScanCols + C * column_group + c];
            float key[R], dots[C];
#pragma unroll
            for (int c = 0; c < C; ++c) dots[c] = 0.0f;
#pragma unroll
            for (int i = 0; i < R; i += 4) {
                const float4 decay4 = g4[(i >> 2) * SPLIT + part], key4 = k4[(i >> 2) * SPLIT + part];
                const float decay[4] = {decay4.x, decay4.y, decay4.z, decay4.w};
                key[i] = key4.x, key[i + 1] = key4.y, key[i + 2] = key4.z, key[i + 3] = key4.w;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        S[c][i + e] *= decay[e];
                        if constexpr (DELTA) dots[c] += S[c][i + e] * key[i + e];
                    }
                }
            }
            if constexpr (DELTA) {
#pragma unroll
                for (int offset = 1; offset < SPLIT; offset <<= 1) {
#pragma unroll
                    for (int c = 0; c < C; ++c) dots[c] += __shfl_xor_sync(0xffffffffu, dots[c], offset);
                }
            }
            float u[C], reads[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                u[c] = DELTA ? beta_s[tt] * (values[c] - dots[c]) : values[c];
                reads[c] = 0.0f;
            }
#pragma unroll
            for (int i = 0; i < R; i += 4) {
                const float4 query4 = q4[(i >> 2) * SPLIT + part];
                const float query[4] = {query4.x, query4.y, query4.z, query4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        S[c][i + e] += key[i + e] * u[c];
                        reads[c] += S[c][i + e] * query[e];
                    }
                }
            }
#pragma unroll
            for (int offset = 1; offset < SPLIT; offset <<= 1) {
#pragma unroll
                for (int c = 0; c < C; ++c) reads[c] += __shfl_xor_sync(0xffffffffu, reads[c], offset);
            }
            if (part == 0) {
                float* destination = out + (static_cast<size_t>(start + t0 + tt) * heads + head) * dv + column;
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (column + c < dv) destination[c] = reads[c];
            }
        }
        __syncthreads();   // this stage is refilled in the next turn
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = ((i >> 2) * SPLIT + part) * 4 + (i & 3);
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (row < dk && column + c < dv) S_base[static_cast<size_t>(row) * dv + column + c] = S[c][i];
    }
}

// grid (tokens, slices of the heads), a warp per head: out[t, h, :] = T(o / sqrt(mean(o^2) + eps) * w * sigmoid(gate[t, h, :]));
// without gates (ag null) the last factor is left out.  FOURS: rows that come in fours, on addresses that do, of at most 128 channels: a lane has
// four neighbours, and a row and its gates are on their way together (2,048 tokens of 8 heads of 128 5.9 us, 11.0 a channel at a time).
template <typename T, bool FOURS>
__global__ void gdr_output_kernel(const float* __restrict__ o, const T* __restrict__ ag, int ag_width, int gate_offset,
                                  const float* __restrict__ norm_weight, T* __restrict__ out, int heads, int dv, float eps, int gate_silu) {
    wait_for_previous_kernel();
    allow_next_kernel();   // the out-projection, launched to start early, may ask for its weights meanwhile
    const int token = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int head = blockIdx.y * warps + warp; head < heads; head += gridDim.y * warps) {
        const float* row = o + (static_cast<size_t>(token) * heads + head) * dv;
        const T* gate = ag != nullptr ? ag + static_cast<size_t>(token) * ag_width + gate_offset + static_cast<size_t>(head) * dv : nullptr;
        T* dst = out + (static_cast<size_t>(token) * heads + head) * dv;
        auto factor_of = [&](float z) { return gate == nullptr ? 1.0f : (gate_silu ? z * sigmoidf_(z) : sigmoidf_(z)); };
        if constexpr (FOURS) {
            float x[4] = {}, z[4] = {}, w[4] = {};
            const int c = 4 * lane;
            if (c < dv) {
                load_four(row + c, x);
                if (gate != nullptr) load_four(gate + c, z);
                load_four(norm_weight + c, w);
            }
            const float sum = warp_sum((x[0] * x[0] + x[1] * x[1]) + (x[2] * x[2] + x[3] * x[3]));
            const float inv = rsqrtf(sum / static_cast<float>(dv) + eps);
            if (c < dv) {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = x[e] * inv * w[e] * factor_of(z[e]);
                if constexpr (sizeof(T) == 4) {
                    *reinterpret_cast<float4*>(dst + c) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
                    const __nv_bfloat162 low = __floats2bfloat162_rn(x[0], x[1]), high = __floats2bfloat162_rn(x[2], x[3]);
                    *reinterpret_cast<uint2*>(dst + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&low), *reinterpret_cast<const uint32_t*>(&high));
                }
            }
        } else {
            float sum = 0.0f;
            for (int c = lane; c < dv; c += 32) sum += row[c] * row[c];
            sum = warp_sum(sum);
            const float inv = rsqrtf(sum / static_cast<float>(dv) + eps);
            for (int c = lane; c < dv; c += 32) dst[c] = from_float<T>(row[c] * inv * norm_weight[c] * factor_of(gate != nullptr ? to_float(gate[c]) : 0.0f));
        }
    }
}

template <int DKP, int SPLIT>
inline int launch_scan(dim3 grid, cudaStream_t stream, const float* q, const float* k, const float* g, const float* v, const float* beta,
                       float* state, float* out, const int* segment_start, const int* segment_length, const int* segment_slot, int heads,
                       int groups, int dk, int dv, int num_slots, int* status, const int* segment_list, bool early) {
    static OncePerDevice once[2];
    auto kernel = beta != nullptr ? gdr_scan_kernel<DKP, SPLIT, true> : gdr_scan_kernel<DKP, SPLIT, false>;
    const cudaError_t allowed = allow_shared_memory(once[beta != nullptr ? 1 : 0], kernel, static_cast<int>(ScanShared<DKP>::kBytes));
    if (allowed != cudaSuccess) return static_cast<int>(allowed);
    return static_cast<int>(launch_early_if(early, kernel, grid, dim3((kScanCols / kScanThreadCols) * SPLIT), ScanShared<DKP>::kBytes, stream, q, k, g, v, beta, state, out,
                                            segment_start, segment_length, segment_slot, heads, groups, dk, dv, num_slots, status, segment_list));
}

}  // namespace lb

extern "C" {

int lb_gdr_prepare(const void* proj, int proj_width, const void* ag, int ag_width, void* conv_state, const float* conv_weight,
                   const float* a_log, const float* dt_bias, float* q_out, float* k_out, float* v_out, float* beta_out, float* g_out,
                   const int* token_segment, const int* segment_start, const int* segment_slot, int tokens, int heads, int groups, int dk,
                   int dv, int taps, int num_slots, float unit_eps, float q_scale, int dtype, int* status, cudaStream_t stream, int update_state,
                   int decay_per_head) {
    if (tokens == 0) return 0;
    if (dk > 32 * lb::kPrepareMaxPerLane || taps < 1 || heads % groups != 0) return -2;
    LB_DISPATCH_DTYPE(dtype, {
        const int units = 2 * groups + 2 * heads;
        const dim3 grid(tokens, (units + 3) / 4);
        // rows that come in fours, on addresses that do: the kernel that reads every input once (each of these sizes is the same for a whole model)
        const auto in_fours = [](const void* address) { return reinterpret_cast<uintptr_t>(address) % (4 * sizeof(T)) == 0; };
        if (!update_state && taps == lb::kPrepareTaps && dk % 4 == 0 && dv % 4 == 0 && dk <= 128 && dv <= 128 && proj_width % 4 == 0 &&
            (decay_per_head || ag_width % 4 == 0) && in_fours(proj) && (decay_per_head || in_fours(ag)) && in_fours(conv_state) && reinterpret_cast<uintptr_t>(conv_weight) % 16 == 0) {
            return static_cast<int>(lb::launch_overlapped(
                lb::gdr_prepare_run_kernel<T>, dim3((tokens + 4 * lb::kPrepareRun - 1) / (4 * lb::kPrepareRun), units), dim3(128), 0, stream, static_cast<const T*>(proj),
                proj_width, static_cast<const T*>(ag), ag_width, static_cast<const T*>(conv_state), conv_weight, a_log, dt_bias, q_out, k_out, v_out, beta_out, g_out, token_segment,
                segment_start, segment_slot, tokens, heads, groups, dk, dv, num_slots, unit_eps, q_scale, status, decay_per_head));
        }
        auto launch = [&](auto kernel, auto* slots) {
            return static_cast<int>(lb::launch_overlapped(kernel, grid, dim3(128), 0, stream, static_cast<const T*>(proj), proj_width, static_cast<const T*>(ag), ag_width, slots,
                                                          conv_weight, a_log, dt_bias, q_out, k_out, v_out, beta_out, g_out, token_segment, segment_start, segment_slot, heads, groups,
                                                          dk, dv, taps, num_slots, unit_eps, q_scale, status, decay_per_head));
        };
        return update_state ? launch(lb::gdr_prepare_kernel<T, true>, static_cast<T*>(conv_state)) : launch(lb::gdr_prepare_kernel<T, false>, static_cast<const T*>(conv_state));
    })
}

int lb_gdr_conv_state(const void* proj, int proj_width, void* conv_state, const int* segment_start, const int* segment_length,
                      const int* segment_slot, int segments, int channels, int taps, int num_slots, int dtype, cudaStream_t stream) {
    if (segments == 0 || taps <= 1) return 0;
    LB_DISPATCH_DTYPE(dtype, {
        return static_cast<int>(lb::launch_overlapped(lb::gdr_conv_state_kernel<T>, dim3(segments, (channels + 255) / 256), dim3(256), 0, stream, static_cast<const T*>(proj), proj_width,
                                                      static_cast<T*>(conv_state), segment_start, segment_length, segment_slot, channels, taps, num_slots));
    })
}

// segment_list (may be null): the portions to run, `segments` of them.
// beta null: the plain linear recurrence (no delta rule).
// few_tokens: the scan's work is short and it starts early (see launch_early_if).  Layers of linear attention with 128 key channels, with an early start and without: 64 single
// tokens 94 and 95.5 us, 64 portions of two 102 and 103, one of 17 30.6 and 32.2, of 48 44.2 and 44.1; five of 20 51 and 48, of 100 105 and 85, one of 130 103 and 70.
int lb_gdr_scan(const float* q, const float* k, const float* g, const float* v, const float* beta, float* state, float* out,
                const int* segment_start, const int* segment_length, const int* segment_slot, int segments, int heads, int groups, int dk, int dv,
                int num_slots, int* status, cudaStream_t stream, const int* segment_list, int few_tokens) {
    if (segments == 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads % groups != 0) return -2;
    const dim3 grid(segments, heads, (dv + lb::kScanCols - 1) / lb::kScanCols);
    auto launch = dk <= 32 ? lb::launch_scan<32, 4> : dk <= 64 ? lb::launch_scan<64, 8> : dk <= 128 ? lb::launch_scan<128, 16> : lb::launch_scan<256, 32>;
    return launch(grid, stream, q, k, g, v, beta, state, out, segment_start, segment_length, segment_slot, heads, groups, dk, dv, num_slots, status, segment_list, few_tokens != 0);
}

int lb_gdr_output(const float* o, const void* ag, int ag_width, int gate_offset, const float* norm_weight, void* out, int tokens, int heads, int dv,
                  float eps, int dtype, cudaStream_t stream, int gate_silu) {
    if (tokens == 0) return 0;
    LB_DISPATCH_DTYPE(dtype, {
        const auto in_fours = [](const void* address) { return reinterpret_cast<uintptr_t>(address) % (4 * sizeof(T)) == 0; };
        const bool fours = dv % 4 == 0 && dv <= 128 && (ag == nullptr || (ag_width % 4 == 0 && gate_offset % 4 == 0 && in_fours(ag))) && in_fours(out) &&
                           ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(norm_weight)) & 15) == 0;
        auto kernel = fours ? lb::gdr_output_kernel<T, true> : lb::gdr_output_kernel<T, false>;
        return static_cast<int>(lb::launch_overlapped(kernel, dim3(tokens, (heads + 3) / 4), dim3(128), 0, stream, o, static_cast<const T*>(ag), ag_width, gate_offset, norm_weight,
                                                      static_cast<T*>(out), heads, dv, eps, gate_silu));
    })
}

}  // extern "C"
