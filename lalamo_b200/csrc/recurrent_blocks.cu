// Long portions of the recurrences of gated_delta.cu and linear_attention.cu, 32 tokens at a time:
//
//   S <- diag(g_t) S;   u_t = beta_t (v_t - S^T k_t)  (or v_t, see the second half);   S <- S + k_t u_t^T;   o_t = S^T q_t
//
// Over a block of tokens that starts from the state S, with D_i the decays' product from the block's start to token i and
// G(i, j) that from token j + 1 to token i (element by element over the key channels),
//
//   u_i = beta_i (v_i - S^T (D_i k_i) - sum_{j<i} A_ij u_j),   A_ij = k_i . (G(i, j) k_j)
//   o_i = S^T (D_i q_i) + sum_{j<=i} B_ij u_j,                 B_ij = q_i . (G(i, j) k_j)
//   S'  = diag(D_end) S + sum_j (G(end, j) k_j) u_j^T
//
// so U = T (V - K~ S) with T = (I + diag(beta) A)^-1 diag(beta), a 32 x 32 lower triangle, and with W = T K~ all that is left to do in
// order is   [U ; O] = [T V ; B T V] + [-W ; Q~ - B W] S   and   S' = diag(D_end) S + K^T U.
//
// `prepare` makes these matrices, one CTA per block and head, all side by side; `walk` goes over a portion's blocks in order, a CTA
// per portion, head and 8 columns of the state, whose matrices arrive by bulk copies some blocks ahead.  All decays enter as
// products of factors of at most one (never as quotients, which overflow under strong decays), everything is 32-bit FMA.
// What bounds it: `walk` reads 50 KB a block through L2 and shared memory for 98 thousand multiply-adds (128 key channels), about
// as many cycles for either; of its 2,440 cycles a block the first product takes 880, the sums over the warps 520, the second
// product 860.  `prepare` is bound by its shared-memory reads.  Measured, 8 heads of 128 x 128, a portion of 2,048 tokens: prepare 55 us, walk
// 94 us (663 us token by token); without the correction, 1,501 + 751 tokens of 64 x 128 heads: 38 + 10 + 20 us (228 us as chunks of 256
// tokens scanned side by side with further columns for their transitions).
#include "tcgen05.cuh"

#include <type_traits>

namespace lb {

constexpr int kBlockTokens = 32, kWalkCols = 8, kBlockThreads = 256;
constexpr int kTrianglePitch = 36;   // floats of a row of a 32 x 32 matrix in shared memory: rows start on 16 bytes, in banks of their own

template <int DKP>
struct BlockPack {
    static constexpr int kRows = 64;                               // rows of [-W ; Q']
    static constexpr int kMatrix = DKP * kRows;                   // their columns one after the other
    static constexpr int kFloats = kMatrix + 32 * DKP + DKP;      // then K^ [32][DKP], then D_end
    static constexpr int kValues = 64 * kWalkCols;                // per 8 columns of the state: [T V ; B T V]
};

template <int DKP>
struct PrepareShared {
    static constexpr int kPitch = DKP + 4;
    static constexpr int kValuePitch = 132;
    // three CTAs share a multiprocessor up to 128 key channels: the values lie where the decays were
    static constexpr int kFloats = 2 * 32 * kPitch + 32 * (kPitch > kValuePitch ? kPitch : kValuePitch) + 3 * 32 * kTrianglePitch + DKP + 32;
    static constexpr int kBytes = kFloats * 4;
};

// N neighbouring floats (N a multiple of 4, or 1 or 2), aligned to their size up to 16 bytes.
template <int N>
__device__ __forceinline__ void load_floats(const float* source, float (&values)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(source + i);
            values[i] = x.x, values[i + 1] = x.y, values[i + 2] = x.z, values[i + 3] = x.w;
        }
    } else if constexpr (N == 2) {
        const float2 x = *reinterpret_cast<const float2*>(source);
        values[0] = x.x, values[1] = x.y;
    } else {
        values[0] = source[0];
    }
}

// The sums over the warp of 32 values a lane: lane l gets that of values[l].
__device__ __forceinline__ float warp_sums_of_32(float (&values)[32], int lane) {
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int n = 0; n < half; ++n) {
            const float keep = upper ? values[n + half] : values[n], give = upper ? values[n] : values[n + half];
            values[n] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return values[0];
}

// first[r][e] += sum_{j <= i} m1[i][j] x[j][column e], second likewise with m2, for the rows i = 4 rg + r, with m1 and m2 given at [j][i]
// (FIRST false: the second alone).  What lies above the diagonal is left out, not multiplied by zero: a token without a number must not
// reach those before it.
template <bool FIRST>
__device__ __forceinline__ void triangle_products(float (&first)[4][4], float (&second)[4][4], const float* m1, const float* m2, const float* x, int x_pitch, int rg) {
    auto add = [&](int j, auto from) {
        const float4 xv = *reinterpret_cast<const float4*>(x + j * x_pitch), b = *reinterpret_cast<const float4*>(m2 + j * kTrianglePitch + 4 * rg);
        const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, bs[4] = {b.x, b.y, b.z, b.w};
        float4 a = b;
        if constexpr (FIRST) a = *reinterpret_cast<const float4*>(m1 + j * kTrianglePitch + 4 * rg);
        [[maybe_unused]] const float as[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int r = from; r < 4; ++r) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if constexpr (FIRST) first[r][e] += as[r] * xs[e];
                second[r][e] += bs[r] * xs[e];
            }
        }
    };
#pragma unroll 4
    for (int j = 0; j < 4 * rg; ++j) add(j, std::integral_constant<int, 0>{});
    add(4 * rg, std::integral_constant<int, 0>{});
    add(4 * rg + 1, std::integral_constant<int, 1>{});
    add(4 * rg + 2, std::integral_constant<int, 2>{});
    add(4 * rg + 3, std::integral_constant<int, 3>{});
}

// The block's keys, queries and decays into shared memory, rows of DKP + 4 floats.  Tokens past the end have no key, no query and no decay, channels
// past dk likewise.
template <int DKP>
__device__ __forceinline__ void load_block(float* k_s, float* q_s, float* g_s, const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ g,
                                           int start, int n, int head, int group, int heads, int groups, int dk) {
    constexpr int P = DKP + 4;
    const int tid = threadIdx.x;
    if (dk % 4 == 0) {
#pragma unroll 4
        for (int index = tid; index < 32 * (DKP / 4); index += kBlockThreads) {
            const int t = index / (DKP / 4), c = 4 * (index % (DKP / 4));
            const bool real = t < n && c < dk;
            const size_t row = static_cast<size_t>(start + t);
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
            *reinterpret_cast<float4*>(k_s + t * P + c) = real ? *reinterpret_cast<const float4*>(k + (row * groups + group) * dk + c) : zero;
            *reinterpret_cast<float4*>(q_s + t * P + c) = real ? *reinterpret_cast<const float4*>(q + (row * groups + group) * dk + c) : zero;
            *reinterpret_cast<float4*>(g_s + t * P + c) = real ? *reinterpret_cast<const float4*>(g + (row * heads + head) * dk + c) : one;
        }
    } else {
        for (int index = tid; index < 32 * DKP; index += kBlockThreads) {
            const int t = index / DKP, c = index % DKP;
            const bool real = t < n && c < dk;
            const size_t row = static_cast<size_t>(start + t);
            k_s[t * P + c] = real ? k[(row * groups + group) * dk + c] : 0.0f;
            q_s[t * P + c] = real ? q[(row * groups + group) * dk + c] : 0.0f;
            g_s[t * P + c] = real ? g[(row * heads + head) * dk + c] : 1.0f;
        }
    }
}

// A[i][j] (DELTA) and B at [j][i] within each half of 16 tokens: a warp takes a column j, carries G(i, j) k_j down the rows, a lane
// DKP / 32 channels.
template <int DKP, bool DELTA>
__device__ __forceinline__ void within_halves(float* a_s, float* bt_s, const float* k_s, const float* q_s, const float* g_s) {
    constexpr int P = DKP + 4, TP = kTrianglePitch, CPL = DKP / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
    for (int j = warp; j < 32; j += kBlockThreads / 32) {
        const int base = j & 16, jj = j & 15;
        float carried[CPL], sums[32];
        load_floats<CPL>(k_s + j * P + lane * CPL, carried);
#pragma unroll
        for (int ii = 0; ii < 16; ++ii) {
            sums[ii] = sums[16 + ii] = 0.0f;
            if (ii >= jj) {
                const int row = (base + ii) * P + lane * CPL;
                float query[CPL];
                load_floats<CPL>(q_s + row, query);
                if (ii > jj) {
                    float decay[CPL];
                    load_floats<CPL>(g_s + row, decay);
#pragma unroll
                    for (int e = 0; e < CPL; ++e) carried[e] *= decay[e];
                    if constexpr (DELTA) {
                        float key[CPL];
                        load_floats<CPL>(k_s + row, key);
#pragma unroll
                        for (int e = 0; e < CPL; ++e) sums[ii] += key[e] * carried[e];
                    }
                }
#pragma unroll
                for (int e = 0; e < CPL; ++e) sums[16 + ii] += query[e] * carried[e];
            }
        }
        const float sum = warp_sums_of_32(sums, lane);
        if (lane < 16) {
            if constexpr (DELTA) a_s[(base + lane) * TP + j] = sum;
            if (base) bt_s[j * TP + lane] = 0.0f;   // rows before the column
        } else {
            bt_s[j * TP + base + lane - 16] = sum;
        }
    }
}

// A and B between the halves, a thread per pair: what of the keys belongs to the lower half is times the decays to its end, the keys and
// queries of the upper half times those from its start.
template <int DKP, bool DELTA>
__device__ __forceinline__ void between_halves(float* a_s, float* bt_s, const float* k_s, const float* q_s) {
    constexpr int P = DKP + 4, TP = kTrianglePitch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = lane & 15, i = 16 + 2 * warp + (lane >> 4);
    float a = 0.0f, b = 0.0f;
#pragma unroll 8
    for (int c = 0; c < DKP; c += 4) {
        const float4 kj = *reinterpret_cast<const float4*>(k_s + j * P + c), qi = *reinterpret_cast<const float4*>(q_s + i * P + c);
        b += qi.x * kj.x;
        b += qi.y * kj.y;
        b += qi.z * kj.z;
        b += qi.w * kj.w;
        if constexpr (DELTA) {
            const float4 ki = *reinterpret_cast<const float4*>(k_s + i * P + c);
            a += ki.x * kj.x;
            a += ki.y * kj.y;
            a += ki.z * kj.z;
            a += ki.w * kj.w;
        }
    }
    if constexpr (DELTA) a_s[i * TP + j] = a;
    bt_s[j * TP + i] = b;
}

// The blocks of all long portions are numbered through: portion 0's, portion 1's, and so on.
struct PortionBlock {
    int portion, block;   // block < 0: there is no such block
};
__device__ __forceinline__ int blocks_before(const int* __restrict__ long_table, const int* __restrict__ segment_length, int entry) {
    int blocks = 0;
    for (int i = 0; i < entry; ++i) blocks += (segment_length[long_table[3 * i]] + kBlockTokens - 1) / kBlockTokens;
    return blocks;
}
__device__ __forceinline__ PortionBlock find_block(const int* __restrict__ long_table, const int* __restrict__ segment_length, int long_portions, int index) {
    for (int i = 0; i < long_portions; ++i) {
        const int portion = long_table[3 * i], blocks = (segment_length[portion] + kBlockTokens - 1) / kBlockTokens;
        if (index < blocks) return PortionBlock{portion, index};
        index -= blocks;
    }
    return PortionBlock{0, -1};
}

// A launch takes the blocks of the numbers window .. window + gridDim.x - 1: scratch is for so many, whatever the step's size.

// grid (blocks, heads).  window + blockIdx.x is a block's number among those of the long portions that `long_table` lists (rows of three
// numbers, the first of which is the portion).
//   q, k [tokens, groups, dk], g [tokens, heads, dk], v [tokens, heads, dv], beta [tokens, heads]
//   pack [block][head][BlockPack::kFloats], vpack [block][head][ceil(dv / 8)][BlockPack::kValues]
template <int DKP>
__global__ void __launch_bounds__(kBlockThreads, DKP <= 128 ? 3 : 1)
recurrent_prepare_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ g, const float* __restrict__ v,
                         const float* __restrict__ beta, float* __restrict__ pack, float* __restrict__ vpack, const int* __restrict__ long_table, int long_portions, const int* __restrict__ segment_start,
                const int* __restrict__ segment_length, int heads, int groups, int dk, int dv, int window) {
    wait_for_previous_kernel();
    allow_next_kernel();
    using Pack = BlockPack<DKP>;
    using Shared = PrepareShared<DKP>;
    constexpr int P = Shared::kPitch, VP = Shared::kValuePitch, TP = kTrianglePitch;
    extern __shared__ __align__(16) float prepare_memory[];
    float* k_s = prepare_memory;            // keys; then those of the lower half times the decays to its end, of the upper times those from its start
    float* q_s = k_s + 32 * P;              // queries; then times the decays from the block's start (lower half), from its own start (upper)
    float* g_s = q_s + 32 * P;              // decays; then K~
    float* v_s = g_s;                       // then values, 128 columns at a time
    float* a_s = g_s + 32 * (P > VP ? P : VP);   // A[i][j]; then B T at [j][i]
    float* bt_s = a_s + 32 * TP;            // B[i][j] at [j][i]
    float* tt_s = bt_s + 32 * TP;           // T[i][j] at [j][i]
    float* d_half = tt_s + 32 * TP;         // the decays' product over the lower half
    float* beta_s = d_half + DKP;
    const PortionBlock here = find_block(long_table, segment_length, long_portions, window + static_cast<int>(blockIdx.x));
    if (here.block < 0) return;
    const int first = kBlockTokens * here.block, n = min(kBlockTokens, segment_length[here.portion] - first);
    const int start = segment_start[here.portion] + first, head = blockIdx.y, group = head / (heads / groups);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* out = pack + (static_cast<size_t>(blockIdx.x) * heads + head) * Pack::kFloats;
    const int slices = (dv + kWalkCols - 1) / kWalkCols;
    float* v_out = vpack + (static_cast<size_t>(blockIdx.x) * heads + head) * slices * Pack::kValues;

    // The first 128 columns' values are on their way from the start: token tid / 8, columns 4 (tid % 8) + 32 i and the next three.
    auto load_values = [&](int column0, float4 (&values)[4]) {
        const int t = tid >> 3;
        const float* row = v + (static_cast<size_t>(start + t) * heads + head) * dv;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = column0 + 4 * (tid & 7) + 32 * i;
            if (dv % 4 == 0) {
                values[i] = t < n && c < dv ? *reinterpret_cast<const float4*>(row + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else {
                values[i].x = t < n && c < dv ? row[c] : 0.0f;
                values[i].y = t < n && c + 1 < dv ? row[c + 1] : 0.0f;
                values[i].z = t < n && c + 2 < dv ? row[c + 2] : 0.0f;
                values[i].w = t < n && c + 3 < dv ? row[c + 3] : 0.0f;
            }
        }
    };
    float4 first_values[4];
    load_values(0, first_values);
    load_block<DKP>(k_s, q_s, g_s, q, k, g, start, n, head, group, heads, groups, dk);
    if (tid < 32) beta_s[tid] = tid < n ? beta[static_cast<size_t>(start + tid) * heads + head] : 0.0f;
    __syncthreads();

    within_halves<DKP, true>(a_s, bt_s, k_s, q_s, g_s);
    __syncthreads();

    // A thread per channel: K^ and D_end from the raw values, then (another thread, up to 128 channels) what the products below
    // read, in place.
    auto state_keys = [&](int c) {
        float* k_hat = out + Pack::kMatrix;
        float product = 1.0f;
#pragma unroll
        for (int j = 31; j >= 0; --j) {
            k_hat[j * DKP + c] = k_s[j * P + c] * product;
            product *= g_s[j * P + c];
        }
        k_hat[32 * DKP + c] = product;
    };
    float k_raw[32], g_raw[32];
    const int in_place = DKP <= 128 ? tid - 128 : tid;   // the channel whose column this thread turns
    const bool turns = in_place >= 0 && in_place < DKP;
    if (turns) {
#pragma unroll
        for (int t = 0; t < 32; ++t) k_raw[t] = k_s[t * P + in_place], g_raw[t] = g_s[t * P + in_place];
    }
    if (DKP <= 128 ? tid < DKP : true) state_keys(tid);
    __syncthreads();
    if (turns) {
        const int c = in_place;
        float lower = 1.0f, product = 1.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            lower *= g_raw[i];
            q_s[i * P + c] *= lower;
            g_s[i * P + c] = k_raw[i] * lower;
        }
        d_half[c] = lower;
#pragma unroll
        for (int j = 15; j >= 0; --j) {
            k_s[j * P + c] = k_raw[j] * product;
            product *= g_raw[j];
        }
        product = 1.0f;
#pragma unroll
        for (int i = 16; i < 32; ++i) {
            product *= g_raw[i];
            q_s[i * P + c] *= product;
            const float key = k_raw[i] * product;
            k_s[i * P + c] = key;
            g_s[i * P + c] = key * lower;
        }
    }
    __syncthreads();

    between_halves<DKP, true>(a_s, bt_s, k_s, q_s);
    __syncthreads();

    const int rg = tid & 7, cg0 = tid >> 3;   // products below: a thread has rows 4 rg .. + 3, columns 4 cg .. + 3
    if (warp == 0) {
        // T, a lane per column: T[i] = beta_i ((i == column) - sum_{j<i} A_ij T[j])
        float t[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            float sums[4] = {i == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < i; j += 4) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + i * TP + j);
                sums[0] -= a.x * t[j];
                if (j + 1 < i) sums[1] -= a.y * t[j + 1];
                if (j + 2 < i) sums[2] -= a.z * t[j + 2];
                if (j + 3 < i) sums[3] -= a.w * t[j + 3];
            }
            t[i] = beta_s[i] * ((sums[0] + sums[1]) + (sums[2] + sums[3]));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(tt_s + lane * TP + i) = make_float4(t[i], t[i + 1], t[i + 2], t[i + 3]);
    }
    __syncthreads();
    // B T at [j][i], in A's place: a thread has rows 4 rg .. + 3 of column j
    const int j = cg0;
    float sums[4] = {};
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
        const float4 b = *reinterpret_cast<const float4*>(bt_s + m * TP + 4 * rg);
        const float t = m >= j ? tt_s[j * TP + m] : 0.0f;
        if (m <= 4 * rg) sums[0] += b.x * t;
        if (m <= 4 * rg + 1) sums[1] += b.y * t;
        if (m <= 4 * rg + 2) sums[2] += b.z * t;
        if (m <= 4 * rg + 3) sums[3] += b.w * t;
    }
    *reinterpret_cast<float4*>(a_s + j * TP + 4 * rg) = make_float4(sums[0], sums[1], sums[2], sums[3]);
    __syncthreads();
    // -W = -T K~ and Q' = Q~ - B T K~, columns one after the other
    for (int cg = cg0; cg < DKP / 4; cg += 32) {
        float w[4][4] = {}, x[4][4] = {};
        triangle_products<true>(w, x, tt_s, a_s, g_s + 4 * cg, P, rg);
        const float4 d = rg >= 4 ? *reinterpret_cast<const float4*>(d_half + 4 * cg) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 own = *reinterpret_cast<const float4*>(q_s + (4 * rg + r) * P + 4 * cg);
            x[r][0] = own.x * d.x - x[r][0], x[r][1] = own.y * d.y - x[r][1], x[r][2] = own.z * d.z - x[r][2], x[r][3] = own.w * d.w - x[r][3];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float* destination = out + (4 * cg + e) * Pack::kRows + 4 * rg;
            *reinterpret_cast<float4*>(destination) = make_float4(-w[0][e], -w[1][e], -w[2][e], -w[3][e]);
            *reinterpret_cast<float4*>(destination + 32) = make_float4(x[0][e], x[1][e], x[2][e], x[3][e]);
        }
    }
    // T V and B T V, 128 columns at a time
    for (int column0 = 0; column0 < dv; column0 += 128) {
        if (column0 > 0) load_values(column0, first_values);
        __syncthreads();   // what lay here has been read
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(v_s + (tid >> 3) * VP + 4 * (tid & 7) + 32 * i) = first_values[i];
        __syncthreads();
        const int column = column0 + 4 * cg0;
        if (column >= slices * kWalkCols) continue;   // (no barrier below but the next turn's, which all threads meet)
        float* destination = v_out + (column / kWalkCols) * Pack::kValues + column % kWalkCols;
        float first[4][4] = {}, second[4][4] = {};
        triangle_products<true>(first, second, tt_s, a_s, v_s + 4 * cg0, VP, rg);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            *reinterpret_cast<float4*>(destination + (4 * rg + r) * kWalkCols) = make_float4(first[r][0], first[r][1], first[r][2], first[r][3]);
            *reinterpret_cast<float4*>(destination + (32 + 4 * rg + r) * kWalkCols) = make_float4(second[r][0], second[r][1], second[r][2], second[r][3]);
        }
    }
}

__device__ __forceinline__ void bulk_load(void* destination, const void* source, uint32_t bytes, uint64_t* barrier) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_address(destination)), "l"(source), "r"(bytes),
                 "r"(smem_address(barrier))
                 : "memory");
}

template <int DKP>
struct WalkShared {
    using Pack = BlockPack<DKP>;
    static constexpr int kStage = Pack::kFloats + Pack::kValues;
    // Three or four blocks on their way at once (two at 256 key channels): a block's copies take longer to arrive than its work takes.
    static constexpr int kStages = DKP <= 32 ? 4 : DKP <= 128 ? 3 : 2;
    static constexpr int kFloats = kStages * kStage + 8 * 64 * kWalkCols /* partial sums */ + DKP * kWalkCols /* S */ + 32 * kWalkCols /* U */;
    static constexpr int kBytes = kFloats * 4;
};

// grid (long portions, heads, ceil(dv / 8)); of each portion the blocks within the window, from the slot's state and back into it.
// A warp owns DKP / 8 key channels: their rows of S stay with it (in registers, and for its own reading in shared memory), it adds up their part of all 64
// rows of the first product, a lane four rows by four columns, and it makes the second product's sums for them, four channels by four
// columns a lane with the tokens shared out over the remaining lanes.  Only the first product's sums and U pass between warps.
template <int DKP>
__global__ void __launch_bounds__(kBlockThreads, DKP <= 64 ? 2 : 1)
recurrent_walk_kernel(const float* __restrict__ pack, const float* __restrict__ vpack, float* __restrict__ state, float* __restrict__ out,
                      const int* __restrict__ long_table, const int* __restrict__ segment_start, const int* __restrict__ segment_length,
                      const int* __restrict__ segment_slot, int heads, int dk, int dv, int num_slots, int* status, int window, int window_blocks) {
    wait_for_previous_kernel();
    allow_next_kernel();
    using Pack = BlockPack<DKP>;
    using Shared = WalkShared<DKP>;
    constexpr int kStages = Shared::kStages;
    constexpr int kChannels = DKP / 8;                  // of a warp
    constexpr int kTokenLanes = 64 / kChannels;         // lanes that share out a block's tokens in the second product
    constexpr int kOwn = kWalkCols * kChannels / 32;    // elements of S a lane: after the sums over the lanes of a token, 16 / kTokenLanes of a tile of 4 x 4
    static_assert(kTokenLanes * (kChannels / 4) == 16 && kOwn * kTokenLanes == 16, "a warp's lanes are its token lanes x groups of four channels x two halves of the columns");
    extern __shared__ __align__(128) float walk_memory[];
    __shared__ uint64_t full[kStages];
    __shared__ int failed;
    float* part_s = walk_memory + kStages * Shared::kStage;   // [warp][64 rows][8 columns]
    float* state_s = part_s + 8 * 64 * kWalkCols;             // [DKP][8]
    float* u_s = state_s + DKP * kWalkCols;                   // [32][8]
    const int portion = long_table[3 * blockIdx.x], offset = blocks_before(long_table, segment_length, blockIdx.x) - window;   // of its blocks' numbers
    const int head = blockIdx.y, slice = blockIdx.z, column0 = slice * kWalkCols, slices = gridDim.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slot = segment_slot[portion];
    if (slot < 0 || slot >= num_slots) {
        if (tid == 0) report_error(status, kBadSlot);
        return;
    }
    const int start = segment_start[portion], length = segment_length[portion];
    const int first = max(0, -offset), blocks = min((length + kBlockTokens - 1) / kBlockTokens, window_blocks - offset) - first;
    if (blocks <= 0) return;
    auto load = [&](int block) {   // one thread; block counts from the portion's first within the window
        float* stage = walk_memory + (block % kStages) * Shared::kStage;
        uint64_t* barrier = &full[block % kStages];
        const size_t index = static_cast<size_t>(offset + first + block) * heads + head;
        barrier_expect(barrier, Shared::kStage * 4);
        bulk_load(stage, pack + index * Pack::kFloats, Pack::kFloats * 4, barrier);
        bulk_load(stage + Pack::kFloats, vpack + (index * slices + slice) * Pack::kValues, Pack::kValues * 4, barrier);
    };
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) barrier_init(&full[s], 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int block = 0; block < min(kStages, blocks); ++block) load(block);
    }
    // The lane's elements of S: of the tile of channels channel0 .. + 3 and columns 4 column_half .. + 3 those that the sums over the token lanes leave
    // here, kOwn neighbours in the order of (channel, column).
    const int token_lane = lane / (32 / kTokenLanes), group = (lane >> 1) % (kChannels / 4), column_half = lane & 1;
    const int channel0 = warp * kChannels + 4 * group;
    const int own_row = channel0 + token_lane * kOwn / 4, own_column = 4 * column_half + token_lane * kOwn % 4;   // kOwn > 4: two whole rows
    float* slot_state = state + (static_cast<size_t>(slot) * heads + head) * dk * dv;
    float S[kOwn];
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        const int row = own_row + (kOwn > 4 ? i / 4 : 0), column = own_column + (kOwn > 4 ? i % 4 : i);
        S[i] = row < dk && column0 + column < dv ? slot_state[static_cast<size_t>(row) * dv + column0 + column] : 0.0f;
        state_s[row * kWalkCols + column] = S[i];
    }
    __syncthreads();
    for (int block = 0; block < blocks; ++block) {
        const float* stage = walk_memory + (block % kStages) * Shared::kStage;
        if (!barrier_wait_busy(&full[block % kStages], (block / kStages) & 1)) atomicExch(&failed, 1);
        {
            // the warp's channels' part of [U ; O]: rows 4 (lane & 15) .. + 3 by columns 4 (lane >> 4) .. + 3
            const float* matrix = stage + warp * kChannels * Pack::kRows + 4 * (lane & 15);
            const float* own = state_s + warp * kChannels * kWalkCols + 4 * (lane >> 4);
            uint64_t acc[4][2] = {};
#pragma unroll
            for (int c = 0; c < kChannels; ++c) {
                const float4 m = *reinterpret_cast<const float4*>(matrix + c * Pack::kRows);
                const ulonglong2 columns = *reinterpret_cast<const ulonglong2*>(own + c * kWalkCols);
                const float rows[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint64_t row = pack2(rows[r], rows[r]);
                    acc[r][0] = fma2(row, columns.x, acc[r][0]);
                    acc[r][1] = fma2(row, columns.y, acc[r][1]);
                }
            }
            // pieces of 16 bytes, two a row; the eight of four rows in an order of their own, so that eight lanes meet no bank twice
            ulonglong2* part = reinterpret_cast<ulonglong2*>(part_s) + warp * 128 + 8 * (lane & 15);
#pragma unroll
            for (int r = 0; r < 4; ++r) part[(2 * r + (lane >> 4)) ^ (lane & 7)] = make_ulonglong2(acc[r][0], acc[r][1]);
        }
        __syncthreads();
        if (failed) {
            if (tid == 0) report_error(status, kWaitTimeout);
            for (int spin = 0; spin < 2000; ++spin) __nanosleep(1000);   // copies in flight land
            return;
        }
        // (every warp is past the block before: its stage may be filled again)
        if (tid == 0 && block > 0 && block - 1 + kStages < blocks) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            load(block - 1 + kStages);
        }
        const float* values = stage + Pack::kFloats;
        const int t0 = kBlockTokens * (first + block), n = min(kBlockTokens, length - t0);
        {
            // two sums a thread, the warps' parts in their order
            const int row = tid >> 2, column = 2 * (tid & 3), piece = 8 * (row >> 2) + ((2 * (row & 3) + (column >> 2)) ^ ((row >> 2) & 7));
            const float* part = part_s + 4 * piece + (column & 3);
            float2 sum = *reinterpret_cast<const float2*>(part);
#pragma unroll
            for (int w = 1; w < 8; ++w) {
                const float2 other = *reinterpret_cast<const float2*>(part + w * 64 * kWalkCols);
                sum.x += other.x, sum.y += other.y;
            }
            const float2 own = *reinterpret_cast<const float2*>(values + row * kWalkCols + column);
            sum.x += own.x, sum.y += own.y;
            if (row < 32) {
                *reinterpret_cast<float2*>(u_s + row * kWalkCols + column) = sum;
            } else if (row - 32 < n) {
                float* destination = out + (static_cast<size_t>(start + t0 + row - 32) * heads + head) * dv + column0 + column;
                if (column0 + column < dv) destination[0] = sum.x;
                if (column0 + column + 1 < dv) destination[1] = sum.y;
            }
        }
        __syncthreads();
        {
            // S <- diag(D_end) S + K^T U: a tile of 4 x 4 over the lane's tokens, then over the token lanes
            const float* k_hat = stage + Pack::kMatrix;
            float tile[16] = {};
#pragma unroll
            for (int i = 0; i < 32 / kTokenLanes; ++i) {
                const int t = i * kTokenLanes + token_lane;
                const float4 key = *reinterpret_cast<const float4*>(k_hat + t * DKP + channel0), u = *reinterpret_cast<const float4*>(u_s + t * kWalkCols + 4 * column_half);
                const float keys[4] = {key.x, key.y, key.z, key.w}, us[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int e = 0; e < 4; ++e) tile[4 * r + e] += keys[r] * us[e];
            }
#pragma unroll
            for (int half = 8, bit = 16; half >= kOwn; half >>= 1, bit >>= 1) {   // (the token lanes are the upper bits of the lane)
                const bool upper = (lane & bit) != 0;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const float keep = upper ? tile[i + half] : tile[i], give = upper ? tile[i] : tile[i + half];
                    tile[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            }
            const float* decays = k_hat + 32 * DKP + own_row;
#pragma unroll
            for (int i = 0; i < kOwn; ++i) {
                S[i] = fmaf(decays[kOwn > 4 ? i / 4 : 0], S[i], tile[i]);
                state_s[(own_row + (kOwn > 4 ? i / 4 : 0)) * kWalkCols + own_column + (kOwn > 4 ? i % 4 : i)] = S[i];
            }
            __syncwarp();   // S is this warp's alone
        }
    }
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        const int row = own_row + (kOwn > 4 ? i / 4 : 0), column = own_column + (kOwn > 4 ? i % 4 : i);
        if (row < dk && column0 + column < dv) slot_state[static_cast<size_t>(row) * dv + column0 + column] = S[i];
    }
}

// ---------------------------------------------------------------------------------------------------- no correction
// Without the delta rule's correction u_j = v_j, and a block turns the state into diag(D_end) S + K^T V whatever S is: that sum, and what a
// block's own tokens give its read-outs (B V), are made side by side, a short pass puts the states in order, element by element,
// and the read-outs get Q~ S, again side by side.

// grid and arguments as recurrent_prepare_kernel's; sums [block][head][dk][dv], decays [block][head][dk]; out [tokens, heads, dv] = B V.
template <int DKP>
__global__ void __launch_bounds__(kBlockThreads, DKP <= 128 ? 3 : 1)
linear_prepare_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ g, const float* __restrict__ v, float* __restrict__ sums,
                      float* __restrict__ decays, float* __restrict__ out, const int* __restrict__ long_table, int long_portions, const int* __restrict__ segment_start,
                const int* __restrict__ segment_length, int heads,
                      int groups, int dk, int dv, int window) {
    wait_for_previous_kernel();
    allow_next_kernel();
    constexpr int P = DKP + 4, VP = 132;
    extern __shared__ __align__(16) float prepare_memory[];
    float* k_s = prepare_memory;   // keys; then as between_halves wants them
    float* q_s = k_s + 32 * P;     // queries; then as between_halves wants them
    float* g_s = q_s + 32 * P;     // decays; then K^
    float* v_s = g_s + 32 * P;     // values, 128 columns at a time
    float* bt_s = v_s + 32 * VP;
    const PortionBlock here = find_block(long_table, segment_length, long_portions, window + static_cast<int>(blockIdx.x));
    if (here.block < 0) return;
    const int first = kBlockTokens * here.block, n = min(kBlockTokens, segment_length[here.portion] - first);
    const int start = segment_start[here.portion] + first, head = blockIdx.y, group = head / (heads / groups);
    const int tid = threadIdx.x;
    const size_t block_head = static_cast<size_t>(blockIdx.x) * heads + head;
    load_block<DKP>(k_s, q_s, g_s, q, k, g, start, n, head, group, heads, groups, dk);
    __syncthreads();
    within_halves<DKP, false>(nullptr, bt_s, k_s, q_s, g_s);
    __syncthreads();
    if (tid < DKP) {
        const int c = tid;
        float product = 1.0f, k_raw[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) k_raw[i] = k_s[i * P + c];
        // K^ in the decays' place and, in the upper half, the queries times the decays from its start; then the lower half's keys
        float upper = 1.0f;
#pragma unroll
        for (int i = 16; i < 32; ++i) {
            upper *= g_s[i * P + c];
            q_s[i * P + c] *= upper;
        }
        float to_middle = 1.0f;
#pragma unroll
        for (int j = 31; j >= 0; --j) {
            const float decay = g_s[j * P + c];
            if (j < 16) {
                k_s[j * P + c] = k_raw[j] * to_middle;
                to_middle *= decay;
            }
            g_s[j * P + c] = (j < 16 ? k_raw[j] : k_s[j * P + c]) * product;
            product *= decay;
        }
        if (c < dk) decays[block_head * dk + c] = product;
    }
    __syncthreads();
    between_halves<DKP, false>(nullptr, bt_s, k_s, q_s);
    const int rg = tid & 7, cg = tid >> 3;       // of B V: rows 4 rg .. + 3, columns 4 cg .. + 3
    const int kg = tid >> 4, wide = tid & 15;    // of K^T V: channels 4 kg .. + 3 (and every 64th), columns 8 wide .. + 7
    for (int column0 = 0; column0 < dv; column0 += 128) {
        __syncthreads();   // B is whole; the columns before these have been read
#pragma unroll 16
        for (int index = tid; index < 32 * 128; index += kBlockThreads) {
            const int t = index >> 7, c = index & 127;
            v_s[t * VP + c] = t < n && column0 + c < dv ? v[(static_cast<size_t>(start + t) * heads + head) * dv + column0 + c] : 0.0f;
        }
        __syncthreads();
        if (column0 + 4 * cg < dv) {
            float unused[4][4], acc[4][4] = {};
            triangle_products<false>(unused, acc, nullptr, bt_s, v_s + 4 * cg, VP, rg);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float* destination = out + (static_cast<size_t>(start + 4 * rg + r) * heads + head) * dv + column0 + 4 * cg;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * rg + r < n && column0 + 4 * cg + e < dv) destination[e] = acc[r][e];
            }
        }
        for (int c = 4 * kg; c < dk; c += 64) {
            float acc[4][8] = {};
#pragma unroll 8
            for (int t = 0; t < 32; ++t) {
                float key[4], value[8];
                load_floats<4>(g_s + t * P + c, key);
                load_floats<8>(v_s + t * VP + 8 * wide, value);
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[r][e] += key[r] * value[e];
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (c + r >= dk) continue;
                const int column = column0 + 8 * wide;
                float* destination = sums + (block_head * dk + c + r) * dv + column;
                if (dv % 4 == 0) {
                    if (column < dv) *reinterpret_cast<float4*>(destination) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
                    if (column + 4 < dv) *reinterpret_cast<float4*>(destination + 4) = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (column + e < dv) destination[e] = acc[r][e];
                }
            }
        }
    }
}

// grid (long portions, heads, pieces of dk * dv): within the window every block's sum becomes the state that the block starts from, the portion's slot the
// state after the last.  One thread an element, eight blocks' loads on their way at a time.
__global__ void __launch_bounds__(kBlockThreads)
linear_states_kernel(float* __restrict__ sums, const float* __restrict__ decays, float* __restrict__ state, const int* __restrict__ long_table,
                     const int* __restrict__ segment_length, const int* __restrict__ segment_slot, int heads, int dk, int dv, int num_slots, int* status,
                     int window, int window_blocks) {
    wait_for_previous_kernel();
    allow_next_kernel();
    const int portion = long_table[3 * blockIdx.x], offset = blocks_before(long_table, segment_length, blockIdx.x) - window;   // of its blocks' numbers
    const int first = max(0, -offset), blocks = min((segment_length[portion] + kBlockTokens - 1) / kBlockTokens, window_blocks - offset) - first;
    const int head = blockIdx.y, element = blockIdx.z * kBlockThreads + threadIdx.x, elements = dk * dv, slot = segment_slot[portion];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0) report_error(status, kBadSlot);
        return;
    }
    if (element >= elements || blocks <= 0) return;
    float* mine = state + (static_cast<size_t>(slot) * heads + head) * elements + element;
    float s = *mine;
    float* block_sums = sums + (static_cast<size_t>(offset + first) * heads + head) * elements + element;
    const float* block_decays = decays + (static_cast<size_t>(offset + first) * heads + head) * dk + element / dv;
    const size_t sum_step = static_cast<size_t>(heads) * elements, decay_step = static_cast<size_t>(heads) * dk;
    for (int b0 = 0; b0 < blocks; b0 += 8) {
        float sum[8], decay[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (b0 + u < blocks) sum[u] = block_sums[(b0 + u) * sum_step], decay[u] = block_decays[(b0 + u) * decay_step];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (b0 + u < blocks) {
                block_sums[(b0 + u) * sum_step] = s;
                s = decay[u] * s + sum[u];
            }
        }
    }
    *mine = s;
}

constexpr int kReadChannels = 64, kReadPitch = 132;   // the read-out takes S in pieces of 64 channels by 128 columns
template <int DKP>
struct ReadShared {
    static constexpr int kPiece = 2 * 32 * (DKP + 4) > kReadChannels * kReadPitch ? 2 * 32 * (DKP + 4) : kReadChannels * kReadPitch;
    static constexpr int kBytes = (kPiece + DKP * kTrianglePitch) * 4;
};

// grid (blocks, heads): out[t] += (D_t q_t)^T S for the block's tokens, S the state that it starts from.  Sums of 16 channels are added up
// by themselves, as the split sums of the token-by-token kernel are.  VECTOR: dv is a multiple of 4.
template <int DKP, bool VECTOR>
__global__ void __launch_bounds__(kBlockThreads)
linear_read_kernel(const float* __restrict__ q, const float* __restrict__ g, const float* __restrict__ states, float* __restrict__ out, const int* __restrict__ long_table, int long_portions, const int* __restrict__ segment_start,
                const int* __restrict__ segment_length, int heads, int groups, int dk, int dv, int window) {
    wait_for_previous_kernel();
    allow_next_kernel();
    constexpr int P = DKP + 4;
    extern __shared__ __align__(16) float prepare_memory[];
    float* q_s = prepare_memory;
    float* g_s = q_s + 32 * P;
    float* piece_s = prepare_memory;
    float* qt_s = prepare_memory + ReadShared<DKP>::kPiece;   // Q~ at [channel][token], rows of kTrianglePitch
    const PortionBlock here = find_block(long_table, segment_length, long_portions, window + static_cast<int>(blockIdx.x));
    if (here.block < 0) return;
    const int first = kBlockTokens * here.block, n = min(kBlockTokens, segment_length[here.portion] - first);
    const int start = segment_start[here.portion] + first, head = blockIdx.y, group = head / (heads / groups), tid = threadIdx.x;
#pragma unroll 8
    for (int index = tid; index < 32 * DKP; index += kBlockThreads) {
        const int t = index / DKP, c = index % DKP;
        const bool real = t < n && c < dk;
        q_s[t * P + c] = real ? q[(static_cast<size_t>(start + t) * groups + group) * dk + c] : 0.0f;
        g_s[t * P + c] = real ? g[(static_cast<size_t>(start + t) * heads + head) * dk + c] : 1.0f;
    }
    __syncthreads();
    if (tid < DKP) {
        float product = 1.0f, query[32];
#pragma unroll
        for (int t = 0; t < 32; ++t) {
            product *= g_s[t * P + tid];
            query[t] = q_s[t * P + tid] * product;
        }
#pragma unroll
        for (int t = 0; t < 32; t += 4) *reinterpret_cast<float4*>(qt_s + tid * kTrianglePitch + t) = make_float4(query[t], query[t + 1], query[t + 2], query[t + 3]);
    }
    __syncthreads();
    const float* S = states + (static_cast<size_t>(blockIdx.x) * heads + head) * dk * dv;
    const int rg = tid & 7, cg = tid >> 3;
    for (int column0 = 0; column0 < dv; column0 += 128) {
        float total[4][4] = {};
        for (int c0 = 0; c0 < dk; c0 += kReadChannels) {
            // a piece of S where the queries and decays were: with its loads inside the products below a block took 30 us
#pragma unroll 8
            for (int index = tid; index < kReadChannels * 32; index += kBlockThreads) {
                const int c = index >> 5, e = 4 * (index & 31);
                const bool real = c0 + c < dk && column0 + e < dv;
                const float* source = S + static_cast<size_t>(c0 + c) * dv + column0 + e;
                float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if constexpr (VECTOR) {
                    if (real) x = *reinterpret_cast<const float4*>(source);
                } else if (real) {
                    x.x = source[0];
                    if (column0 + e + 1 < dv) x.y = source[1];
                    if (column0 + e + 2 < dv) x.z = source[2];
                    if (column0 + e + 3 < dv) x.w = source[3];
                }
                *reinterpret_cast<float4*>(piece_s + c * kReadPitch + e) = x;
            }
            __syncthreads();
            const int channels = min(kReadChannels, DKP - c0);   // (those past dk are zeros on both sides)
            for (int c1 = 0; c1 < channels; c1 += 16) {
                float acc[4][4] = {};
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    float tokens[4], row[4];
                    load_floats<4>(qt_s + (c0 + c1 + c) * kTrianglePitch + 4 * rg, tokens);
                    load_floats<4>(piece_s + (c1 + c) * kReadPitch + 4 * cg, row);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[r][e] += tokens[r] * row[e];
                }
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int e = 0; e < 4; ++e) total[r][e] += acc[r][e];
            }
            __syncthreads();
        }
        const int column = column0 + 4 * cg;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (4 * rg + r >= n || column >= dv) continue;
            float* destination = out + (static_cast<size_t>(start + 4 * rg + r) * heads + head) * dv + column;
            if constexpr (VECTOR) {
                const float4 own = *reinterpret_cast<const float4*>(destination);
                *reinterpret_cast<float4*>(destination) = make_float4(own.x + total[r][0], own.y + total[r][1], own.z + total[r][2], own.w + total[r][3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (column + e < dv) destination[e] += total[r][e];
            }
        }
    }
}

// beta null: `pack` holds the blocks' sums, then their decays; `vpack` is not used.
template <int DKP>
int launch_recurrent_blocks(const float* q, const float* k, const float* g, const float* v, const float* beta, float* pack, float* vpack, float* state, float* out,
                            int most_blocks, int window_blocks, const int* long_table, int long_portions, const int* segment_start,
                            const int* segment_length, const int* segment_slot, int heads, int groups, int dk, int dv, int num_slots, int* status, cudaStream_t stream) {
    const dim3 blocks(window_blocks, heads), threads(kBlockThreads);
    // Which of them start early (see launch_early_if), as measured with launches in a stream and in a recorded graph.  The walk, except where two CTAs share a multiprocessor and
    // there are no more CTAs than multiprocessors: the delta rule over 4,096 tokens of 64 key channels 343 us with an early start and 271 without, 128 channels 369 and
    // 371.  Linear attention's first and last kernel with more blocks than two to a multiprocessor (1,500 tokens of 128 key channels 133 and 137 us; 1,000 116 and 105,
    // 300 90 and 75), the last with 64 key channels also where it has few (500 tokens 58.7 and 60.4; 850 74.7 and 72.3, the first without in all four).
    const int sms = multiprocessor_count(), grid = window_blocks * heads;
    cudaError_t error = cudaSuccess;
    if (beta != nullptr) {
        static OncePerDevice prepared, walked;
        auto prepare = recurrent_prepare_kernel<DKP>;
        auto walk = recurrent_walk_kernel<DKP>;
        if (allow_shared_memory(prepared, prepare, PrepareShared<DKP>::kBytes) != cudaSuccess) return static_cast<int>(cudaGetLastError());
        if (allow_shared_memory(walked, walk, WalkShared<DKP>::kBytes) != cudaSuccess) return static_cast<int>(cudaGetLastError());
        const bool walk_early = DKP > 64 || long_portions * heads * ((dv + kWalkCols - 1) / kWalkCols) > sms;
        for (int window = 0; window < most_blocks && error == cudaSuccess; window += window_blocks) {
            error = launch_overlapped(prepare, blocks, threads, PrepareShared<DKP>::kBytes, stream, q, k, g, v, beta, pack, vpack, long_table, long_portions, segment_start,
                                      segment_length, heads, groups, dk, dv, window);
            if (error == cudaSuccess)
                error = launch_early_if(walk_early, walk, dim3(long_portions, heads, (dv + kWalkCols - 1) / kWalkCols), threads, WalkShared<DKP>::kBytes, stream, pack, vpack, state,
                                        out, long_table, segment_start, segment_length, segment_slot, heads, dk, dv, num_slots, status, window, window_blocks);
        }
        return static_cast<int>(error != cudaSuccess ? error : cudaGetLastError());
    }
    static OncePerDevice prepared, read, read_any;
    auto prepare = linear_prepare_kernel<DKP>;
    auto read_out = dv % 4 == 0 ? linear_read_kernel<DKP, true> : linear_read_kernel<DKP, false>;
    constexpr int prepare_bytes = (3 * 32 * (DKP + 4) + 32 * 132 + 32 * kTrianglePitch) * 4, read_bytes = ReadShared<DKP>::kBytes;
    if (allow_shared_memory(prepared, prepare, prepare_bytes) != cudaSuccess) return static_cast<int>(cudaGetLastError());
    if (allow_shared_memory(dv % 4 == 0 ? read : read_any, read_out, read_bytes) != cudaSuccess) return static_cast<int>(cudaGetLastError());
    float* decays = pack + static_cast<size_t>(window_blocks) * heads * dk * dv;
    const bool prepare_early = grid > 2 * sms, read_early = grid > 2 * sms || (DKP <= 64 && 3 * grid <= 4 * sms);
    for (int window = 0; window < most_blocks && error == cudaSuccess; window += window_blocks) {
        error = launch_early_if(prepare_early, prepare, blocks, threads, prepare_bytes, stream, q, k, g, v, pack, decays, out, long_table, long_portions, segment_start, segment_length,
                                heads, groups, dk, dv, window);
        if (error == cudaSuccess)
            error = launch_overlapped(linear_states_kernel, dim3(long_portions, heads, (dk * dv + kBlockThreads - 1) / kBlockThreads), threads, 0, stream, pack, decays, state,
                                      long_table, segment_length, segment_slot, heads, dk, dv, num_slots, status, window, window_blocks);
        if (error == cudaSuccess)
            error = launch_early_if(read_early, read_out, blocks, threads, read_bytes, stream, q, g, pack, out, long_table, long_portions, segment_start, segment_length, heads, groups,
                                    dk, dv, window);
    }
    return static_cast<int>(error != cudaSuccess ? error : cudaGetLastError());
}

}  // namespace lb

extern "C" {

// Floats of `pack` and of `vpack` that one block of 32 tokens of one head needs (0: key sizes that the blocks do not take).
int lb_recurrent_pack_floats(int dk, int dv, int delta) {
    if (dk < 1 || dk > 256) return 0;
    if (!delta) return dk * dv + dk;
    return dk <= 32 ? lb::BlockPack<32>::kFloats : dk <= 64 ? lb::BlockPack<64>::kFloats : dk <= 128 ? lb::BlockPack<128>::kFloats : lb::BlockPack<256>::kFloats;
}
int lb_recurrent_value_floats(int dv, int delta) { return delta ? (dv + lb::kWalkCols - 1) / lb::kWalkCols * 64 * lb::kWalkCols : 0; }

// The long portions of `long_table`, block by block, from and into their state slots.  `most_blocks`: no fewer than their
// blocks of 32 tokens together; they are taken `window_blocks` at a time, for which `pack` and `vpack` have room in every head (the
// states pass from one window to the next through their slots, in 32 bits as they are: the results are the same).  beta null: no delta rule.
int lb_recurrent_blocks(const float* q, const float* k, const float* g, const float* v, const float* beta, float* pack, float* vpack, float* state, float* out,
                        int most_blocks, int window_blocks, const int* long_table, int long_portions, const int* segment_start,
                        const int* segment_length, const int* segment_slot, int heads, int groups, int dk, int dv, int num_slots, int* status, cudaStream_t stream) {
    if (long_portions == 0 || most_blocks == 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads % groups != 0 || window_blocks < 1) return -2;
    auto launch = dk <= 32 ? lb::launch_recurrent_blocks<32> : dk <= 64 ? lb::launch_recurrent_blocks<64> : dk <= 128 ? lb::launch_recurrent_blocks<128> : lb::launch_recurrent_blocks<256>;
    return launch(q, k, g, v, beta, pack, vpack, state, out, most_blocks, window_blocks, long_table, long_portions, segment_start, segment_length, segment_slot,
                  heads, groups, dk, dv, num_slots, status, stream);
}

}  // extern "C"
