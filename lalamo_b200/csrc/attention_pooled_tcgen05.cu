// Sigmoid-weighted attention with pooled blocks (see attention_pooled.cu) for portions of prompts on the fifth-generation tensor cores.
//
// A CTA takes 128 query rows = a tile's consecutive tokens x up to four query heads of one K/V head.  Rows of the cache come 64 at a time by TMA
// through four stages, keys and values in panels of their own, in the order of the kernel on mma.sync: pooled blocks from block 0 on, then positions
// from the multiple of 64 at or below the tile's first visible one.  Scores (two tiles), the weights over the scores they came from and the sums live
// in tensor memory; the values are read as an operand that is contiguous along its columns.
//   warps 0-7  two threads a row, 32 scores each: there is no denominator, so that nothing is exchanged and nothing rescaled
//   warp 8     allocates tensor memory; one lane issues O += P V of a tile, then S = Q K^T of the tile after next
//   warp 9     asks for the boxes of the positions, and copies the pooled blocks
// What bounds it: the weighing warps' dependent instructions, with the transcendental unit as the busiest pipe (45 % of the time on average, issue slots 54 %).  Two
// CTAs share a multiprocessor, so that every warp finds scores to weigh.  Written out a weight takes four
// of its operations, tanh(x) = 1 - 2 / (1 + 2^(2 x log2 e)) and 1 / (1 + 2^-y); here a polynomial stands for the tanh where all of a thread's scores
// are within half of the cap (else it is written out), and two weights share a reciprocal: three operations for two weights.  Measured, 16 heads over 4, a
// window of 1,024 and blocks of 8: a prompt of 3,000 48 us (mma.sync 118 and 14 to add up two shares; 65 with the tiles of one head after the other's, which
// left multiprocessors idle at the end, and one score an instruction), 2,048 37 us (93), 200 14 us (24).  A multiprocessor takes 1.1 us for 64 rows.
// Every wait is bounded and reports through the status word.
#include "tcgen05.cuh"

#include <type_traits>

namespace lb {

constexpr int kPtRows = 128, kPtKeys = 64, kPtThreads = 320, kPtStages = 4;
constexpr int kPtPanel = kPtKeys * 128;           // 64 rows of 64 channels
constexpr int kPtStage = 2 * kPtPanel;            // keys, values
constexpr float kPtMostX = 0.5f;                  // of a score over the cap, for the polynomial
constexpr float kPtMostExponent = 60.0f;          // of 2^y in a weight's 1 / (1 + 2^y) up to which two weights share a reciprocal: their denominators then have a product

struct PooledTcParams {
    const __nv_bfloat16* pooled_pages;
    __nv_bfloat16* out;
    float* partial;          // shares > 1: [share][row][head][64], 32-bit sums not yet turned back
    const int* tiles;        // [num_tiles][2]: first row, count
    const int* positions;
    const int* token_segment;
    const int* block_table;
    const int* pool_table;
    const float* head_bias;  // or null
    const float* v_freq;     // or null
    int* status;
    int page_size, num_pages, max_blocks;
    int pool_rows, pool_pages, pool_max_blocks;
    int heads, groups, head_block, tile_tokens, window, pool, v_interleaved, total_rows;
    float scale, cap;
};

__device__ __forceinline__ void pt_load_32(uint32_t address, float (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]),
          "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]),
          "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(address)
        : "memory");
}

__device__ __forceinline__ float pt_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float pt_reciprocal(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The weights of a row's scores: 1 / (1 + 2^y), y = -(cap tanh(s scale / cap) + bias) log2 e.
struct PooledWeights {
    float slope, offset;                // y = s q((s scale / cap)^2) slope + offset with tanh(x) = x q(x^2)
    float q1, q2, q3, q4;               // the polynomial's coefficients, for s^2
    float most;                         // |s| up to which it stands for the tanh (negative: never)
    float to_exponent, wide_slope, wide_offset;   // written out: r = 1 / (1 + 2^(s to_exponent)), y = r wide_slope + wide_offset
    __device__ __forceinline__ PooledWeights(float scale, float cap, float bias) {
        constexpr float kLog2e = 1.4426950408889634f;
        slope = -scale * kLog2e;
        offset = -bias * kLog2e;
        const float a = cap > 0.0f ? scale / cap : 0.0f, a2 = a * a;
        // least largest relative error (1.5e-8) of x q(x^2) against tanh(x) on |x| <= 1/2
        q1 = -0.33333148378404964f * a2;
        q2 = 0.1332598730088283f * a2 * a2;
        q3 = -0.053052951160387156f * a2 * a2 * a2;
        q4 = 0.017256992378932703f * a2 * a2 * a2 * a2;
        // (tanh(1/2) is 0.4622: with its exponents beyond the bound, a row's weights are written out)
        most = cap > 0.0f && (0.4622f * cap + fabsf(bias)) * kLog2e <= kPtMostExponent ? kPtMostX / fabsf(a) : -1.0f;
        to_exponent = 2.0f * a * kLog2e;
        wide_slope = 2.0f * cap * kLog2e;
        wide_offset = -(cap + bias) * kLog2e;
    }
    // whether no y is beyond kPtMostExponent, without a cap, for scores of at most `top`
    __device__ __forceinline__ bool near(float top) const { return fmaf(top, fabsf(slope), fabsf(offset)) <= kPtMostExponent; }
    // -log2 of what a weight's denominator adds to one, of two neighbours' scores; two 32-bit values an instruction where the form allows
    template <int FORM>   // 0: no cap, 1: the polynomial, 2: written out
    __device__ __forceinline__ uint64_t exponents(uint64_t s) const {
        const uint64_t slopes = pack2(slope, slope), offsets = pack2(offset, offset);
        if constexpr (FORM == 0) return fma2(s, slopes, offsets);
        else if constexpr (FORM == 1) {
            const uint64_t u = mul2(s, s);
            uint64_t q = fma2(pack2(q4, q4), u, pack2(q3, q3));
            q = fma2(q, u, pack2(q2, q2));
            q = fma2(q, u, pack2(q1, q1));
            q = fma2(q, u, pack2(1.0f, 1.0f));
            return fma2(q, mul2(s, slopes), offsets);
        } else {
            float s0, s1;
            unpack2(s, s0, s1);
            return pack2(fmaf(pt_reciprocal(1.0f + pt_exp2(s0 * to_exponent)), wide_slope, wide_offset), fmaf(pt_reciprocal(1.0f + pt_exp2(s1 * to_exponent)), wide_slope, wide_offset));
        }
    }
    // the two weights, rounded; NEAR: both exponents are within kPtMostExponent.  Beyond it each weight has a reciprocal of its own, down to the least
    // normal number (2^-126), as in the kernels of single tokens
    template <int FORM, bool NEAR>
    __device__ __forceinline__ uint32_t pair(float s0, float s1) const {
        float y0, y1, d0, d1, w0, w1;
        unpack2(exponents<FORM>(pack2(s0, s1)), y0, y1);
        unpack2(add2(pack2(pt_exp2(y0), pt_exp2(y1)), pack2(1.0f, 1.0f)), d0, d1);
        if constexpr (NEAR) {
            const float r = pt_reciprocal(d0 * d1);
            unpack2(mul2(pack2(d1, d0), pack2(r, r)), w0, w1);
        } else {
            w0 = pt_reciprocal(d0), w1 = pt_reciprocal(d1);
        }
        const __nv_bfloat162 weights = __floats2bfloat162_rn(w0, w1);
        return *reinterpret_cast<const uint32_t*>(&weights);
    }
};

// grid (tiles * groups * ceil(heads per group / head_block), shares), 320 threads: the tiles with most rows, of all heads, start first.
__global__ void __launch_bounds__(kPtThreads, 2)
pooled_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_16, const __grid_constant__ CUtensorMap map_32,
                                const PooledTcParams p) {
    extern __shared__ unsigned char raw_shared[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_shared) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* stages = base;
    unsigned char* q_tile = stages + kPtStages * kPtStage;
    uint64_t* barriers = reinterpret_cast<uint64_t*>(q_tile + kPtRows * 128);
    uint64_t* q_full = barriers;
    uint64_t* full = barriers + 1;                     // [kPtStages]
    uint64_t* free_again = full + kPtStages;           // [kPtStages]
    uint64_t* s_full = free_again + kPtStages;         // [2]
    uint64_t* p_full = s_full + 2;                     // [2]
    uint64_t* done = p_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    float2* turns = reinterpret_cast<float2*>(barriers + 32);   // [warp][token of the warp's rows][16 pairs of channels]: cosine, sine
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per_group = p.heads / p.groups, head_blocks = (per_group + p.head_block - 1) / p.head_block;
    const int tile_index = (gridDim.x - 1 - blockIdx.x) / (p.groups * head_blocks), unit = blockIdx.x % (p.groups * head_blocks);   // (a prompt's last tiles)
    const int group = unit / head_blocks, first_head = (unit % head_blocks) * p.head_block;   // in the group
    const int first_row = p.tiles[2 * tile_index], count = min(p.tile_tokens, p.tiles[2 * tile_index + 1]);
    const int segment = p.token_segment[first_row], p_first = p.positions[first_row], p_last = p_first + count - 1;
    const int blocks_seen = p.pool > 0 ? max(0, p_last - p.window + 1) / p.pool : 0;    // by the tile's last token
    const int first_key = max(0, p_first - p.window + 1);
    const int pooled_tiles = (blocks_seen + kPtKeys - 1) / kPtKeys;
    const int first_token_tile = first_key / kPtKeys, all_tiles = pooled_tiles + p_last / kPtKeys - first_token_tile + 1;
    const int tile_begin = static_cast<int>(static_cast<long long>(all_tiles) * blockIdx.y / gridDim.y);
    const int tiles = static_cast<int>(static_cast<long long>(all_tiles) * (blockIdx.y + 1) / gridDim.y) - tile_begin;
    // the CTA's tile-th tile: pooled blocks or positions, the first of them, and which of them some query of the tile sees
    struct Rows {
        bool pooled;
        int base, low, high;
    };
    auto rows_of = [&](int tile) {
        const int listed = tile_begin + tile;
        const bool pooled = listed < pooled_tiles;
        return Rows{pooled, pooled ? listed * kPtKeys : (first_token_tile + listed - pooled_tiles) * kPtKeys, pooled ? 0 : first_key, pooled ? blocks_seen - 1 : p_last};
    };

    if (threadIdx.x == 0) {
        barrier_init(q_full, 1);
        for (int s = 0; s < kPtStages; ++s) {
            barrier_init(&full[s], 1);
            barrier_init(&free_again[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            barrier_init(&s_full[s], 1);
            barrier_init(&p_full[s], 8);   // one arrival per weighing warp
        }
        barrier_init(done, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(tmem_slot)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    wait_for_previous_kernel();   // launched to start early: the queries, the newest rows and blocks are there from here on
    allow_next_kernel();
    const uint32_t tmem_output = *tmem_slot, tmem_scores = tmem_output + 64;   // two tiles of 64 columns

    if (warp == 9) {
        if (lane == 0) {
            barrier_expect(q_full, static_cast<uint32_t>(p.tile_tokens * p.head_block * 128));
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_address(q_tile)), "l"(&map_q),
                         "r"(smem_address(q_full)), "r"(0), "r"(group * per_group + first_head), "r"(first_row)
                         : "memory");
        }
        // Tiles of pooled blocks come first.  Their pages have a few rows each: a row's 256 bytes by 16 lanes, zeros for rows that no query of the tile sees, a tile on its way
        // while the one before arrives.
        bool bad = false, ok = true;
        const int pooled_here = max(0, min(pooled_tiles - tile_begin, tiles));
        auto arrive = [&](int tile) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // what this thread copied, seen by the products
            __syncwarp();
            if (lane == 0) barrier_arrive(&full[tile % kPtStages]);
        };
        auto wait_for_stage = [&](int tile) {
            return tile < kPtStages || __all_sync(0xffffffffu, barrier_wait_parked(&free_again[tile % kPtStages], (tile / kPtStages - 1) & 1));
        };
        for (int tile = 0; tile < pooled_here && ok; ++tile) {
            const int base_row = rows_of(tile).base;
            int rows[2];   // of the tile's rows `lane` and 32 + lane: where they lie
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int where = base_row + 32 * h + lane, column = where / p.pool_rows;
                rows[h] = -1;
                if (where < blocks_seen) {
                    const int page = column < p.pool_max_blocks ? p.pool_table[static_cast<size_t>(segment) * p.pool_max_blocks + column] : -1;
                    if (page < 0 || page >= p.pool_pages) bad = true;
                    else rows[h] = page * p.pool_rows + where % p.pool_rows;
                }
            }
            if (!wait_for_stage(tile)) {
                ok = false;
                break;
            }
            unsigned char* stage = stages + (tile % kPtStages) * kPtStage;
            const int chunk = lane & 15;
#pragma unroll 8
            for (int r = 0; r < kPtKeys; r += 2) {
                const int row = r + (lane >> 4), from = __shfl_sync(0xffffffffu, r < 32 ? rows[0] : rows[1], row & 31);
                const uint32_t to = smem_address(stage) + static_cast<uint32_t>((chunk >> 3) * kPtPanel + row * 128 + (((chunk ^ row) & 7) << 4));
                const __nv_bfloat16* source = p.pooled_pages + (from < 0 ? 0 : (static_cast<size_t>(from) * p.groups + group) * 128 + chunk * 8);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(source), "r"(from < 0 ? 0 : 16) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (tile > 0) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                arrive(tile - 1);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (pooled_here > 0 && ok) arrive(pooled_here - 1);
        // Positions: the first row in the pages of the tile's 16-row block `lane` (lanes 0 to 3), -1 where no query of the tile sees any of it (it is not
        // loaded); looked up a tile ahead.  Lanes 0 to 3 then ask for one box each, keys or values of 32 rows, or for two of 16 where the blocks are no
        // neighbours.
        auto look_up = [&](int tile) {
            if (lane >= 4 || tile >= tiles) return -1;
            const int first = rows_of(tile).base + 16 * lane;
            if (first + 15 < first_key || first > p_last) return -1;
            const int column = first / p.page_size;
            const int page = column < p.max_blocks ? p.block_table[static_cast<size_t>(segment) * p.max_blocks + column] : -1;
            if (page < 0 || page >= p.num_pages) {
                bad = true;
                return -1;
            }
            return page * p.page_size + (first - column * p.page_size);
        };
        int rows_ahead = look_up(pooled_here);
        const int x = group * 128 + (lane & 1) * 64;
        for (int tile = pooled_here; tile < tiles && ok; ++tile) {
            const int s = tile % kPtStages, rows = rows_ahead;
            rows_ahead = look_up(tile + 1);
            const uint32_t blocks = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, rows >= 0)));
            const int first = __shfl_sync(0xffffffffu, rows, lane & 2), second = __shfl_sync(0xffffffffu, rows, (lane & 2) + 1);
            if (!wait_for_stage(tile)) {
                ok = false;
                break;
            }
            if (lane == 0) barrier_expect(&full[s], blocks * 16u * 256u);
            __syncwarp();
            if (lane < 4) {
                unsigned char* to = stages + s * kPtStage + (lane & 1) * kPtPanel + (lane >> 1) * 32 * 128;
                if (first >= 0 && second == first + 16) {
                    tma_load_2d(to, &map_32, x, first, &full[s]);
                } else {
                    if (first >= 0) tma_load_2d(to, &map_16, x, first, &full[s]);
                    if (second >= 0) tma_load_2d(to + 16 * 128, &map_16, x, second, &full[s]);
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicExch(&failed, 1);
        if (__any_sync(0xffffffffu, bad) && lane == 0) report_error(p.status, kBadPage);
    } else if (warp == 8 && lane == 0) {
        const uint32_t idesc_scores = instruction_descriptor<kPtKeys>(), idesc_output = instruction_descriptor<64>() | (1u << 16);   // V is contiguous along its columns
        const uint64_t desc_q = tile_descriptor(q_tile);
        auto issue_scores = [&](int tile) {
            const int s = tile % kPtStages;
            if (!barrier_wait_parked(&full[s], (tile / kPtStages) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t desc_k = tile_descriptor(stages + s * kPtStage);
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_f16(tmem_scores + (tile & 1) * kPtKeys, desc_q + 2 * k, desc_k + 2 * k, idesc_scores, k > 0);
            mma_commit(&s_full[tile & 1]);
            return true;
        };
        bool ok = barrier_wait(q_full, 0);   // also where the share has no tiles: the copy lands before the CTA ends
        for (int tile = 0; tile < min(2, tiles) && ok; ++tile) ok = issue_scores(tile);
        for (int tile = 0; tile < tiles && ok; ++tile) {
            if (!barrier_wait_parked(&p_full[tile & 1], (tile >> 1) & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int s = tile % kPtStages;
            const uint64_t desc_v = tile_descriptor(stages + s * kPtStage + kPtPanel);   // one panel of 64 columns, groups of 8 rows 1024 bytes apart
            const uint32_t weights = tmem_scores + (tile & 1) * kPtKeys;                  // of the first 32 rows in columns 0 to 15, of the others from column 32 on
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_f16_from_tmem(tmem_output, weights + (k >> 1) * 32 + (k & 1) * 8, desc_v + 128 * k, idesc_output, tile > 0 || k > 0);
            mma_commit(&free_again[s]);
            if (tile + 1 == tiles) mma_commit(done);
            if (tile + 2 < tiles) ok = issue_scores(tile + 2);
        }
        if (!ok) atomicExch(&failed, 1);
    } else if (warp < 8) {
        // Row r is token r / head_block of the tile's, head r % head_block of the CTA's; rows past the tile's are computed and not stored.
        const int quarter = warp & 3, half = warp >> 2;   // of tensor memory's lanes; of a tile's columns and of the output's pairs of channels
        const int row = quarter * 32 + lane;
        const int token_real = row / p.head_block, token_local = min(token_real, count - 1), head_local = row % p.head_block;
        const bool valid_row = token_real < count && first_head + head_local < per_group;
        const int head = group * per_group + min(first_head + head_local, per_group - 1);
        const int position = p_first + token_local;
        const int pools_of_row = p.pool > 0 ? max(0, position - p.window + 1) / p.pool : 0;
        const int pools_of_first = p.pool > 0 ? max(0, p_first - p.window + 1) / p.pool : 0;
        const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16;
        const PooledWeights weights(p.scale, p.cap, p.head_bias != nullptr ? p.head_bias[head] : 0.0f);
        // cosines and sines of the warp's tokens, while the first rows are on their way
        const int first_token = quarter * 32 / p.head_block, most_tokens = 31 / p.head_block + 2;
        float2* own_turns = turns + warp * most_tokens * 16;
        if (p.v_freq != nullptr && gridDim.y == 1) {
            for (int i = lane; i < most_tokens * 16; i += 32) {
                float sine, cosine;
                sincosf(static_cast<float>(p_first + first_token + i / 16) * p.v_freq[16 * half + i % 16], &sine, &cosine);
                own_turns[i] = make_float2(cosine, sine);
            }
            __syncwarp();
        }
        bool ok = true;
        auto wait_together = [](uint64_t* barrier, uint32_t parity) { return __all_sync(0xffffffffu, barrier_wait_parked(barrier, parity)); };
        for (int tile = 0; tile < tiles; ++tile) {
            const int s = tile & 1;
            const uint32_t scores = tmem_scores + s * kPtKeys + 32 * half + lane_field;
            const Rows here = rows_of(tile);
            if (!wait_together(&s_full[s], (tile >> 1) & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float raw[32];
            pt_load_32(scores, raw);
            // which of its 32 the row sees: all of them in most tiles
            const bool all_seen = here.pooled ? here.base + kPtKeys <= pools_of_first : here.base + kPtKeys - 1 <= p_first && here.base + p.window > p_last;
            uint32_t seen = 0xffffffffu;
            if (!all_seen) {
                const int key0 = here.base + 32 * half;
                const int low = here.pooled ? 0 : position - p.window + 1, high = here.pooled ? pools_of_row - 1 : position;
                seen = 0u;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const bool visible = key0 + i >= low && key0 + i <= high;
                    if (!visible) raw[i] = 0.0f;   // what lies there may be no number, and two weights share a reciprocal
                    seen |= visible ? 1u << i : 0u;
                }
            }
            uint32_t packed[16];
            auto weigh = [&](auto form, auto near) {
#pragma unroll
                for (int i = 0; i < 16; ++i) packed[i] = weights.template pair<decltype(form)::value, decltype(near)::value>(raw[2 * i], raw[2 * i + 1]);
            };
            float top = 0.0f;
#pragma unroll
            for (int i = 0; i < 32; i += 2) asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(top) : "f"(top), "f"(raw[i]), "f"(raw[i + 1]));
            // (by the row's own scores alone: what shares the warp changes no bit)
            if (!(p.cap > 0.0f)) {
                if (weights.near(top)) weigh(std::integral_constant<int, 0>{}, std::true_type{});
                else weigh(std::integral_constant<int, 0>{}, std::false_type{});
            } else if (top <= weights.most) {
                weigh(std::integral_constant<int, 1>{}, std::true_type{});
            } else {
                weigh(std::integral_constant<int, 2>{}, std::false_type{});
            }
            __syncwarp();
            if (!all_seen) {
#pragma unroll
                for (int i = 0; i < 16; ++i) packed[i] &= ((seen >> (2 * i)) & 1u ? 0x0000ffffu : 0u) | ((seen >> (2 * i + 1)) & 1u ? 0xffff0000u : 0u);
                if (here.base < here.low || here.base + kPtKeys - 1 > here.high) {
                    // Rows no query of the tile sees hold whatever was left there, or were not loaded: a weight of zero does not silence a value that is not
                    // finite.  All of a row's bytes are cleared, whatever their order within it.
                    const int where = here.base + static_cast<int>(threadIdx.x >> 2);
                    if (!wait_together(&full[tile % kPtStages], (tile / kPtStages) & 1)) {   // (long over)
                        ok = false;
                        break;
                    }
                    if (where < here.low || where > here.high) {
                        uint4* destination = reinterpret_cast<uint4*>(stages + (tile % kPtStages) * kPtStage + kPtPanel + (threadIdx.x >> 2) * 128 + (threadIdx.x & 3) * 32);
                        destination[0] = destination[1] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
            }
            tmem_store_16(scores, packed);   // over this thread's own scores
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();   // every lane's, before the warp's one arrival
            if (lane == 0) barrier_arrive(&p_full[s]);
        }
        if (ok && tiles > 0 && !wait_together(done, 0)) ok = false;
        if (!ok) atomicExch(&failed, 1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // the thread's 32 of the row's channels: the first and second of pairs 16 half .. + 15
        const int step = p.v_interleaved ? 16 : 32, begin = p.v_interleaved ? 32 * half : 16 * half;
        uint32_t low[16], high[16];
        tmem_load_16(tmem_output + lane_field + begin, low);
        tmem_load_16(tmem_output + lane_field + begin + step, high);
        if (tiles == 0) {   // a share without tiles has no products
#pragma unroll
            for (int i = 0; i < 16; ++i) low[i] = high[i] = 0u;
        }
        if (valid_row && ok) {
            const size_t offset = (static_cast<size_t>(first_row + token_local) * p.heads + head) * 64 + begin;
            if (p.partial != nullptr) {
                float* destination = p.partial + static_cast<size_t>(blockIdx.y) * p.total_rows * p.heads * 64 + offset;
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    *reinterpret_cast<uint4*>(destination + i) = make_uint4(low[i], low[i + 1], low[i + 2], low[i + 3]);
                    *reinterpret_cast<uint4*>(destination + step + i) = make_uint4(high[i], high[i + 1], high[i + 2], high[i + 3]);
                }
            } else {
                const float2* turn = own_turns + (token_local - first_token) * 16;
                float a[16], b[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) a[i] = __uint_as_float(low[i]), b[i] = __uint_as_float(high[i]);
                if (p.v_freq != nullptr && !p.v_interleaved) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float2 t = turn[i];
                        const float turned = a[i] * t.x + b[i] * t.y;
                        b[i] = b[i] * t.x - a[i] * t.y;
                        a[i] = turned;
                    }
                } else if (p.v_freq != nullptr) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float2 t = turn[i / 2], u = turn[8 + i / 2];
                        const float first = a[i] * t.x + a[i + 1] * t.y, third = b[i] * u.x + b[i + 1] * u.y;
                        a[i + 1] = a[i + 1] * t.x - a[i] * t.y;
                        b[i + 1] = b[i + 1] * u.x - b[i] * u.y;
                        a[i] = first;
                        b[i] = third;
                    }
                }
                __nv_bfloat162 first[8], second[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) first[i] = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]), second[i] = __floats2bfloat162_rn(b[2 * i], b[2 * i + 1]);
                uint4* destination = reinterpret_cast<uint4*>(p.out + offset);
                destination[0] = *reinterpret_cast<const uint4*>(&first[0]);
                destination[1] = *reinterpret_cast<const uint4*>(&first[4]);
                destination = reinterpret_cast<uint4*>(p.out + offset + step);
                destination[0] = *reinterpret_cast<const uint4*>(&second[0]);
                destination[1] = *reinterpret_cast<const uint4*>(&second[4]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (failed) {
        // Let whatever copies are still in flight land before the shared memory goes away.
        if (threadIdx.x == 0) report_error(p.status, kWaitTimeout);
        for (int spin = 0; spin < 2000; ++spin) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_output), "r"(256) : "memory");
}

// Rows of `channels` bfloat16 in boxes of 64 channels and `box_rows` rows, 128-byte swizzle.
static bool pooled_row_map(CUtensorMap* map, const void* base, int channels, long long rows, int box_rows) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(channels), static_cast<cuuint64_t>(rows)}, strides[1] = {static_cast<cuuint64_t>(channels) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)}, steps[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the shares' sums, added in their order, turned back and rounded (attention_pooled.cu)
void launch_pooled_finish(const float* partial, int shares, __nv_bfloat16* out, const int* positions, int total_rows, int heads, int dv, const float* v_freq, int v_interleaved,
                          const int* tiles, int num_tiles, int tile_tokens, cudaStream_t stream);

}  // namespace lb

extern "C" {

// As lb_pooled_attention_mma, for heads of 64 key and 64 value channels and token pages of a multiple of 16 rows; a tile has at most 128 / head_block
// tokens (16 * (8 / head_block), as there).  Returns -2 for sizes it does not take, -5 if no tensor map could be made.
int lb_pooled_attention_tcgen05(const void* q, const void* pages, const void* pooled_pages, void* out, const int* tiles, int num_tiles, const int* positions,
                                const int* token_segment, const int* block_table, const int* pool_table, int heads, int groups, int page_size,
                                int num_pages, int max_blocks, int pool_rows, int pool_pages, int pool_max_blocks, int head_block, float scale, float cap,
                                const float* head_bias, int window, int pool, const float* v_freq, int v_interleaved, int* status, cudaStream_t stream, int shares,
                                float* partial, int total_rows) {
    if (num_tiles == 0) return 0;
    if (shares < 1 || shares > 64 || (shares > 1 && partial == nullptr)) return -2;
    if (shares == 1) partial = nullptr;
    if (groups < 1 || heads % groups != 0 || page_size < 16 || page_size % 16 != 0 || num_pages < 1 || window < 1 || pool < 0 || head_block < 1 || head_block > 4 ||
        total_rows < 1 || (pool > 0 && (pool_rows < 1 || pool_pages < 1 || pooled_pages == nullptr)) ||
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages) | reinterpret_cast<uintptr_t>(pooled_pages) | reinterpret_cast<uintptr_t>(out) |
          reinterpret_cast<uintptr_t>(partial)) & 15))
        return -2;
    lb::EncodeTiled encode = lb::encode_tiled();
    if (encode == nullptr) return -5;
    const int per_group = heads / groups, tile_tokens = 16 * (8 / head_block), channels = groups * 128;
    const long long rows = static_cast<long long>(num_pages) * page_size, pooled = pool > 0 ? static_cast<long long>(pool_pages) * pool_rows : 0;
    if (rows > 0x7fffffffll || pooled > 0x7fffffffll) return -2;
    CUtensorMap map_q, map_16, map_32;
    {
        const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(total_rows)}, strides[2] = {128, static_cast<cuuint64_t>(heads) * 128};
        const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(head_block), static_cast<cuuint32_t>(tile_tokens)}, steps[3] = {1, 1, 1};
        if (encode(&map_q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -5;
    }
    if (!lb::pooled_row_map(&map_16, pages, channels, rows, 16) || !lb::pooled_row_map(&map_32, pages, channels, rows, 32)) return -5;
    lb::PooledTcParams p;
    p.pooled_pages = static_cast<const __nv_bfloat16*>(pooled_pages);
    p.out = static_cast<__nv_bfloat16*>(out);
    p.partial = partial;
    p.tiles = tiles;
    p.positions = positions;
    p.token_segment = token_segment;
    p.block_table = block_table;
    p.pool_table = pool_table;
    p.head_bias = head_bias;
    p.v_freq = v_freq;
    p.status = status;
    p.page_size = page_size, p.num_pages = num_pages, p.max_blocks = max_blocks;
    p.pool_rows = pool > 0 ? pool_rows : 1, p.pool_pages = pool_pages, p.pool_max_blocks = pool_max_blocks;
    p.heads = heads, p.groups = groups, p.head_block = head_block, p.tile_tokens = tile_tokens, p.window = window, p.pool = pool;
    p.v_interleaved = v_interleaved, p.total_rows = total_rows;
    p.scale = scale, p.cap = cap;
    const size_t shared = lb::kPtStages * lb::kPtStage + lb::kPtRows * 128 + 256 /* barriers */ + 8 * (31 / head_block + 2) * 16 * sizeof(float2) + 1024 /* alignment */;
    static lb::OncePerDevice once;
    const cudaError_t allowed = lb::allow_shared_memory(once, lb::pooled_attention_tcgen05_kernel, 120 * 1024);
    if (allowed != cudaSuccess) return static_cast<int>(allowed);
    const dim3 grid(static_cast<unsigned>(num_tiles) * groups * ((per_group + head_block - 1) / head_block), shares);
    const cudaError_t launched = lb::launch_overlapped(lb::pooled_attention_tcgen05_kernel, grid, dim3(lb::kPtThreads), shared, stream, map_q, map_16, map_32, p);
    if (launched != cudaSuccess) return static_cast<int>(launched);
    if (shares > 1) lb::launch_pooled_finish(partial, shares, p.out, positions, total_rows, heads, 64, v_freq, v_interleaved, tiles, num_tiles, tile_tokens, stream);
    return LB_LAUNCH_RESULT();
}

}  // extern "C"
