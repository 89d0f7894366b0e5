// Latent attention (see attention_latent.cu) on the fifth-generation tensor cores.
//
// A CTA takes one item: up to 128 query rows = consecutive tokens of one request x all heads, which share the cached rows
// [latent | rope].  The rows come in tiles of 128 that start at multiples of 128 from the request's first token, by TMA into a
// ring of two tiles, and serve both products from there: as K for S = Q K^T (K-major, panels of 64 channels and one of the rotated
// ones), and, their latent panels, as V for O += P V (the same bytes, read as an operand that is contiguous along its columns).
// O (128 x latent), two tiles of scores and, over the scores they came from, the rounded probabilities live in tensor memory.
//   warps 0-7  two threads a row, 64 scores each in registers: they exchange their maxima through shared memory, rescale O where a row's maximum has
//              grown (a maximum that may lag by 2^8, so that O rarely has to be, takes 2 us less and has the largest weights rounded: an error of 0.00197
//              against 0.00182), write P and add up what they wrote
//   warp 8     allocates tensor memory; one lane issues, two tiles at a time, O += P V of both, then S = Q K^T of the next two: what the ring
//              waits for and what the softmax takes lie under the other tile's products
//   warp 9     asks for the ring's boxes, a quarter of a tile as soon as the second product has read it
// What bounds it: 2 tiles take 8,000 to 9,400 cycles, of which the products would take 5,700 (they read 250 KB of operands a tile from shared memory), the
// softmax of the second tile that nothing covers 1,300, and the rest is the wait for the next tiles' boxes (the copy engine's time per box: rows 576 bytes
// apart lie across lines).  A ring of a third tile finds no room beside the queries.  Measured, 16 heads over 256 + 32 channels, 1,023
// tokens behind 1,500 under a window of 2,048: 55 us (250 us on mma.sync, eight warps); 512 behind 4,096: 56 (196); 64 tokens that decode behind
// 1,000 each: 30 (50); 8 behind 4,000 each: 24 (34).  Pages that are not neighbours: 63 us.  Tried: the rows by cp.async of three warps (73 us), the rotated
// channels by cp.async of two (63 us).
// Every wait is bounded and reports through the status word.
#include "tcgen05.cuh"

namespace lb {

constexpr int kLtRows = 128, kLtKeys = 128, kLtThreads = 320;
constexpr int kLtPanelBytes = 2 * kLtKeys * 128;   // of a latent panel's ring: two tiles of 128 rows of 64 channels
constexpr int kLtMostShared = 226 * 1024;          // beside the kernel's few static bytes

struct LatentTcParams {
    __nv_bfloat16* out;      // [tokens][heads][latent]
    float* partial;          // splits > 1: [tokens][heads][split][latent + 2] (O unnormalised, maximum in base-2 units, sum)
    const int* items;        // [num_items][2]: first token row, count
    const int* positions;
    const int* token_segment;
    const int* block_table;
    const float* sink;       // [heads] or null
    int* status;
    int page_size, num_pages, max_blocks;
    int num_heads, latent, rope, splits, window;
    float scale_log2;
};

// A K-major tile whose rows of `row_bytes` (32, 64 or 128) are swizzled over their own length.
__device__ __forceinline__ uint64_t lt_narrow_descriptor(const void* tile, int row_bytes) {
    const uint64_t address = smem_address(tile), layout = row_bytes == 128 ? 2 : row_bytes == 64 ? 4 : 6;
    return ((address & 0x3FFFFull) >> 4) | (1ull << 16) | (static_cast<uint64_t>(8 * row_bytes >> 4) << 32) | (1ull << 46) | (layout << 61);
}
// 16 rows of the latent panels as an operand contiguous along its columns: panels (64 columns) kLtPanelBytes apart, groups of 8 rows 1024 bytes.
__device__ __forceinline__ uint64_t lt_value_descriptor(const void* rows) {
    const uint64_t address = smem_address(rows);
    return ((address & 0x3FFFFull) >> 4) | (static_cast<uint64_t>(kLtPanelBytes >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ float lt_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lt_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// grid (items, splits), 320 threads.
__global__ void __launch_bounds__(kLtThreads, 1)
latent_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q_rope, const __grid_constant__ CUtensorMap map_16_rows,
                                const __grid_constant__ CUtensorMap map_16_rope, const __grid_constant__ CUtensorMap map_32_rows,
                                const __grid_constant__ CUtensorMap map_32_rope, const LatentTcParams p) {
    extern __shared__ unsigned char raw_shared[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_shared) + 1023) & ~static_cast<uintptr_t>(1023));
    const int panels = p.latent / 64, rope_bytes = 2 * p.rope;
    unsigned char* ring = base;                                       // [panel][256 rows][128 bytes]
    unsigned char* q_tile = ring + panels * kLtPanelBytes;            // [panel][128 rows][128 bytes]
    unsigned char* ring_rope = q_tile + panels * kLtRows * 128;       // [256 rows][rope_bytes]
    unsigned char* q_rope = ring_rope + 2 * kLtKeys * rope_bytes;     // [128 rows][rope_bytes]
    float* exchange = reinterpret_cast<float*>(q_rope + kLtRows * rope_bytes);   // [2][2][128]: maxima by tile parity and half; at the end the sums
    uint64_t* barriers = reinterpret_cast<uint64_t*>(exchange + 4 * kLtRows);
    uint64_t* q_full = barriers;
    uint64_t* k_full = barriers + 1;     // [2]
    uint64_t* k_free = barriers + 3;     // [2][4]: quarters of a tile
    uint64_t* s_full = barriers + 11;    // [2]
    uint64_t* p_full = barriers + 13;    // [2]
    uint64_t* pv_done = barriers + 15;   // [2]
    uint64_t* rows_met = barriers + 17;  // [4]: both warps of 32 rows have left their maxima
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(barriers + 21);
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = gridDim.x - 1 - blockIdx.x, split = blockIdx.y;   // a prompt's last items see the most rows: they start first
    const int first_token = p.items[2 * item], count = p.items[2 * item + 1];
    const int segment = p.token_segment[first_token], first_position = p.positions[first_token], last_position = first_position + count - 1;
    const int lowest = p.window > 0 ? max(0, first_position - p.window + 1) : 0;   // the lowest row any query of the item sees
    // this CTA's share of the item's tiles
    const int tile_lo = lowest / kLtKeys, tile_hi = last_position / kLtKeys + 1, per_split = (tile_hi - tile_lo + p.splits - 1) / p.splits;
    const int tile_begin = tile_lo + split * per_split, tiles = max(0, min(tile_hi, tile_begin + per_split) - tile_begin);

    if (threadIdx.x == 0) {
        barrier_init(q_full, 1);
        for (int s = 0; s < 2; ++s) {
            barrier_init(&k_full[s], 1);
            barrier_init(&s_full[s], 1);
            barrier_init(&p_full[s], 8);   // one arrival per softmax warp
            barrier_init(&pv_done[s], 1);
        }
        for (int s = 0; s < 8; ++s) barrier_init(&k_free[s], 1);
        for (int s = 0; s < 4; ++s) barrier_init(&rows_met[s], 2);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    wait_for_previous_kernel();   // launched to start early: the queries and the newest rows are there from here on
    allow_next_kernel();
    const uint32_t tmem_output = *tmem_slot, tmem_scores = tmem_output + 256;   // scores: two tiles of 128 columns

    if (warp == 9) {
        // A lane per panel (the last for the rotated channels) and quarter of a tile: one box of 32 rows where the quarter's two blocks of 16 are neighbours in
        // the pages, two of 16 where they are not.
        const bool rotated = lane == panels;
        const CUtensorMap *wide = rotated ? &map_32_rope : &map_32_rows, *narrow = rotated ? &map_16_rope : &map_16_rows;
        unsigned char* panel = rotated ? ring_rope : ring + lane * kLtPanelBytes;
        const int pitch = rotated ? rope_bytes : 128;
        if (lane == 0 && tiles > 0) {
            barrier_expect(q_full, static_cast<uint32_t>(panels * kLtRows * 128 + kLtRows * rope_bytes));
            for (int c = 0; c < panels; ++c) tma_load_2d(q_tile + c * kLtRows * 128, &map_q, 64 * c, first_token * p.num_heads, q_full);
            tma_load_2d(q_rope, &map_q_rope, p.latent, first_token * p.num_heads, q_full);
        }
        // The first row in the pages of the tile's 16-row block `lane` (lanes 0 to 7), -1 where no query of the item sees any of it (it is not loaded: its
        // scores are masked and its values cleared by the softmax warps); looked up a tile ahead.
        bool bad = false;
        auto look_up = [&](int tile) {
            const int first = (tile_begin + tile) * kLtKeys + 16 * lane;
            if (lane >= 8 || tile >= tiles || first + 15 < lowest || first > last_position) return -1;
            const int column = first / p.page_size;
            const int page = column < p.max_blocks ? p.block_table[static_cast<size_t>(segment) * p.max_blocks + column] : -1;
            if (page < 0 || page >= p.num_pages) {
                bad = true;
                return -1;
            }
            return page * p.page_size + (first - column * p.page_size);
        };
        int rows_ahead = look_up(0);
        bool ok = true;
        for (int tile = 0; tile < tiles && ok; ++tile) {
            const int s = tile & 1, rows = rows_ahead;
            rows_ahead = look_up(tile + 1);
            const uint32_t blocks = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, rows >= 0)));
            for (int quarter = 0; quarter < 4; ++quarter) {
                const int first = __shfl_sync(0xffffffffu, rows, 2 * quarter), second = __shfl_sync(0xffffffffu, rows, 2 * quarter + 1);
                if (tile >= 2 && !__all_sync(0xffffffffu, barrier_wait_parked(&k_free[4 * s + quarter], ((tile >> 1) - 1) & 1))) {
                    ok = false;
                    break;
                }
                // (the tile before in this half of the ring has been read, so its phase of the barrier is over)
                if (quarter == 0 && lane == 0) barrier_expect(&k_full[s], blocks * 32u * static_cast<uint32_t>(p.latent + p.rope));
                __syncwarp();
                if (lane <= panels) {
                    unsigned char* to = panel + (s * kLtKeys + 32 * quarter) * pitch;
                    const int x = rotated ? p.latent : 64 * lane;
                    if (first >= 0 && second == first + 16) {
                        tma_load_2d(to, wide, x, first, &k_full[s]);
                    } else {
                        if (first >= 0) tma_load_2d(to, narrow, x, first, &k_full[s]);
                        if (second >= 0) tma_load_2d(to + 16 * pitch, narrow, x, second, &k_full[s]);
                    }
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) atomicExch(&failed, 1);
        if (__any_sync(0xffffffffu, bad) && lane == 0) report_error(p.status, kBadPage);
    } else if (warp == 8 && lane == 0) {
        const uint32_t idesc_scores = instruction_descriptor<kLtKeys>();
        const uint32_t idesc_output = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) /* B contiguous along its columns */ | (static_cast<uint32_t>(p.latent >> 3) << 17) |
                                      (static_cast<uint32_t>(kLtRows >> 4) << 24);
        auto issue_scores = [&](int tile) {
            const int s = tile & 1;
            if (!barrier_wait_parked(&k_full[s], (tile >> 1) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t scores = tmem_scores + s * kLtKeys;
            for (int c = 0; c < panels; ++c) {
                const uint64_t desc_q = tile_descriptor(q_tile + c * kLtRows * 128), desc_k = tile_descriptor(ring + c * kLtPanelBytes + s * kLtKeys * 128);
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_f16(scores, desc_q + 2 * k, desc_k + 2 * k, idesc_scores, c > 0 || k > 0);
            }
            const uint64_t desc_q = lt_narrow_descriptor(q_rope, rope_bytes), desc_k = lt_narrow_descriptor(ring_rope + s * kLtKeys * rope_bytes, rope_bytes);
            for (int k = 0; k < p.rope / 16; ++k) mma_f16(scores, desc_q + 2 * k, desc_k + 2 * k, idesc_scores, true);
            mma_commit(&s_full[s]);
            return true;
        };
        auto issue_output = [&](int tile) {
            const int s = tile & 1;
            if (!barrier_wait_parked(&p_full[s], (tile >> 1) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t weights = tmem_scores + s * kLtKeys;   // of the first 64 rows in columns 0 to 31, of the others from column 64 on
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                mma_f16_from_tmem(tmem_output, weights + (k >> 2) * 64 + (k & 3) * 8, lt_value_descriptor(ring + (s * kLtKeys + 16 * k) * 128), idesc_output, tile > 0 || k > 0);
                if (k & 1) mma_commit(&k_free[4 * s + (k >> 1)]);
            }
            mma_commit(&pv_done[s]);
            return true;
        };
        bool ok = tiles == 0 || barrier_wait(q_full, 0);
        for (int tile = 0; tile < min(2, tiles) && ok; ++tile) ok = issue_scores(tile);
        for (int tile = 0; tile < tiles && ok; tile += 2) {
            for (int next = tile; next < min(tile + 2, tiles) && ok; ++next) ok = issue_output(next);
            for (int next = tile + 2; next < min(tile + 4, tiles) && ok; ++next) ok = issue_scores(next);
        }
        if (!ok) atomicExch(&failed, 1);
    } else if (warp < 8) {
        // Row r is token r / heads of the item's, head r % heads; rows past the item's are computed and not stored.
        const int quarter = warp & 3, half = warp >> 2;   // tensor memory's lanes 32 (warp % 4) on are this warp's
        const int row = quarter * 32 + lane;
        const int token_local = min(row / p.num_heads, count - 1), head = row % p.num_heads;
        const bool valid_row = row < count * p.num_heads;
        const int row_position = first_position + token_local;
        const int row_first = p.window > 0 ? max(0, row_position - p.window + 1) : 0;
        const int last_first = p.window > 0 ? max(0, last_position - p.window + 1) : 0;   // the first row the item's last query sees
        const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16;
        const int share = p.latent / 2, channel0 = half * share;   // of O's columns
        float reference = -INFINITY, row_sum = 0.0f;
        bool ok = true;
        auto wait_together = [](uint64_t* barrier, uint32_t parity) { return __all_sync(0xffffffffu, barrier_wait_parked(barrier, parity)); };
        // What this thread has written to `exchange` is there for its row's other thread, and the other's for this one: bounded, as a named barrier is not.
        auto meet = [&](int turn) {
            __syncwarp();
            if (lane == 0) barrier_arrive(&rows_met[quarter]);
            return __all_sync(0xffffffffu, barrier_wait_busy(&rows_met[quarter], turn & 1));
        };
        for (int tile = 0; tile < tiles; ++tile) {
            const int s = tile & 1, key0 = (tile_begin + tile) * kLtKeys + 64 * half;
            const uint32_t scores = tmem_scores + s * kLtKeys + 64 * half + lane_field;
            if (!wait_together(&s_full[s], (tile >> 1) & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t raw[64];
            tmem_load_64(scores, raw);
            if (key0 + 63 > first_position || key0 < last_first) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (key0 + i < row_first || key0 + i > row_position) raw[i] = 0xff800000u;   // minus infinity
            }
            float tops[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 64; i += 2) tops[(i >> 1) & 3] = lt_max3(tops[(i >> 1) & 3], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]));
            float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
            float* maxima = exchange + s * 2 * kLtRows;
            maxima[half * kLtRows + row] = top;
            if (!meet(tile)) {   // (a tile's maxima lie apart from the tile's before)
                ok = false;
                break;
            }
            top = fmaxf(top, maxima[(half ^ 1) * kLtRows + row]) * p.scale_log2;   // the scale is positive
            const float moved = fmaxf(reference, top), shift = moved == -INFINITY ? 0.0f : moved;   // a row that has seen nothing yet: every term below is 2^-inf = 0
            const float rescale = lt_exp2(reference - shift);
            reference = moved;
            if (tile > 0 && __any_sync(0xffffffffu, rescale != 1.0f)) {
                // (the products before the last are done, or these scores would not be there: the barrier's phase is the last's or the one after)
                if (!wait_together(&pv_done[s ^ 1], ((tile - 1) >> 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c = 0; c < share; c += 32) {
                    uint32_t held[32];
                    tmem_load_32(tmem_output + lane_field + channel0 + c, held);
#pragma unroll
                    for (int i = 0; i < 32; ++i) held[i] = __float_as_uint(__uint_as_float(held[i]) * rescale);
                    tmem_store_32(tmem_output + lane_field + channel0 + c, held);
                }
            }
            float sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                uint32_t packed[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float low = lt_exp2(fmaf(__uint_as_float(raw[32 * part + 2 * i]), p.scale_log2, -shift));
                    const float high = lt_exp2(fmaf(__uint_as_float(raw[32 * part + 2 * i + 1]), p.scale_log2, -shift));
                    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
                    packed[i] = *reinterpret_cast<const uint32_t*>(&pair);
                    // the sums add what the product uses: the rounded probabilities
                    sums[i & 3] += __uint_as_float(packed[i] << 16) + __uint_as_float(packed[i] & 0xffff0000u);
                }
                tmem_store_16(scores + 16 * part, packed);   // over this thread's own scores
            }
            row_sum = row_sum * rescale + ((sums[0] + sums[1]) + (sums[2] + sums[3]));
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            const int tile_key = (tile_begin + tile) * kLtKeys;
            if (tile_key < lowest || tile_key + kLtKeys - 1 > last_position) {
                // Rows no query of the item sees hold whatever was left there, or were not loaded: a zero probability does not silence a
                // value that is not finite.  All of a row's bytes are cleared, whatever their order within it.
                if (!wait_together(&k_full[s], (tile >> 1) & 1)) {   // (long over)
                    ok = false;
                    break;
                }
                const int key = tile_key + static_cast<int>(threadIdx.x >> 1);
                if (key < lowest || key > last_position) {
                    for (int c = threadIdx.x & 1; c < panels; c += 2) {
                        uint4* destination = reinterpret_cast<uint4*>(ring + c * kLtPanelBytes + (s * kLtKeys + static_cast<int>(threadIdx.x >> 1)) * 128);
#pragma unroll
                        for (int i = 0; i < 8; ++i) destination[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();   // every lane's, before the warp's one arrival
            if (lane == 0) barrier_arrive(&p_full[s]);
        }
        if (ok && tiles > 0 && !wait_together(&pv_done[(tiles - 1) & 1], ((tiles - 1) >> 1) & 1)) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // The maxima of the tile before the last are read before its partner writes the last's; the sums lie where no maximum of the last tile does.
        float* totals = exchange + (tiles & 1) * 2 * kLtRows;
        totals[half * kLtRows + row] = row_sum;
        if (!ok || !meet(tiles)) {
            ok = false;
            atomicExch(&failed, 1);
        }
        const float sum = totals[row] + totals[kLtRows + row];
        const size_t out_row = static_cast<size_t>(first_token) * p.num_heads + row;
        if (p.splits == 1) {
            float norm = sum > 0.0f ? 1.0f / sum : 0.0f;
            if (p.sink != nullptr) {
                // the sink joins the sum as 2^(sink log2 e - reference), computed on the side that cannot overflow
                const float gap = p.sink[head] * 1.4426950408889634f - (reference == -INFINITY ? 0.0f : reference);
                norm = reference == -INFINITY ? 0.0f : (gap > 0.0f ? exp2f(-gap) / (sum * exp2f(-gap) + 1.0f) : 1.0f / (sum + exp2f(gap)));
            }
#pragma unroll 1
            for (int c = 0; c < share; c += 32) {
                uint32_t held[32];
                tmem_load_32(tmem_output + lane_field + channel0 + c, held);
                if (valid_row && ok) {
                    uint4* destination = reinterpret_cast<uint4*>(p.out + out_row * p.latent + channel0 + c);
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 values;
                        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&values);
#pragma unroll
                        for (int e = 0; e < 4; ++e) pairs[e] = __floats2bfloat162_rn(__uint_as_float(held[i + 2 * e]) * norm, __uint_as_float(held[i + 2 * e + 1]) * norm);
                        destination[i / 8] = values;
                    }
                }
                __syncwarp();
            }
        } else {
            float* destination = p.partial + (out_row * p.splits + split) * (p.latent + 2);
#pragma unroll 1
            for (int c = 0; c < share; c += 32) {
                uint32_t held[32];
                tmem_load_32(tmem_output + lane_field + channel0 + c, held);
                if (valid_row && ok) {
#pragma unroll
                    for (int i = 0; i < 32; i += 2)   // a share without tiles has no products: zeros
                        *reinterpret_cast<float2*>(destination + channel0 + c + i) = tiles > 0 ? make_float2(__uint_as_float(held[i]), __uint_as_float(held[i + 1])) : make_float2(0.0f, 0.0f);
                }
                __syncwarp();
            }
            if (half == 0 && valid_row && ok) {
                destination[p.latent] = reference;
                destination[p.latent + 1] = sum;
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
    if (warp == 8) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_output), "r"(512) : "memory");
    }
}

static size_t latent_tcgen05_shared(int latent, int rope) {
    return static_cast<size_t>(2 * kLtKeys + kLtRows) * 2 * (latent + rope) + 4 * kLtRows * sizeof(float) + 256 /* barriers */ + 1024 /* alignment */;
}

// Rows of `channels` bfloat16, in boxes of `box_channels` x `box_rows`, swizzled over a box's row.
static bool latent_row_map(CUtensorMap* map, const void* base, int channels, long long rows, int box_channels, int box_rows) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(channels), static_cast<cuuint64_t>(rows)}, strides[1] = {static_cast<cuuint64_t>(channels) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_channels), static_cast<cuuint32_t>(box_rows)}, steps[2] = {1, 1};
    const CUtensorMapSwizzle swizzle = box_channels == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : box_channels == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the shares' sums, merged in their order (attention_latent.cu)
void launch_latent_merge(const float* partial, __nv_bfloat16* out, int rows, int splits, int latent, const float* sink, int num_heads, cudaStream_t stream);

}  // namespace lb

extern "C" {

// bfloat16; latent 64, 128, 192 or 256, rope 16, 32 or 64, pages of a multiple of 16 rows, a positive scale.  items as for lb_latent_attention_mma, each at
// most 128 / num_heads tokens.  partial: splits > 1 only, [tokens][heads][splits][latent + 2] floats.  Returns -2 for sizes it does not take,
// -5 if no tensor map could be made.
int lb_latent_attention_tcgen05(const void* q, const void* pages, void* out, float* partial, const int* items, int num_items, const int* positions,
                                const int* token_segment, const int* block_table, int tokens, int num_heads, int latent, int rope, int page_size,
                                int num_pages, int max_blocks, float scale, int window, int splits, int* status, cudaStream_t stream, const float* sink) {
    if (num_items == 0 || tokens == 0) return 0;
    const size_t shared = lb::latent_tcgen05_shared(latent, rope);
    if (latent < 64 || latent > 256 || latent % 64 != 0 || (rope != 16 && rope != 32 && rope != 64) || page_size < 16 || page_size % 16 != 0 || num_pages < 1 || num_heads < 1 ||
        num_heads > lb::kLtRows || !(scale > 0.0f) || splits < 1 || splits > 65535 || (splits > 1 && partial == nullptr) || shared > lb::kLtMostShared ||
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages) | reinterpret_cast<uintptr_t>(out)) & 15))
        return -2;
    CUtensorMap map_q, map_q_rope, map_16_rows, map_16_rope, map_32_rows, map_32_rope;
    const long long query_rows = static_cast<long long>(tokens) * num_heads, rows = static_cast<long long>(num_pages) * page_size;
    if (query_rows > 0x7fffffffll || rows > 0x7fffffffll) return -2;
    if (!lb::latent_row_map(&map_q, q, latent + rope, query_rows, 64, lb::kLtRows) || !lb::latent_row_map(&map_q_rope, q, latent + rope, query_rows, rope, lb::kLtRows) ||
        !lb::latent_row_map(&map_16_rows, pages, latent + rope, rows, 64, 16) || !lb::latent_row_map(&map_16_rope, pages, latent + rope, rows, rope, 16) ||
        !lb::latent_row_map(&map_32_rows, pages, latent + rope, rows, 64, 32) || !lb::latent_row_map(&map_32_rope, pages, latent + rope, rows, rope, 32))
        return -5;
    static lb::OncePerDevice once;
    const cudaError_t allowed = lb::allow_shared_memory(once, lb::latent_attention_tcgen05_kernel, lb::kLtMostShared);
    if (allowed != cudaSuccess) return static_cast<int>(allowed);
    lb::LatentTcParams p;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.partial = partial;
    p.items = items;
    p.positions = positions;
    p.token_segment = token_segment;
    p.block_table = block_table;
    p.sink = sink;
    p.status = status;
    p.page_size = page_size;
    p.num_pages = num_pages;
    p.max_blocks = max_blocks;
    p.num_heads = num_heads;
    p.latent = latent;
    p.rope = rope;
    p.splits = splits;
    p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    const cudaError_t launched = lb::launch_overlapped(lb::latent_attention_tcgen05_kernel, dim3(num_items, splits), dim3(lb::kLtThreads), shared, stream, map_q, map_q_rope, map_16_rows,
                                                       map_16_rope, map_32_rows, map_32_rope, p);
    if (launched != cudaSuccess) return static_cast<int>(launched);
    if (splits > 1) lb::launch_latent_merge(partial, p.out, tokens * num_heads, splits, latent, sink, num_heads, stream);
    return LB_LAUNCH_RESULT();
}

}  // extern "C"
