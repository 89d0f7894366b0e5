// Paged attention for portions of prompts on the fifth-generation tensor cores: scores and output
// live in tensor memory, keys, values and queries arrive by TMA.
//
// One CTA handles up to 128 rows = (consecutive tokens of one request) x (the query heads of one K/V
// head), which all see the same keys and values.  Keys are visited in tiles of 64, starting at a
// multiple of 64 whatever the portion's start.  Value heads of 64 channels run on the second kernel (two threads a row).  Roles in the first:
//   warp 0     one lane asks for Q once (a 3-D box: channels x the K/V head's query heads x tokens) and,
//              per tile and 16-key block, for a box of K rows (128-byte swizzle) and a box of the
//              transposed V page (32-byte swizzle), into two stages;
//   warp 1     allocates tensor memory; one lane issues  S = Q K^T  (M 128, N 64, four steps over the
//              64 channels) and, once the probabilities are in shared memory,  O += P V  (N 128
//              channels, four steps of 16 keys, one per V box);
//   warps 2-5  a thread per row: read the row's 64 scores from tensor memory, mask on edge tiles,
//              update the row's reference exponent and sum (32-bit, base 2, no shuffles: the row is
//              the thread's own), rescale the row of O in tensor memory when the exponent moved, write
//              P (bfloat16) into shared memory in the operand's swizzled layout; at the end divide the
//              row of O by its sum and store it.
// Two CTAs share an SM, so that one's softmax runs under the other's products.  Every wait is bounded and reports through the status word.
// Takes key heads of up to 64 channels (multiples of 8, padded with zeros to 64 by the copies' out-of-bounds fill), value heads of 64 or
// 128, pages that are multiples of 16 keys, up to 128 query heads per K/V
// head.  Several key heads may share a value head (the maps of differential attention); the output is bfloat16 or, for a
// consumer that goes on in 32-bit, float32.
#include <type_traits>

#include "tcgen05.cuh"

namespace lb {

constexpr int kTaRows = 128;      // rows of a tile (lanes of tensor memory)
constexpr int kTaKeys = 64;       // keys per tile
constexpr int kTaChannels = 64;    // channels of a 128-byte swizzled row
constexpr int kTaThreads = 192;
constexpr int kTaTileTokens = 32;  // tokens of a tile record
constexpr float kTaMaxSlack = 8.0f;   // how far a row's maximum may outgrow its reference exponent (base 2)

struct TaParams {
    void* out;              // [tokens, heads, value_dim], bfloat16 or float32
    int keys_per_value;     // key heads that share a value head
    int out_float;
    const int* tiles;       // [num_tiles, 2]: first token, count <= 32
    const int* positions;
    const int* token_segment;
    const int* block_table;
    int num_heads, num_groups, tokens_per_cta;
    int page_size, num_pages, max_blocks, window;
    int keep_first;   // under a window: the request's first keys that stay visible (0: none)
    int page_shift;   // log2 of page_size if that is a power of two, else -1
    int split_tiles;  // > 0: the grid is pairs of CTAs (a cluster of two per tile record); a tile with at least this many key tiles is shared by its pair
    float scale_log2;
    int* status;
};

constexpr int kTaValues = 128;     // channels of a value head in the kernel with a thread a row

struct TaShared {
    static constexpr int kQBytes = kTaRows * kTaChannels * 2;          // 16 KB
    static constexpr int kPBytes = kTaRows * kTaKeys * 2;              // 16 KB
    static constexpr int kKeyBytes = kTaKeys * kTaChannels * 2;        // 8 KB: four boxes of 16 rows
    static constexpr int kValueBox = kTaValues * 32;                   // kTaValues channels x 16 keys
    static constexpr int kValueBytes = 4 * kValueBox;
    static constexpr int kStageBytes = kKeyBytes + kValueBytes;
    static constexpr int kBytes = kQBytes + kPBytes + 2 * kStageBytes + 1024 /* alignment */ + 256 /* barriers */;
    static constexpr int kColumns = 256;   // of tensor memory: scores, output
};

__device__ __forceinline__ void tma_load_3d(void* destination, const CUtensorMap* map, int x, int y, int z, uint64_t* barrier) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_address(destination)), "l"(map), "r"(smem_address(barrier)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* destination, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* barrier) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_address(destination)), "l"(map), "r"(smem_address(barrier)), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}

// Descriptor of a K-major tile with 32-byte swizzle: rows of 32 bytes (16 keys), groups of 8 rows 256 bytes apart.
__device__ __forceinline__ uint64_t value_box_descriptor(const void* tile) {
    const uint64_t address = smem_address(tile);
    return ((address & 0x3FFFFull) >> 4) | (1ull << 16) | (static_cast<uint64_t>(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float exp2_hardware(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// grid (tile records x K/V heads, 1, parts of a record), 192 threads: the records with most keys, of all heads, start first.
__global__ void __launch_bounds__(kTaThreads, 2)   // two CTAs per SM: one's softmax runs under the other's products
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                         const TaParams p) {
    using Shared = TaShared;
    extern __shared__ unsigned char raw_shared[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_shared) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* q_tile = base;
    unsigned char* p_tile = base + Shared::kQBytes;
    unsigned char* stages = p_tile + Shared::kPBytes;
    uint64_t* barriers = reinterpret_cast<uint64_t*>(stages + 2 * Shared::kStageBytes);
    uint64_t* q_full = barriers;
    // Keys and values have barriers of their own: a stage's keys are free again as soon as S = Q K^T of
    // their tile is done, a whole softmax before its values are, and the keys of the tile after next
    // are then on their way that much earlier (with one barrier for both, the next tile's S waited
    // 0.7 us for its keys in every turn of the loop).
    uint64_t* k_full = barriers + 1;     // [2]
    uint64_t* k_free = barriers + 3;     // [2]
    uint64_t* v_full = barriers + 14;    // [2]
    uint64_t* v_free = barriers + 16;    // [2]
    uint64_t* s_ready = barriers + 5;
    uint64_t* p_ready = barriers + 6;
    uint64_t* pv_done = barriers + 7;
    uint64_t* s_free = barriers + 8;     // every softmax thread has read its row of scores for the last time
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(barriers + 9);
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int heads_per_group = p.num_heads / p.num_groups;
    const int index = gridDim.x - 1 - blockIdx.x, record = index / p.num_groups;   // listed in the order of the tokens: the last ones of a prompt see the most keys
    const int group = index % p.num_groups, value_group = group / p.keys_per_value;
    const int first_token = p.tiles[2 * record] + p.tokens_per_cta * blockIdx.z;
    const int count = min(p.tokens_per_cta, p.tiles[2 * record + 1] - p.tokens_per_cta * static_cast<int>(blockIdx.z));
    if (count <= 0) return;   // the whole CTA: nothing has been set up yet
    const int segment = p.token_segment[first_token];
    const int first_position = p.positions[first_token], last_position = first_position + count - 1;
    const int first_visible = p.window > 0 ? max(0, first_position - p.window + 1) : 0;   // of the tile's first token
    // The 64-key tiles the CTA walks, counted through: those of the kept first keys, then those from the window's first
    // key on (one run from key 0 where the two meet); key0_of() gives the first key of the CTA's tile-th tile.
    int window_begin = (first_visible / kTaKeys) * kTaKeys;
    const int kept_wanted = (p.keep_first + kTaKeys - 1) / kTaKeys;
    int kept_tiles = 0;
    if (kept_wanted > 0) {
        if (kept_wanted < window_begin / kTaKeys) kept_tiles = kept_wanted;
        else window_begin = 0;
    }
    const int num_key_tiles = kept_tiles + (last_position - window_begin) / kTaKeys + 1;
    auto key0_of = [&](int tile) { return tile < kept_tiles ? tile * kTaKeys : window_begin + (tile - kept_tiles) * kTaKeys; };

    if (threadIdx.x == 0) {
        barrier_init(q_full, 1);
        for (int s = 0; s < 2; ++s) {
            barrier_init(&k_full[s], 1);
            barrier_init(&k_free[s], 1);
            barrier_init(&v_full[s], 1);
            barrier_init(&v_free[s], 1);
        }
        barrier_init(s_ready, 1);
        barrier_init(p_ready, 4);   // one arrival per softmax warp
        barrier_init(pv_done, 1);
        barrier_init(s_free, 4);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(tmem_slot)), "r"(Shared::kColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The out-projection that follows may ask for its weights meanwhile: it takes tensor memory of its own, so only now that this
    // CTA has its share (and launched early itself, it reads what the kernel before writes from here on).
    wait_for_previous_kernel();
    allow_next_kernel();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_scores = tmem_base, tmem_output = tmem_base + kTaKeys;

    if (warp == 0) {
        // Producer: the warp's first four lanes take one block of 16 keys each (its place in the block
        // table, its two boxes), so a tile costs the scheduler a quarter of the instructions one lane
        // would need; the other lanes idle along.
        if (lane == 0) {
            barrier_expect(q_full, static_cast<uint32_t>(p.tokens_per_cta * heads_per_group * kTaChannels * 2));
            tma_load_3d(q_tile, &map_q, 0, group * heads_per_group, first_token, q_full);
        }
        bool bad = false;
        // Blocks of 16 keys that some token of the tile sees and that have a page; the others are not
        // loaded (their scores are masked and their values cleared by the softmax warps).  A tile's entries
        // of the block table are read one tile ahead, so that the read's latency is not between a freed
        // stage and its next boxes.
        auto look_up = [&](int tile, int& page, int& offset) {
            page = -1;
            offset = 0;
            const int block_first = key0_of(tile) + 16 * lane;
            if (lane < 4 && tile < num_key_tiles && (block_first + 15 >= first_visible || block_first < p.keep_first) && block_first <= last_position) {
                const int column = p.page_shift >= 0 ? block_first >> p.page_shift : block_first / p.page_size;
                const int entry = column < p.max_blocks ? p.block_table[static_cast<size_t>(segment) * p.max_blocks + column] : -1;
                if (entry >= 0 && entry < p.num_pages) {
                    page = entry;
                    offset = block_first - column * p.page_size;
                } else {
                    bad = true;
                }
            }
        };
        int page, offset;
        look_up(0, page, offset);
        for (int tile = 0; tile < num_key_tiles; ++tile) {
            const int s = tile & 1;
            unsigned char* keys = stages + s * Shared::kStageBytes;
            unsigned char* values = keys + Shared::kKeyBytes;
            const int this_page = page, this_offset = offset;
            look_up(tile + 1, page, offset);
            const uint32_t blocks = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, this_page >= 0)));
            if (tile >= 2 && !__all_sync(0xffffffffu, barrier_wait_parked(&k_free[s], ((tile >> 1) - 1) & 1))) {
                atomicExch(&failed, 1);
                break;
            }
            if (lane == 0) barrier_expect(&k_full[s], 2048u * blocks);
            if (this_page >= 0) tma_load_4d(keys + lane * 2048, &map_k, 0, group, this_offset, this_page, &k_full[s]);
            if (tile >= 2 && !__all_sync(0xffffffffu, barrier_wait_parked(&v_free[s], ((tile >> 1) - 1) & 1))) {
                atomicExch(&failed, 1);
                break;
            }
            if (lane == 0) barrier_expect(&v_full[s], static_cast<uint32_t>(Shared::kValueBox) * blocks);
            if (this_page >= 0) tma_load_4d(values + lane * Shared::kValueBox, &map_v, this_offset, 0, value_group, this_page, &v_full[s]);
        }
        if (__any_sync(0xffffffffu, bad) && lane == 0) report_error(p.status, kBadPage);
    } else if (warp == 1 && lane == 0) {
        // Product issuer.  It waits parked: CTAs' issuers polling on one scheduler take the ALU slots
        // of the softmax warps there, and every tile waits for its slowest softmax warp.
        constexpr uint32_t idesc_scores = instruction_descriptor<kTaKeys>(), idesc_output = instruction_descriptor<kTaValues>();   // N = 64 keys; 128 channels
        bool ok = barrier_wait(q_full, 0);
        if (!ok) atomicExch(&failed, 1);
        const uint64_t desc_q = tile_descriptor(q_tile), desc_p = tile_descriptor(p_tile);
        // S = Q K^T of tile t + 1 is issued as soon as the softmax threads have read S of tile t for the
        // last time, before their P is complete: it runs under the rest of their work, and the scores of
        // the next tile are there when they come for them.
        auto issue_scores = [&](int tile) {
            if (!barrier_wait_parked(&k_full[tile & 1], (tile >> 1) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t desc_k = tile_descriptor(stages + (tile & 1) * Shared::kStageBytes);
#pragma unroll
            for (int k = 0; k < kTaChannels / 16; ++k) mma_f16(tmem_scores, desc_q + 2 * k, desc_k + 2 * k, idesc_scores, k > 0);   // padded channels add zeros
            mma_commit(s_ready);
            mma_commit(&k_free[tile & 1]);
            return true;
        };
        if (ok && !issue_scores(0)) {
            atomicExch(&failed, 1);
            ok = false;
        }
        for (int tile = 0; tile < num_key_tiles && ok; ++tile) {
            const int s = tile & 1;
            unsigned char* values = stages + s * Shared::kStageBytes + Shared::kKeyBytes;
            if (tile + 1 < num_key_tiles) {
                if (!barrier_wait_parked(s_free, tile & 1)) {
                    atomicExch(&failed, 1);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!issue_scores(tile + 1)) {
                    atomicExch(&failed, 1);
                    break;
                }
            }
            if (!barrier_wait_parked(p_ready, tile & 1) || !barrier_wait_parked(&v_full[s], (tile >> 1) & 1)) {
                atomicExch(&failed, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int k = 0; k < kTaKeys / 16; ++k) mma_f16(tmem_output, desc_p + 2 * k, value_box_descriptor(values + k * Shared::kValueBox), idesc_output, tile > 0 || k > 0);
            mma_commit(&v_free[s]);
            mma_commit(pv_done);
        }
    } else if (warp >= 2) {
        // A thread per row.  Row r is token r / heads_per_group of the CTA's tokens, query head r % heads_per_group.
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const int token_local = row / heads_per_group, head_local = row - token_local * heads_per_group;
        const bool valid_row = token_local < count;
        const int row_position = first_position + token_local;
        const int row_first = p.window > 0 ? max(0, row_position - p.window + 1) : 0;
        const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16;
        float reference = -INFINITY, row_sum = 0.0f;
        bool ok = true;
        // The warp's lanes leave the loop together or not at all: what follows a wait is warp-wide.
        // They wait parked in hardware: polling warps would take the ALU slots that the other CTA's softmax needs.
        auto wait_together = [](uint64_t* barrier, uint32_t parity) {
            // every lane waits on the same barrier (one instruction per warp, as for one lane; no exchange after it)
            return __all_sync(0xffffffffu, barrier_wait_parked(barrier, parity));
        };
        for (int tile = 0; tile < num_key_tiles; ++tile) {
            const int s = tile & 1;
            const int key0 = key0_of(tile);
            if (!wait_together(s_ready, tile & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // Only tiles that reach past some token's own position, or before some token's window, need masks.
            const bool needs_mask = key0 + kTaKeys - 1 > first_position || (p.window > 0 && key0 < last_position - p.window + 1);
            // The row is read twice, 32 scores at a time (once for its maximum, once for its terms): a
            // thread then needs half the registers.  Both passes exist with and
            // without the mask, chosen by one branch per tile: with the test inside the loops the mask's
            // comparisons ran for every score of every tile, and the ALU pipe was the kernel's limit.
            float tops[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            auto row_maximum = [&](auto masked) {
                constexpr bool kMasked = decltype(masked)::value;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t raw[32];
                    tmem_load_32(tmem_scores + lane_field + 32 * half, raw);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float pair[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            pair[e] = __uint_as_float(raw[i + e]);
                            if constexpr (kMasked) {
                                const int key = key0 + 32 * half + i + e;
                                if ((key < row_first && key >= p.keep_first) || key > row_position) pair[e] = -INFINITY;
                            }
                        }
                        tops[(i >> 1) & 3] = max3(tops[(i >> 1) & 3], pair[0], pair[1]);   // one instruction for two scores
                    }
                }
            };
            if (needs_mask) row_maximum(std::true_type{});
            else row_maximum(std::false_type{});
            float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
            // `reference` is the exponent the row's terms are taken relative to; it follows the row's maximum
            // only when that has grown by more than 2^8, so that the output is rarely rescaled.
            top *= p.scale_log2;   // the scale is positive
            const float moved = top > reference + kTaMaxSlack ? top : reference;
            const float shift = moved == -INFINITY ? 0.0f : moved;   // a row that has seen no key yet: every term below is 2^-inf = 0
            const float rescale = exp2_hardware(reference - shift);
            reference = moved;
            if (tile > 0) {
                // The products of the tile before have finished: P may be overwritten and O rescaled.
                if (!wait_together(pv_done, (tile - 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (__any_sync(0xffffffffu, rescale != 1.0f)) {
#pragma unroll
                    for (int half = 0; half < kTaValues / 32; ++half) {
                        uint32_t held[32];
                        tmem_load_32(tmem_output + lane_field + 32 * half, held);
#pragma unroll
                        for (int i = 0; i < 32; ++i) held[i] = __float_as_uint(__uint_as_float(held[i]) * rescale);
                        tmem_store_32(tmem_output + lane_field + 32 * half, held);
                    }
                }
            }
            float partials[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint64_t sums2[4] = {0ull, 0ull, 0ull, 0ull};   // pairs of 0.0f
            const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2), shift2 = pack2(-shift, -shift);
            const uint32_t p_row = smem_address(p_tile) + static_cast<uint32_t>(row) * 128u;   // a 32-bit shared-memory address: plain shared stores
            auto row_terms = [&](auto masked) {
                constexpr bool kMasked = decltype(masked)::value;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t raw[32];
                    tmem_load_32(tmem_scores + lane_field + 32 * half, raw);
                    if (half == 1) {
                        // the row's scores are in registers: the next tile's may overwrite them
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) barrier_arrive(s_free);
                    }
#pragma unroll
                    for (int chunk = 0; chunk < 4; ++chunk) {
                        uint4 packed;
                        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float terms[2];
                            if constexpr (kMasked) {
#pragma unroll
                                for (int e = 0; e < 2; ++e) {
                                    const int index = 8 * chunk + 2 * i + e;
                                    float score = __uint_as_float(raw[index]);
                                    const int key = key0 + 32 * half + index;
                                    if ((key < row_first && key >= p.keep_first) || key > row_position) score = -INFINITY;
                                    terms[e] = exp2_hardware(fmaf(score, p.scale_log2, -shift));
                                }
                                partials[i] += terms[0] + terms[1];
                            } else {
                                // two scores per instruction: the scaled difference, and the running sums
                                const int index = 8 * chunk + 2 * i;
                                float low, high;
                                unpack2(fma2(pack2(__uint_as_float(raw[index]), __uint_as_float(raw[index + 1])), scale2, shift2), low, high);
                                terms[0] = exp2_hardware(low);
                                terms[1] = exp2_hardware(high);
                                sums2[i] = add2(sums2[i], pack2(terms[0], terms[1]));
                            }
                            pairs[i] = __floats2bfloat162_rn(terms[0], terms[1]);
                        }
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"   // the operand's 128-byte swizzle
                                     ::"r"(p_row + static_cast<uint32_t>(((4 * half + chunk) ^ (row & 7)) << 4)), "r"(packed.x), "r"(packed.y), "r"(packed.z), "r"(packed.w)
                                     : "memory");
                    }
                }
            };
            if (needs_mask) row_terms(std::true_type{});
            else row_terms(std::false_type{});
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float low, high;
                unpack2(sums2[i], low, high);
                partials[i] += low + high;
            }
            const float partial = (partials[0] + partials[1]) + (partials[2] + partials[3]);
            row_sum = row_sum * rescale + partial;
            if (needs_mask) {
                // Keys outside [first visible, last position] of the tile hold whatever was left in the page,
                // or were not loaded at all: clear their values, since a zero probability does not silence
                // a non-finite value in the product.  128 channels x 64 keys, a thread per channel.
                if (!wait_together(&v_full[s], (tile >> 1) & 1)) {
                    ok = false;
                    break;
                }
                unsigned char* values = stages + s * Shared::kStageBytes + Shared::kKeyBytes;
                constexpr int kKeysHere = kTaKeys * kTaValues / kTaRows;
                const int channel = row % kTaValues, key_part = row / kTaValues;
                for (int i = 0; i < kKeysHere; ++i) {
                    const int local_key = kKeysHere * key_part + i, key = key0 + local_key;
                    if ((key < first_visible && key >= p.keep_first) || key > last_position) {
                        const int block = local_key >> 4, in_block = local_key & 15;
                        // 32-byte swizzle: the 16-byte half of a 32-byte row is flipped in rows 4-7 of every 8
                        unsigned char* address = values + block * Shared::kValueBox + channel * 32 + ((((in_block >> 3) ^ (channel >> 2)) & 1) << 4) + (in_block & 7) * 2;
                        *reinterpret_cast<__nv_bfloat16*>(address) = __float2bfloat16_rn(0.0f);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // P and the cleared values, seen by the products
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();   // every lane's P, fenced, before the warp's one arrival
            if (lane == 0) barrier_arrive(p_ready);
        }
        if (ok && !wait_together(pv_done, (num_key_tiles - 1) & 1)) ok = false;
        if (!ok) atomicExch(&failed, 1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inverse = row_sum > 0.0f ? 1.0f / row_sum : 0.0f;
        const size_t out_row = (static_cast<size_t>(first_token + token_local) * p.num_heads + group * heads_per_group + head_local) * kTaValues;
#pragma unroll
        for (int half = 0; half < kTaValues / 32; ++half) {
            uint32_t held[32];
            tmem_load_32(tmem_output + lane_field + 32 * half, held);
            if (valid_row && ok) {
#pragma unroll
                for (int chunk = 0; chunk < 4; ++chunk) {
                    const int channel = 32 * half + 8 * chunk;
                    float values[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) values[i] = __uint_as_float(held[8 * chunk + i]) * inverse;
                    if (p.out_float) {
                        float4* destination = reinterpret_cast<float4*>(static_cast<float*>(p.out) + out_row + channel);
                        destination[0] = make_float4(values[0], values[1], values[2], values[3]);
                        destination[1] = make_float4(values[4], values[5], values[6], values[7]);
                    } else {
                        uint4 packed;
                        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                        for (int i = 0; i < 4; ++i) pairs[i] = __floats2bfloat162_rn(values[2 * i], values[2 * i + 1]);
                        *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + out_row + channel) = packed;
                    }
                }
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
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Shared::kColumns) : "memory");
    }
}

// ---- value heads of 64 channels: two threads a row
// The same roles, products and tiles, with what fits beside 64 value channels: two tiles of scores, the probabilities over the scores they came from (A of the second
// product from tensor memory), four stages, and two CTAs a multiprocessor with eight softmax warps each.  A row's two threads have 32 keys of
// every tile each, with an exponent, a sum and an output of their own (O += P V of keys 0 to 31 and of 32 to 63 go to different columns): they exchange
// nothing until the end, where the two halves are added like the shares of two CTAs.
// What bounds it: a tile's products and what lies between them (0.5 us a tile and multiprocessor without any softmax: a batch of products takes about 250
// cycles beside its own), then the exponential unit (0.28 us).  Measured, prompts of 2,048 tokens, 32 heads over 8: 43 us (56 with a thread a row and three
// CTAs a multiprocessor, 45 of them after the records with most keys went first); 16 heads over 4 under a window of 1,024 19 us (29); 300 behind 3,000, pairs of
// CTAs 33 us (45).  Tried: tiles of 128 keys, the even and the odd ones on four warps each, one CTA a multiprocessor: 43 us behind 4,000 keys (52), but 66 us for a
// prompt of 2,048, whose CTAs' starts and ends nothing covers.
constexpr int kThThreads = 320, kThStages = 4;
constexpr int kThKeyBytes = kTaKeys * kTaChannels * 2, kThValueBox = 64 * 32, kThStageBytes = kThKeyBytes + 4 * kThValueBox;
constexpr int kThQBytes = kTaRows * kTaChannels * 2;
constexpr int kThBytes = kThStages * kThStageBytes + kThQBytes + 4 * kTaRows * 4 /* exponents, sums */ + 256 /* barriers */ + 1024 /* alignment */;

// grid (tile records x K/V heads (PAIRED: x 2), 1, parts of a record): the records with most keys, of all heads, start first.
template <bool PAIRED>
__global__ void __launch_bounds__(kThThreads, 2)
attention_tcgen05_halves_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const TaParams p) {
    extern __shared__ unsigned char raw_shared[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_shared) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* stages = base;
    unsigned char* q_tile = stages + kThStages * kThStageBytes;
    float* halves = reinterpret_cast<float*>(q_tile + kThQBytes);   // [exponent, sum][half][128 rows]
    uint64_t* barriers = reinterpret_cast<uint64_t*>(halves + 4 * kTaRows);
    uint64_t* q_full = barriers;
    uint64_t* full = barriers + 1;                  // [kThStages]
    uint64_t* free_again = full + kThStages;        // [kThStages]
    uint64_t* s_full = free_again + kThStages;      // [2]
    uint64_t* p_full = s_full + 2;                  // [2]
    uint64_t* pv_done = p_full + 2;                 // [2]
    uint64_t* rows_met = pv_done + 2;               // [4]: both warps of 32 rows have left their exponents and sums
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rows_met + 4);
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int heads_per_group = p.num_heads / p.num_groups;
    const int index = static_cast<int>(PAIRED ? (gridDim.x - 1 - blockIdx.x) >> 1 : gridDim.x - 1 - blockIdx.x), record = index / p.num_groups;
    const int group = index % p.num_groups, value_group = group / p.keys_per_value;
    // Two CTAs (a cluster) stand behind every tile record and head: where the tile sees many keys,
    // each takes half of them and CTA 0 merges the halves at the end (CTA 1 sends its output, exponent and sum
    // into CTA 0's shared memory); where it sees few, CTA 1 leaves at once.  What bounds a launch of few tiles
    // is the chain of 64-key steps of its longest tile, and this halves it.
    const int rank = PAIRED ? static_cast<int>(cluster_rank()) : 0;
    const int first_token = p.tiles[2 * record] + p.tokens_per_cta * blockIdx.z;
    const int count = min(p.tokens_per_cta, p.tiles[2 * record + 1] - p.tokens_per_cta * static_cast<int>(blockIdx.z));
    if (count <= 0) return;   // the whole CTA (and its partner): nothing has been set up yet
    const int segment = p.token_segment[first_token];
    const int first_position = p.positions[first_token], last_position = first_position + count - 1;
    const int first_visible = p.window > 0 ? max(0, first_position - p.window + 1) : 0;   // of the tile's first token
    int window_begin = (first_visible / kTaKeys) * kTaKeys;
    const int kept_wanted = (p.keep_first + kTaKeys - 1) / kTaKeys;
    int kept_tiles = 0;
    if (kept_wanted > 0) {
        if (kept_wanted < window_begin / kTaKeys) kept_tiles = kept_wanted;
        else window_begin = 0;
    }
    int tiles = kept_tiles + (last_position - window_begin) / kTaKeys + 1, first_listed = 0;
    const bool shared_tile = PAIRED && tiles >= p.split_tiles;
    if (PAIRED && !shared_tile && rank == 1) return;   // CTA 0 does this tile alone and uses no cluster barrier
    if (shared_tile) {
        const int lower = tiles / 2;
        if (rank == 1) first_listed = lower;
        tiles = rank == 0 ? lower : tiles - lower;
    }
    auto key0_of = [&](int tile) {
        const int listed = first_listed + tile;
        return listed < kept_tiles ? listed * kTaKeys : window_begin + (listed - kept_tiles) * kTaKeys;
    };

    if (threadIdx.x == 0) {
        barrier_init(q_full, 1);
        for (int s = 0; s < kThStages; ++s) {
            barrier_init(&full[s], 1);
            barrier_init(&free_again[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            barrier_init(&s_full[s], 1);
            barrier_init(&p_full[s], 8);   // one arrival per softmax warp
            barrier_init(&pv_done[s], 1);
        }
        for (int s = 0; s < 4; ++s) barrier_init(&rows_met[s], 2);
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
    // The out-projection that follows may ask for its weights meanwhile: it takes tensor memory of its own, so only now that this
    // CTA has its share (and launched early itself, it reads what the kernel before writes from here on).
    wait_for_previous_kernel();
    allow_next_kernel();
    const uint32_t tmem_output = *tmem_slot, tmem_scores = tmem_output + 128;   // two halves of 64 columns, two tiles of 64 columns

    if (warp == 9) {
        // Lanes 0 to 3: a tile's blocks of 16 keys, lanes 4 to 7: their values, a box each.
        if (lane == 0) {
            barrier_expect(q_full, static_cast<uint32_t>(p.tokens_per_cta * heads_per_group * kTaChannels * 2));
            tma_load_3d(q_tile, &map_q, 0, group * heads_per_group, first_token, q_full);
        }
        // Blocks that some token of the tile sees and that have a page; the others are not loaded (their scores are masked and their values cleared by the
        // softmax warps).  A tile's entries of the block table are read one tile ahead.
        bool bad = false, ok = true;
        auto look_up = [&](int tile, int& page, int& offset) {
            page = -1;
            offset = 0;
            if (lane >= 8 || tile >= tiles) return;
            const int first = key0_of(tile) + 16 * (lane & 3);
            if ((first + 15 < first_visible && first >= p.keep_first) || first > last_position) return;
            const int column = p.page_shift >= 0 ? first >> p.page_shift : first / p.page_size;
            const int entry = column < p.max_blocks ? p.block_table[static_cast<size_t>(segment) * p.max_blocks + column] : -1;
            if (entry >= 0 && entry < p.num_pages) page = entry, offset = first - column * p.page_size;
            else bad = true;
        };
        int page, offset;
        look_up(0, page, offset);
        for (int tile = 0; tile < tiles; ++tile) {
            const int s = tile % kThStages, this_page = page, this_offset = offset;
            look_up(tile + 1, page, offset);
            const uint32_t boxes = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, this_page >= 0)));
            if (tile >= kThStages && !__all_sync(0xffffffffu, barrier_wait_parked(&free_again[s], (tile / kThStages - 1) & 1))) {
                ok = false;
                break;
            }
            if (lane == 0) barrier_expect(&full[s], 2048u * boxes);
            __syncwarp();
            unsigned char* keys = stages + s * kThStageBytes;
            if (this_page >= 0) {
                if (lane < 4) tma_load_4d(keys + lane * 2048, &map_k, 0, group, this_offset, this_page, &full[s]);
                else tma_load_4d(keys + kThKeyBytes + (lane - 4) * kThValueBox, &map_v, this_offset, 0, value_group, this_page, &full[s]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicExch(&failed, 1);
        if (__any_sync(0xffffffffu, bad) && lane == 0) report_error(p.status, kBadPage);
    } else if (warp == 8) {
        if (lane == 0) {
            constexpr uint32_t idesc = instruction_descriptor<64>();   // 64 keys; 64 channels
            const uint64_t desc_q = tile_descriptor(q_tile);
            auto issue_scores = [&](int tile) {
                const int s = tile % kThStages;
                if (!barrier_wait_parked(&full[s], (tile / kThStages) & 1)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t desc_k = tile_descriptor(stages + s * kThStageBytes);
#pragma unroll
                for (int k = 0; k < kTaChannels / 16; ++k) mma_f16(tmem_scores + (tile & 1) * kTaKeys, desc_q + 2 * k, desc_k + 2 * k, idesc, k > 0);   // padded channels add zeros
                mma_commit(&s_full[tile & 1]);
                return true;
            };
            bool ok = barrier_wait(q_full, 0);
            for (int tile = 0; tile < min(2, tiles) && ok; ++tile) ok = issue_scores(tile);
            for (int tile = 0; tile < tiles && ok; ++tile) {
                if (!barrier_wait_parked(&p_full[tile & 1], (tile >> 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int s = tile % kThStages;
                const unsigned char* values = stages + s * kThStageBytes + kThKeyBytes;
                const uint32_t weights = tmem_scores + (tile & 1) * kTaKeys;   // of the first 32 keys in columns 0 to 15, of the others from column 32 on
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma_f16_from_tmem(tmem_output + (k >> 1) * 64, weights + (k >> 1) * 32 + (k & 1) * 8, value_box_descriptor(values + k * kThValueBox), idesc, tile > 0 || (k & 1));
                mma_commit(&free_again[s]);
                mma_commit(&pv_done[tile & 1]);
                if (tile + 2 < tiles) ok = issue_scores(tile + 2);
            }
            if (!ok) atomicExch(&failed, 1);
        }
        __syncwarp();
    } else {
        // Row r is token r / heads_per_group of the CTA's tokens, query head r % heads_per_group.
        const int quarter = warp & 3, half = warp >> 2;   // of tensor memory's lanes; of a tile's keys
        const int row = quarter * 32 + lane;
        const int token_local = row / heads_per_group, head_local = row - token_local * heads_per_group;
        const bool valid_row = token_local < count, valid_warp = quarter * 32 < count * heads_per_group;
        const int row_position = first_position + token_local;
        const int row_first = p.window > 0 ? max(0, row_position - p.window + 1) : 0;
        const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16, own_output = tmem_output + 64 * half + lane_field;
        float reference = -INFINITY, row_sum = 0.0f;
        bool ok = true;
        // every lane waits parked in hardware on the same barrier; they leave the loop together or not at all
        auto wait_together = [](uint64_t* barrier, uint32_t parity) { return __all_sync(0xffffffffu, barrier_wait_parked(barrier, parity)); };
        for (int tile = 0; tile < tiles; ++tile) {
            const int s = tile & 1, tile_key = key0_of(tile), key0 = tile_key + 32 * half;
            const uint32_t scores = tmem_scores + s * kTaKeys + 32 * half + lane_field;
            if (!wait_together(&s_full[s], (tile >> 1) & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // Only tiles that reach past some token's own position, or before some token's window, need masks.
            const bool needs_mask = tile_key + kTaKeys - 1 > first_position || (p.window > 0 && tile_key < last_position - p.window + 1);
            if (valid_warp) {   // (rows that are none are neither worked on nor stored: what lies in their place reaches no other)
                uint32_t raw[32];
                tmem_load_32_together(scores, raw);
                if (needs_mask) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = key0 + i;
                        if ((key < row_first && key >= p.keep_first) || key > row_position) raw[i] = 0xff800000u;   // minus infinity
                    }
                }
                float tops[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int i = 0; i < 32; i += 2) tops[(i >> 1) & 3] = max3(tops[(i >> 1) & 3], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]));   // one instruction for two scores
                const float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3])) * p.scale_log2;   // the scale is positive
                // `reference` is the exponent the half row's terms are taken relative to; it follows its maximum
                // only when that has grown by more than 2^8, so that the output is rarely rescaled.
                const float moved = top > reference + kTaMaxSlack ? top : reference;
                const float shift = moved == -INFINITY ? 0.0f : moved;   // nothing seen yet: every term below is 2^-inf = 0
                const float rescale = exp2_hardware(reference - shift);
                reference = moved;
                if (tile > 0 && __any_sync(0xffffffffu, rescale != 1.0f)) {
                    // (the products before the last are done, or these scores would not be there: the barrier's phase is the last's or the one after)
                    if (!wait_together(&pv_done[s ^ 1], ((tile - 1) >> 1) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                    for (int c = 0; c < 64; c += 16) {
                        uint32_t held[16];
                        tmem_load_16(own_output + c, held);
#pragma unroll
                        for (int i = 0; i < 16; ++i) held[i] = __float_as_uint(__uint_as_float(held[i]) * rescale);
                        tmem_store_16(own_output + c, held);
                    }
                }
                uint64_t sums2[2] = {0ull, 0ull};   // pairs of 0.0f
                const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2), shift2 = pack2(-shift, -shift);
                uint32_t packed[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    // two scores per instruction: the scaled difference, and the running sums
                    float low, high;
                    unpack2(fma2(pack2(__uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1])), scale2, shift2), low, high);
                    const float terms[2] = {exp2_hardware(low), exp2_hardware(high)};
                    sums2[i & 1] = add2(sums2[i & 1], pack2(terms[0], terms[1]));
                    const __nv_bfloat162 pair = __floats2bfloat162_rn(terms[0], terms[1]);
                    packed[i] = *reinterpret_cast<const uint32_t*>(&pair);
                }
                tmem_store_16(scores, packed);   // over this thread's own scores
                float low, high;
                unpack2(add2(sums2[0], sums2[1]), low, high);
                row_sum = row_sum * rescale + (low + high);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            if (needs_mask) {
                // Keys outside [first visible, last position] of the tile hold whatever was left in the page,
                // or were not loaded at all: clear their values, since a zero probability does not silence
                // a non-finite value in the product.  64 channels x 64 keys, four threads per channel.
                if (!wait_together(&full[tile % kThStages], (tile / kThStages) & 1)) {   // (long over)
                    ok = false;
                    break;
                }
                const int channel = threadIdx.x & 63, block = threadIdx.x >> 6;
                unsigned char* box = stages + (tile % kThStages) * kThStageBytes + kThKeyBytes + block * kThValueBox + channel * 32;
                for (int i = 0; i < 16; ++i) {
                    const int key = tile_key + 16 * block + i;
                    // 32-byte swizzle: the 16-byte half of a 32-byte row is flipped in rows 4-7 of every 8
                    if ((key < first_visible && key >= p.keep_first) || key > last_position)
                        *reinterpret_cast<__nv_bfloat16*>(box + ((((i >> 3) ^ (channel >> 2)) & 1) << 4) + (i & 7) * 2) = __float2bfloat16_rn(0.0f);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // seen by the products
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();   // every lane's, before the warp's one arrival
            if (lane == 0) barrier_arrive(&p_full[s]);
        }
        if (ok && tiles > 0 && !wait_together(&pv_done[(tiles - 1) & 1], ((tiles - 1) >> 1) & 1)) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // the row's halves: an exponent and a sum for both, and what each output counts
        halves[half * kTaRows + row] = reference;
        halves[(2 + half) * kTaRows + row] = row_sum;
        __syncwarp();
        if (lane == 0) barrier_arrive(&rows_met[quarter]);
        if (!ok || !wait_together(&rows_met[quarter], 0)) {
            ok = false;
            atomicExch(&failed, 1);
        }
        const float first_reference = halves[row], second_reference = halves[kTaRows + row];
        float top = fmaxf(first_reference, second_reference);
        float weights[2] = {top == -INFINITY ? 0.0f : exp2_hardware(first_reference - top), top == -INFINITY ? 0.0f : exp2_hardware(second_reference - top)};
        row_sum = halves[2 * kTaRows + row] * weights[0] + halves[3 * kTaRows + row] * weights[1];
        const int channel0 = 32 * half;   // this thread's channels of the row's 64
        float values[32];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            uint32_t first[16], second[16];
            tmem_load_16(tmem_output + lane_field + channel0 + 16 * part, first);
            tmem_load_16(tmem_output + 64 + lane_field + channel0 + 16 * part, second);
#pragma unroll
            for (int i = 0; i < 16; ++i) values[16 * part + i] = __uint_as_float(first[i]) * weights[0] + __uint_as_float(second[i]) * weights[1];
        }
        // A tile shared by two CTAs: when both have been through their keys (first cluster barrier: CTA 0's
        // shared memory is free), CTA 1 sends its unnormalised output row, exponent and sum there; after the
        // second barrier CTA 0 merges.  The other warps of both CTAs meet the same barriers below.
        float* const received = reinterpret_cast<float*>(stages);               // [128 rows][64]
        float* const received_scalars = reinterpret_cast<float*>(q_tile);       // [128 rows][2]
        if (shared_tile) cluster_sync();
        if (shared_tile && rank == 1) {
            const uint32_t remote_row = cluster_address(received + row * 64 + channel0, 0), remote_scalars = cluster_address(received_scalars + row * 2, 0);
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote_row + static_cast<uint32_t>(i * 4)), "f"(values[i]), "f"(values[i + 1]),
                             "f"(values[i + 2]), "f"(values[i + 3])
                             : "memory");
            if (half == 0) asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(remote_scalars), "f"(top), "f"(row_sum) : "memory");
        }
        if (shared_tile) cluster_sync();
        if (rank == 0) {
            if (shared_tile) {
                const float other_top = received_scalars[row * 2], most = fmaxf(top, other_top);
                const float mine = most == -INFINITY ? 0.0f : exp2_hardware(top - most), theirs = most == -INFINITY ? 0.0f : exp2_hardware(other_top - most);
                row_sum = row_sum * mine + received_scalars[row * 2 + 1] * theirs;
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 other = *reinterpret_cast<const float4*>(received + row * 64 + channel0 + i);
                    values[i] = values[i] * mine + other.x * theirs, values[i + 1] = values[i + 1] * mine + other.y * theirs;
                    values[i + 2] = values[i + 2] * mine + other.z * theirs, values[i + 3] = values[i + 3] * mine + other.w * theirs;
                }
            }
            const float inverse = row_sum > 0.0f ? 1.0f / row_sum : 0.0f;
            if (valid_row && ok) {
                const size_t out_row = (static_cast<size_t>(first_token + token_local) * p.num_heads + group * heads_per_group + head_local) * 64 + channel0;
                if (p.out_float) {
                    float4* destination = reinterpret_cast<float4*>(static_cast<float*>(p.out) + out_row);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        destination[i] = make_float4(values[4 * i] * inverse, values[4 * i + 1] * inverse, values[4 * i + 2] * inverse, values[4 * i + 3] * inverse);
                } else {
                    uint4* destination = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + out_row);
#pragma unroll
                    for (int chunk = 0; chunk < 4; ++chunk) {
                        uint4 packed;
                        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                        for (int i = 0; i < 4; ++i) pairs[i] = __floats2bfloat162_rn(values[8 * chunk + 2 * i] * inverse, values[8 * chunk + 2 * i + 1] * inverse);
                        destination[chunk] = packed;
                    }
                }
            }
        }
    }
    if (shared_tile && warp >= 8) {
        // loader and issuer: the two cluster barriers of the softmax warps above
        cluster_sync();
        cluster_sync();
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

// A tensor map of bfloat16 elements with up to four dimensions (innermost first).
static bool make_paged_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes, const cuuint32_t* box,
                           CUtensorMapSwizzle swizzle) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint32_t element_strides[4] = {1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, static_cast<cuuint32_t>(rank), const_cast<void*>(base), dims, strides_bytes, box, element_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace lb

extern "C" {

// Same arguments as lb_attention_prefill plus the number of tokens in q, the size of a value head (0: head_dim), the number of
// value heads (0: num_groups; a divisor of them otherwise) and whether `out` is float32.  Returns 0, a CUDA error, -2 for
// sizes the kernel does not take (key heads beyond 64 channels or no multiples of 8, value heads of other than 64 or 128, page_size no multiple of 16, more than 128
// query heads per K/V head, a scale that is not positive, split tiles with heads other than 64, pointers not 16-byte aligned), -5 if no
// tensor map could be made.
int lb_attention_prefill_tcgen05(const void* q, const void* k_pages, const void* v_pages, void* out, const int* tiles, int num_tiles, int tokens,
                                 const int* positions, const int* token_segment, const int* block_table, int num_heads, int num_groups,
                                 int head_dim, int page_size, int num_pages, int max_blocks, float scale, int window, int split_tiles, int* status,
                                 cudaStream_t stream, int keep_first, int value_dim, int value_groups, int out_float) {
    // split_tiles > 0: a pair of CTAs per tile record; a tile that sees at least that many tiles of 64 keys is
    // shared by its pair (for launches of few tiles, which the longest tile's chain of keys bounds).
    if (num_tiles == 0 || tokens == 0) return 0;
    if (split_tiles < 0 || split_tiles == 1 || keep_first < 0) return -2;
    if (value_dim <= 0) value_dim = head_dim;
    if (value_groups <= 0) value_groups = num_groups;
    if (head_dim < 8 || head_dim > lb::kTaChannels || head_dim % 8 != 0 || (value_dim != 64 && value_dim != 128) || page_size % 16 != 0 || num_groups < 1 ||
        num_groups % value_groups != 0 || num_heads % num_groups != 0 || num_heads / num_groups > lb::kTaRows || !(scale > 0.0f))
        return -2;
    if (split_tiles > 0 && (head_dim != 64 || value_dim != 64)) return -2;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages) | reinterpret_cast<uintptr_t>(out)) & 15)
        return -2;
    const int heads_per_group = num_heads / num_groups;
    lb::TaParams p;
    p.out = out;
    p.keys_per_value = num_groups / value_groups;
    p.out_float = out_float;
    p.tiles = tiles;
    p.positions = positions;
    p.token_segment = token_segment;
    p.block_table = block_table;
    p.num_heads = num_heads;
    p.num_groups = num_groups;
    p.tokens_per_cta = lb::kTaRows / heads_per_group < lb::kTaTileTokens ? lb::kTaRows / heads_per_group : lb::kTaTileTokens;
    p.page_size = page_size;
    p.page_shift = -1;
    for (int shift = 0; shift < 31; ++shift)
        if ((1 << shift) == page_size) p.page_shift = shift;
    p.num_pages = num_pages;
    p.max_blocks = max_blocks;
    p.window = window;
    p.keep_first = window > 0 ? keep_first : 0;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.status = status;

    CUtensorMap map_q, map_k, map_v;
    {
        const cuuint64_t dims[3] = {static_cast<cuuint64_t>(head_dim), static_cast<cuuint64_t>(num_heads), static_cast<cuuint64_t>(tokens)};
        const cuuint64_t strides[2] = {static_cast<cuuint64_t>(head_dim) * 2, static_cast<cuuint64_t>(num_heads) * head_dim * 2};
        const cuuint32_t box[3] = {static_cast<cuuint32_t>(lb::kTaChannels), static_cast<cuuint32_t>(heads_per_group), static_cast<cuuint32_t>(p.tokens_per_cta)};
        if (!lb::make_paged_map(&map_q, q, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -5;
    }
    {
        const cuuint64_t dims[4] = {static_cast<cuuint64_t>(head_dim), static_cast<cuuint64_t>(num_groups), static_cast<cuuint64_t>(page_size),
                                    static_cast<cuuint64_t>(num_pages)};
        const cuuint64_t strides[3] = {static_cast<cuuint64_t>(head_dim) * 2, static_cast<cuuint64_t>(num_groups) * head_dim * 2,
                                       static_cast<cuuint64_t>(page_size) * num_groups * head_dim * 2};
        const cuuint32_t box[4] = {static_cast<cuuint32_t>(lb::kTaChannels), 1, 16, 1};
        if (!lb::make_paged_map(&map_k, k_pages, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -5;
    }
    {
        const cuuint64_t dims[4] = {static_cast<cuuint64_t>(page_size), static_cast<cuuint64_t>(value_dim), static_cast<cuuint64_t>(value_groups),
                                    static_cast<cuuint64_t>(num_pages)};
        const cuuint64_t strides[3] = {static_cast<cuuint64_t>(page_size) * 2, static_cast<cuuint64_t>(value_dim) * page_size * 2,
                                       static_cast<cuuint64_t>(value_groups) * value_dim * page_size * 2};
        const cuuint32_t box[4] = {16, static_cast<cuuint32_t>(value_dim), 1, 1};
        if (!lb::make_paged_map(&map_v, v_pages, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_32B)) return -5;
    }
    p.split_tiles = split_tiles;
    const unsigned parts = static_cast<unsigned>((lb::kTaTileTokens + p.tokens_per_cta - 1) / p.tokens_per_cta);
    if (value_dim == 128) {
        static lb::OncePerDevice configured;
        if (lb::allow_shared_memory(configured, lb::attention_tcgen05_kernel, lb::TaShared::kBytes) != cudaSuccess) return static_cast<int>(cudaGetLastError());
        return static_cast<int>(lb::launch_overlapped(lb::attention_tcgen05_kernel, dim3(static_cast<unsigned>(num_tiles) * num_groups, 1, parts), dim3(lb::kTaThreads),
                                                      lb::TaShared::kBytes, stream, map_q, map_k, map_v, p));
    }
    static lb::OncePerDevice configured, configured_paired;
    if (lb::allow_shared_memory(configured, lb::attention_tcgen05_halves_kernel<false>, lb::kThBytes) != cudaSuccess ||
        lb::allow_shared_memory(configured_paired, lb::attention_tcgen05_halves_kernel<true>, lb::kThBytes) != cudaSuccess)
        return static_cast<int>(cudaGetLastError());
    if (split_tiles == 0) {
        return static_cast<int>(lb::launch_overlapped(lb::attention_tcgen05_halves_kernel<false>, dim3(static_cast<unsigned>(num_tiles) * num_groups, 1, parts), dim3(lb::kThThreads), lb::kThBytes,
                                                      stream, map_q, map_k, map_v, p));
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2u * num_tiles * num_groups, 1, parts);
    config.blockDim = dim3(lb::kThThreads);
    config.dynamicSmemBytes = lb::kThBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = 2;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = lb::overlap_launches() ? 1 : 0;
    config.attrs = attribute;
    config.numAttrs = 2;
    const cudaError_t launched = cudaLaunchKernelEx(&config, lb::attention_tcgen05_halves_kernel<true>, map_q, map_k, map_v, p);
    if (launched != cudaSuccess) return static_cast<int>(launched);
    return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
