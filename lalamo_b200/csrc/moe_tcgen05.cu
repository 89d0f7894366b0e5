// The routed experts' products of many (token, expert) pairs on the fifth-generation tensor cores.  Pairs are sorted by
// expert, their tokens' rows gathered into that order, and two products run over the experts' ragged row counts:
//     hidden[place] = act(gate[e] x) * (up[e] x)   (or act(up[e] x))          out[pair] = down[e] hidden[place]
//
// A persistent CTA walks over items, an item being 128 sorted rows of one expert (the accumulator's lanes) times `bn` rows of
// its matrices (the accumulator's columns; the gated product has bn / 2 rows of `up` and the same rows of `gate` side by side,
// so that a thread of the epilogue holds both sides of a hidden value).  Warp 0 loads (TMA, 128-byte swizzle, 64 columns of K a
// stage), warp 1 issues tcgen05.mma into one of two accumulators, warps 2 to 9 read the other one out: a thread holds a
// row, sets 32 columns of it down in shared memory and sends them off as one bulk copy, wherever that row goes.
// What bounds it: with hundreds of rows an expert the way from L2 (an item reads 48 KB for 512 cycles of products; 12.5 TB/s
// over all multiprocessors while it runs); with a few rows an expert the stream of the experts' matrices from HBM, each
// read once.  Measured, 16 experts of 2048 x 2048, 4 a token: 2,048 tokens 144 us up and 81 us down (950 and 850 TFLOP/s; 632 and 379 us
// on mma.sync tiles of 64 x 64), 8 tokens, caches cold, 96 us in all (130 us where every pair streams its expert's rows).
// Every wait on a barrier is bounded, as in gemm_tcgen05.cu.
#include "tcgen05.cuh"

#include <type_traits>

namespace lb {

constexpr int kMoeRows = 128, kMoeBlockK = 64, kMoeThreads = 320, kMoeStagesMost = 8;
constexpr int kMoeStageArea = 196608;         // bytes of shared memory for the stages: four of 48 KB, or more of smaller ones
constexpr int kMoePitch = 80;                 // bytes of an epilogue thread's row of 64: 16-byte pieces of eight lanes in eight banks' worth
constexpr int kMoeMaxExperts = 1024;

struct MoeTcParams {
    const int* offsets;         // [experts + 1]: expert e's pairs have the places offsets[e] .. offsets[e + 1]
    const int* sorted;          // the pair at each place
    const float* pair_weight;   // up: the sums are multiplied by the pair's (may be null)
    void* out;                  // up: hidden, bfloat16, by place; down: 32-bit, by pair; rows of n_total
    int experts, n_total, k_total, bn, stages, box_rows, activation;
    float limit;
    int* status;
};

// n / d for d of one and more: the hardware's reciprocal, and one correction by the remainder, which the fused operation gives exactly (P.
// Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  The compiler's own
// division has a branch for every value, so that a thread's 64 values of an item follow one another: with it 32 pairs of 2048 x 2048 experts took
// 128 us instead of 97.
__device__ __forceinline__ float moe_tc_quotient(float n, float d) {
    const float scale = d > 0x1p64f ? 0x1p-64f : 1.0f;   // beyond 2^126 the reciprocal is nothing
    n *= scale, d *= scale;
    const float reciprocal = __fdividef(1.0f, d), q = n * reciprocal, rest = fmaf(-d, q, n);
    return rest == rest ? fmaf(rest, reciprocal, q) : q;   // infinite n or d: q as it is
}

// The activations and roundings of the streaming kernels (moe_activate and moe_hidden in moe.cu), the activation known outside the loops.
template <int ACTIVATION>
__device__ __forceinline__ float moe_tc_activate(float v) {
    if constexpr (ACTIVATION == 0) return moe_tc_quotient(v, 1.0f + expf(-v));                            // silu
    else if constexpr (ACTIVATION == 1) return 0.5f * v * (1.0f + erff(v * 0.70710678118654752440f));    // gelu (exact)
    else return v;
}
template <int ACTIVATION>
__device__ __forceinline__ float moe_tc_hidden(float gate, float up, float limit) {
    using T = __nv_bfloat16;
    if constexpr (ACTIVATION == kSigmoidLimit) {
        const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
        return moe_tc_quotient(g, 1.0f + expf(-kSigmoidLimitSlope * g)) * (u + 1.0f);
    } else {
        return round_to<T>(moe_tc_activate<ACTIVATION>(round_to<T>(gate))) * round_to<T>(up);
    }
}
template <typename Use>
__device__ __forceinline__ void with_activation(int activation, Use&& use) {
    if (activation == 0) use(std::integral_constant<int, 0>{});
    else if (activation == 1) use(std::integral_constant<int, 1>{});
    else if (activation == kSigmoidLimit) use(std::integral_constant<int, kSigmoidLimit>{});
    else use(std::integral_constant<int, 2>{});
}

__device__ __forceinline__ void bulk_store_row(void* global_destination, const void* source, int bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(global_destination), "r"(smem_address(source)), "r"(bytes) : "memory");
}

// MODE 1: gated up, 2: plain up, 0: down.
template <int MODE>
__global__ void __launch_bounds__(kMoeThreads, 1)
moe_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_gate,
                   const MoeTcParams p) {
    constexpr bool GATED = MODE == 1, UP = MODE != 0;
    extern __shared__ unsigned char raw_shared[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_shared) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* staging = tiles + kMoeStageArea;                                              // two halves of 128 rows of kMoePitch
    int* tile_start = reinterpret_cast<int*>(staging + 2 * kMoeRows * kMoePitch);                // [experts + 1]: row tiles before each expert's
    int* row_start = tile_start + p.experts + 1;                                                 // [experts + 1]: the offsets
    __shared__ uint64_t full[kMoeStagesMost], empty[kMoeStagesMost], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;

    allow_next_kernel();   // the next product's CTAs fit beside these no more than these beside one another
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMoeStagesMost; ++s) {
            barrier_init(&full[s], 1);
            barrier_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            barrier_init(&tmem_full[a], 1);
            barrier_init(&tmem_empty[a], 8);   // the epilogue's warps
        }
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    wait_for_previous_kernel();
    if (warp == 0) {
        // row tiles before each expert, 32 experts at a time
        int before = 0;
        for (int e0 = 0; e0 < p.experts; e0 += 32) {
            const int e = e0 + lane;
            const int begin = e < p.experts ? p.offsets[e] : 0;
            const int mine = e < p.experts ? (p.offsets[e + 1] - begin + kMoeRows - 1) / kMoeRows : 0;
            int sum = mine;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, sum, offset);
                if (lane >= offset) sum += other;
            }
            if (e < p.experts) tile_start[e] = before + sum - mine, row_start[e] = begin;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) tile_start[p.experts] = before, row_start[p.experts] = p.offsets[p.experts];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    const int columns = GATED ? p.bn / 2 : p.bn;   // rows of a matrix per item
    const int n_tiles = (p.n_total + columns - 1) / columns;
    const int num_items = tile_start[p.experts] * n_tiles;
    const int blocks = (p.k_total + kMoeBlockK - 1) / kMoeBlockK;
    const int stage_bytes = kMoeRows * kMoeBlockK * 2 + p.bn * kMoeBlockK * 2;

    // Items of one expert lie together, those with the same rows of its matrices next to one another.
    struct Item {
        int expert, first, rows, n0;
    };
    auto item_of = [&](int item) {
        int low = 0, high = p.experts;   // the last expert whose items begin at or before this one
        while (high - low > 1) {
            const int middle = (low + high) >> 1;
            if (tile_start[middle] * n_tiles <= item) low = middle;
            else high = middle;
        }
        const int tiles_here = tile_start[low + 1] - tile_start[low];
        const int rest = item - tile_start[low] * n_tiles;
        const int begin = row_start[low], m = rest % tiles_here;
        return Item{low, begin + m * kMoeRows, min(kMoeRows, row_start[low + 1] - begin - m * kMoeRows), rest / tiles_here * columns};
    };

    if (warp == 0 && lane == 0) {
        int issued = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
            const Item it = item_of(item);
            const int b_row = it.expert * p.n_total + it.n0;
            const int a_rows = (it.rows + p.box_rows - 1) / p.box_rows * p.box_rows;   // what the rows past them hold reaches no row that is stored
            for (int block = 0; block < blocks; ++block, ++issued) {
                const int s = issued % p.stages, round = issued / p.stages;
                if (round > 0 && !barrier_wait(&empty[s], (round - 1) & 1)) {
                    atomicExch(&failed, 1);
                    ok = false;
                    break;
                }
                unsigned char* stage = tiles + s * stage_bytes;
                barrier_expect(&full[s], (a_rows + p.bn) * kMoeBlockK * 2);
                for (int r = 0; r < a_rows; r += p.box_rows) tma_load_2d(stage + r * kMoeBlockK * 2, &map_a, block * kMoeBlockK, it.first + r, &full[s]);
                unsigned char* b = stage + kMoeRows * kMoeBlockK * 2;
                tma_load_2d(b, &map_b, block * kMoeBlockK, b_row, &full[s]);
                if constexpr (GATED) tma_load_2d(b + columns * kMoeBlockK * 2, &map_gate, block * kMoeBlockK, b_row, &full[s]);
            }
        }
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.bn >> 3) << 17) | (static_cast<uint32_t>(kMoeRows >> 4) << 24);
        int consumed = 0, local = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x, ++local) {
            const int accumulator = local & 1, use = local >> 1;
            if (use > 0 && !barrier_wait(&tmem_empty[accumulator], (use - 1) & 1)) {
                atomicExch(&failed, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(accumulator * 256);
            for (int block = 0; block < blocks; ++block, ++consumed) {
                const int s = consumed % p.stages, round = consumed / p.stages;
                if (!barrier_wait(&full[s], round & 1)) {
                    atomicExch(&failed, 1);
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned char* stage = tiles + s * stage_bytes;
                const uint64_t desc_a = tile_descriptor(stage), desc_b = tile_descriptor(stage + kMoeRows * kMoeBlockK * 2);
#pragma unroll
                for (int k = 0; k < kMoeBlockK / 16; ++k) mma_f16(tmem_d, desc_a + 2 * k, desc_b + 2 * k, idesc, block > 0 || k > 0);
                mma_commit(&empty[s]);
            }
            if (ok) mma_commit(&tmem_full[accumulator]);
        }
    } else if (warp >= 2) {
        const int quarter = warp & 3;            // of the accumulator's lanes
        const int half = (warp - 2) >> 2;        // every second chunk of 32 columns
        const int row = quarter * 32 + lane;
        unsigned char* mine = staging + (half * kMoeRows + row) * kMoePitch;
        int local = 0;
        for (int item = blockIdx.x; item < num_items; item += gridDim.x, ++local) {
            const int accumulator = local & 1, use = local >> 1;
            const Item it = item_of(item);
            const bool real = row < it.rows;
            const int pair = real && (!UP || p.pair_weight != nullptr) ? p.sorted[it.first + row] : 0;
            const float factor = UP && p.pair_weight != nullptr && real ? p.pair_weight[pair] : 1.0f;
            const bool arrived = barrier_wait(&tmem_full[accumulator], use & 1);
            if (!__all_sync(0xffffffffu, arrived)) {
                atomicExch(&failed, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(accumulator * 256) + (static_cast<uint32_t>(quarter * 32) << 16);
            const size_t out_row = static_cast<size_t>(UP ? it.first + row : pair) * p.n_total;
#pragma unroll 1
            for (int c = 32 * half; c < columns; c += 64) {
                const int here = min(32, p.n_total - it.n0 - c);   // a multiple of 8
                if (here <= 0) break;
                uint32_t v[32];
                tmem_load_32(tmem_d + static_cast<uint32_t>(c), v);
                // this thread's row of the chunk before has been read (it is written by nobody else)
                if constexpr (UP) {
                    __nv_bfloat162 packed[16];
                    if constexpr (GATED) {
                        uint32_t g[32];
                        tmem_load_32(tmem_d + static_cast<uint32_t>(columns + c), g);
                        with_activation(p.activation, [&](auto activation) {
                            constexpr int A = decltype(activation)::value;
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                packed[i] = __floats2bfloat162_rn(moe_tc_hidden<A>(__uint_as_float(g[2 * i]) * factor, __uint_as_float(v[2 * i]) * factor, p.limit),
                                                                  moe_tc_hidden<A>(__uint_as_float(g[2 * i + 1]) * factor, __uint_as_float(v[2 * i + 1]) * factor, p.limit));
                        });
                    } else {
                        with_activation(p.activation, [&](auto activation) {
                            constexpr int A = decltype(activation)::value;
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                packed[i] = __floats2bfloat162_rn(moe_tc_activate<A>(__uint_as_float(v[2 * i]) * factor), moe_tc_activate<A>(__uint_as_float(v[2 * i + 1]) * factor));
                        });
                    }
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(mine + 16 * i) = *reinterpret_cast<const uint4*>(&packed[4 * i]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    if (real) bulk_store_row(static_cast<__nv_bfloat16*>(p.out) + out_row + it.n0 + c, mine, here * 2);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                } else if (real) {
                    float4* destination = reinterpret_cast<float4*>(static_cast<float*>(p.out) + out_row + it.n0 + c);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (4 * i < here)
                            destination[i] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) barrier_arrive(&tmem_empty[accumulator]);
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (failed) {
        if (threadIdx.x == 0) report_error(p.status, kWaitTimeout);
        for (int spin = 0; spin < 2000; ++spin) __nanosleep(1000);   // copies in flight land
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}

// Pairs sorted by expert: offsets[e] .. offsets[e + 1] are the places of expert e's pairs in `sorted` (pairs whose expert is no
// expert are left out).  One block; the order of an expert's pairs among themselves is whatever the shared-memory counters
// give, which changes no result: every pair's row is computed by itself.
__global__ void moe_sort_kernel(const int* __restrict__ chosen, int pairs, int experts, int* __restrict__ offsets, int* __restrict__ sorted) {
    extern __shared__ int counters[];   // experts counts, then experts cursors
    int* cursors = counters + experts;
    allow_next_kernel();
    for (int e = threadIdx.x; e < experts; e += blockDim.x) counters[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e >= 0 && e < experts) atomicAdd(&counters[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int e = 0; e < experts; ++e) {
            offsets[e] = total;
            cursors[e] = total;
            total += counters[e];
        }
        offsets[experts] = total;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e >= 0 && e < experts) sorted[atomicAdd(&cursors[e], 1)] = p;
    }
}

// gathered[place] = x[sorted[place] / top], 16 bytes a thread; one block a place.
__global__ void __launch_bounds__(128)
moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ offsets, const int* __restrict__ sorted, uint4* __restrict__ gathered, int experts, int top,
                  int pieces) {
    allow_next_kernel();
    wait_for_previous_kernel();
    const int place = blockIdx.x;
    if (place >= offsets[experts]) return;
    const uint4* source = x + static_cast<size_t>(sorted[place] / top) * pieces;
    uint4* destination = gathered + static_cast<size_t>(place) * pieces;
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) destination[i] = source[i];
}

// Both at once for up to kMoeArrangePairs pairs: a block a pair, which counts the pairs before its own in the order of the experts (and, of one expert, of the
// pairs), leaves its place and copies its row; one more block makes the offsets.  8 tokens of 4 experts: one launch of 4 us for two of 3 and 4.  Every block reads all
// pairs, work that grows with their square.  Both products with two launches and with one, 16 experts of 1024 x 1152 and 64 of 1024 x 512: 32 pairs 34.3 and 32.8 us, 30.6 and
// 27.9; 512 43.6 and 43.0, 54.4 and 52.6; 1,024 45.5 and 45.3, 57.5 and 55.8; 2,048 61.9 and 62.5, 62.4 and 62.1; 4,096 82.9 and 90.3, 73.0 and 79.4.
constexpr int kMoeArrangePairs = 1024;
__global__ void __launch_bounds__(128)
moe_arrange_kernel(const uint4* __restrict__ x, const int* __restrict__ chosen, int pairs, int experts, int top, int pieces, int* __restrict__ offsets, int* __restrict__ sorted,
                   uint4* __restrict__ gathered) {
    extern __shared__ int counters[];   // experts (the last block's), or four warps' counts
    wait_for_previous_kernel();
    allow_next_kernel();
    const int pair = blockIdx.x, tid = threadIdx.x;
    if (pair == pairs) {
        for (int e = tid; e < experts; e += blockDim.x) counters[e] = 0;
        __syncthreads();
        for (int p = tid; p < pairs; p += blockDim.x) {
            const int e = chosen[p];
            if (e >= 0 && e < experts) atomicAdd(&counters[e], 1);
        }
        __syncthreads();
        if (tid == 0) {
            int total = 0;
            for (int e = 0; e < experts; ++e) {
                offsets[e] = total;
                total += counters[e];
            }
            offsets[experts] = total;
        }
        return;
    }
    const int own = chosen[pair];
    if (own < 0 || own >= experts) return;   // no expert: left out
    int before = 0;
    for (int p = tid; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e >= 0 && (e < own || (e == own && p < pair))) ++before;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if ((tid & 31) == 0) counters[tid >> 5] = before;
    __syncthreads();
    const int place = counters[0] + counters[1] + counters[2] + counters[3];
    if (tid == 0) sorted[place] = pair;
    const uint4* source = x + static_cast<size_t>(pair / top) * pieces;
    uint4* destination = gathered + static_cast<size_t>(place) * pieces;
    for (int i = tid; i < pieces; i += blockDim.x) destination[i] = source[i];
}

// A [rows, k] bfloat16 matrix seen through boxes of [box_rows, 64] with 128-byte swizzle; what lies outside reads as zero.
static bool moe_map(CUtensorMap* map, const void* base, long long rows, int k, int box_rows) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {kMoeBlockK, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t element_strides[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
int launch_moe_tcgen05(const void* a, const void* b, const void* gate, int pairs, MoeTcParams p, cudaStream_t stream) {
    // Columns an item: 256, since what an item loads of its sorted rows is then shared by most; half of that where it would leave
    // more than half of the multiprocessors without an item.  Guessed: every second expert ends in a partly filled tile of 128
    // rows.  Measured, both products: 16 experts of 1024 x 1152, 16 tokens of 4 experts 52 us with 128 columns, 56 with 256; of
    // 2048 x 2048, 8 tokens 97 us with 256, 114 with 128, and 2,048 tokens 247 against 384 (64 columns: slower everywhere).
    const int used = pairs < p.experts ? pairs : p.experts;
    const int row_tiles = (pairs + kMoeRows - 1) / kMoeRows > used ? (pairs + kMoeRows - 1) / kMoeRows + used / 2 : used;
    const int whole = MODE == 1 ? 128 : 256;
    p.bn = 2 * row_tiles * ((p.n_total + whole - 1) / whole) >= multiprocessor_count() ? 256 : 128;
    const int stage_bytes = (kMoeRows + p.bn) * kMoeBlockK * 2;
    p.stages = kMoeStageArea / stage_bytes < kMoeStagesMost ? kMoeStageArea / stage_bytes : kMoeStagesMost;
    CUtensorMap map_a, map_b, map_gate;
    const long long rows = static_cast<long long>(p.experts) * p.n_total;
    // Sorted rows come in boxes: of 32 where experts have few (8 tokens of 2048 x 2048: 97 us, 105 with boxes of 128), else one of
    // 128 a stage (2,048 tokens: 247 us, 284 with four of 32).
    p.box_rows = pairs < 64 * used ? 32 : kMoeRows;
    const int columns = MODE == 1 ? p.bn / 2 : p.bn;   // a box's rows, at most 256
    if (!moe_map(&map_a, a, pairs, p.k_total, p.box_rows) || !moe_map(&map_b, b, rows, p.k_total, columns) ||
        !moe_map(&map_gate, gate != nullptr ? gate : b, rows, p.k_total, columns)) return -5;
    auto kernel = moe_tcgen05_kernel<MODE>;
    constexpr int most = 1024 + kMoeStageArea + 2 * kMoeRows * kMoePitch + 2 * (kMoeMaxExperts + 1) * 4;
    static OncePerDevice configured;
    if (allow_shared_memory(configured, kernel, most) != cudaSuccess) return static_cast<int>(cudaGetLastError());
    return static_cast<int>(launch_overlapped(kernel, dim3(multiprocessor_count()), dim3(kMoeThreads), static_cast<size_t>(most), stream, map_a, map_b, map_gate, p));
}

}  // namespace lb

extern "C" {

// The grouped path (bfloat16; width and ff multiples of 8; at most 1024 experts): sorts the pairs by expert into
// `offsets` [experts + 1] and `sorted` [pairs], gathers their rows into `gathered` [pairs, width], then the two grouped products.
// `hidden` is [pairs, ff] (rows in sorted order), `out` [pairs, width] in 32-bit (rows in pair order; rows of pairs without an
// expert are not written).
int lb_moe_experts_grouped(const void* x, const void* gate, const void* up, const void* down, const int* chosen, int* offsets, int* sorted, void* gathered, void* hidden,
                           float* out, int pairs, int top, int width, int ff, int experts, int activation, cudaStream_t stream, float limit, const float* pair_weight,
                           int* status) {
    if (pairs == 0) return 0;
    if (width % 8 != 0 || ff % 8 != 0 || experts < 1 || experts > lb::kMoeMaxExperts) return -2;
    cudaError_t error;
    if (pairs <= lb::kMoeArrangePairs) {
        error = lb::launch_overlapped(lb::moe_arrange_kernel, dim3(pairs + 1), dim3(128), (experts > 4 ? experts : 4) * sizeof(int), stream, static_cast<const uint4*>(x), chosen, pairs,
                                      experts, top, width / 8, offsets, sorted, static_cast<uint4*>(gathered));
    } else {
        lb::moe_sort_kernel<<<1, 1024, 2 * experts * sizeof(int), stream>>>(chosen, pairs, experts, offsets, sorted);
        error = cudaGetLastError();
        if (error == cudaSuccess)
            error = lb::launch_overlapped(lb::moe_gather_kernel, dim3(pairs), dim3(128), 0, stream, static_cast<const uint4*>(x), offsets, sorted, static_cast<uint4*>(gathered), experts,
                                          top, width / 8);
    }
    if (error != cudaSuccess) return static_cast<int>(error);
    lb::MoeTcParams p = {};
    p.offsets = offsets, p.sorted = sorted, p.experts = experts, p.activation = activation, p.limit = limit, p.status = status;
    lb::MoeTcParams first = p, second = p;
    first.pair_weight = pair_weight, first.out = hidden, first.n_total = ff, first.k_total = width;
    second.out = out, second.n_total = width, second.k_total = ff;
    const int code = gate != nullptr ? lb::launch_moe_tcgen05<1>(gathered, up, gate, pairs, first, stream) : lb::launch_moe_tcgen05<2>(gathered, up, nullptr, pairs, first, stream);
    if (code != 0) return code;
    return lb::launch_moe_tcgen05<0>(hidden, down, nullptr, pairs, second, stream);
}

}  // extern "C"
