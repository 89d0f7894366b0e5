// The 32-bit path's matrix products:  Y[m, n] = sum_k X[m, k] * W[n, k]  in plain 32-bit multiply-adds, X [M, K] and W [N, K] with their rows
// along K.  A CTA of four warps takes BM rows of X and 64 rows of W, K in blocks of 32 columns through three stages of shared memory as they lie (rows of 36
// floats, so that eight neighbouring rows' pieces of 16 bytes meet no bank twice); a thread has BM / 8 x 4 sums and reads 16 bytes, four columns, of each of its
// rows at a time.  Where the tiles alone leave multiprocessors idle, or the last round of them nearly empty, a cluster of up to eight CTAs shares out K: each leaves
// its sums in its shared memory, and each adds up a part of the tile from all of them, in their order.
// What bounds it: the multiply-adds (128 a cycle and multiprocessor; operands' dispatch), and for a few rows of X the stream of W.
#include "common.cuh"

namespace lb {

constexpr int kF32Threads = 128, kF32Columns = 64, kF32Block = 32, kF32Pitch = 36, kF32Stages = 3;

struct Float32Params {
    const float* x;
    const float* w;
    float* out;
    int m, n, k, x_stride;
};

template <int BM>
struct Float32Shared {
    static constexpr int kStage = (BM + kF32Columns) * kF32Pitch;   // floats
    static constexpr int kTilePitch = kF32Columns + 4;
    static constexpr int kBytes = kF32Stages * kStage * 4;
    static_assert(BM * kTilePitch <= kF32Stages * kStage, "the sums fit where the stages were");
};

__device__ __forceinline__ void float32_copy(float* destination, const float* source, bool real) {
    const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(destination));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(source), "r"(real ? 16 : 0) : "memory");
}

// grid (tiles of W's rows, tiles of X's rows, slices of K); a cluster is the slices of a tile.
template <int BM>
__global__ void __launch_bounds__(kF32Threads)
gemm_float32_kernel(const Float32Params p) {
    using Shared = Float32Shared<BM>;
    constexpr int TM = BM / 8, TN = kF32Columns / 16;
    extern __shared__ __align__(16) float float32_memory[];
    wait_for_previous_kernel();
    allow_next_kernel();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mg = (warp & 1) * 4 + (lane >> 3), ng = (warp >> 1) * 8 + (lane & 7);   // the thread's rows of X: mg + 8 i, of W: ng + 16 j
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * kF32Columns;
    const int blocks_in_all = (p.k + kF32Block - 1) / kF32Block, per_slice = (blocks_in_all + static_cast<int>(gridDim.z) - 1) / static_cast<int>(gridDim.z);
    const int first = blockIdx.z * per_slice, blocks = max(0, min(blocks_in_all, first + per_slice) - first);
    auto load = [&](int block) {
        if (block < blocks) {
            float* stage = float32_memory + (block % kF32Stages) * Shared::kStage;
            const int k0 = (first + block) * kF32Block, row = tid >> 3, column = 4 * (tid & 7);
            const bool in_k = k0 + column < p.k;   // (k is a multiple of 4)
#pragma unroll
            for (int r = 0; r < BM; r += 16) {
                const bool real = in_k && m0 + r + row < p.m;
                float32_copy(stage + (r + row) * kF32Pitch + column, real ? p.x + static_cast<size_t>(m0 + r + row) * p.x_stride + k0 + column : p.x, real);
            }
#pragma unroll
            for (int r = 0; r < kF32Columns; r += 16) {
                const bool real = in_k && n0 + r + row < p.n;
                float32_copy(stage + (BM + r + row) * kF32Pitch + column, real ? p.w + static_cast<size_t>(n0 + r + row) * p.k + k0 + column : p.w, real);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[TM][TN] = {};
    for (int block = 0; block < kF32Stages - 1; ++block) load(block);
    for (int block = 0; block < blocks; ++block) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kF32Stages - 2) : "memory");
        __syncthreads();   // the block is there, and the one before it has been read
        load(block + kF32Stages - 1);
        const float* x_s = float32_memory + (block % kF32Stages) * Shared::kStage + mg * kF32Pitch;
        const float* w_s = float32_memory + (block % kF32Stages) * Shared::kStage + (BM + ng) * kF32Pitch;
#pragma unroll
        for (int c = 0; c < kF32Block; c += 4) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(w_s + 16 * j * kF32Pitch + c);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(x_s + 8 * i * kF32Pitch + c);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(x.x, w[j].x, acc[i][j]);
                    acc[i][j] = fmaf(x.y, w[j].y, acc[i][j]);
                    acc[i][j] = fmaf(x.z, w[j].z, acc[i][j]);
                    acc[i][j] = fmaf(x.w, w[j].w, acc[i][j]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (gridDim.z == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int row = m0 + mg + 8 * i;
#pragma unroll
            for (int j = 0; j < TN; ++j)
                if (row < p.m && n0 + ng + 16 * j < p.n) p.out[static_cast<size_t>(row) * p.n + n0 + ng + 16 * j] = acc[i][j];
        }
        return;
    }
    // the sums of the cluster's CTAs, each adding up its share of the tile's rows
    __syncthreads();   // the last block has been read
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) float32_memory[(mg + 8 * i) * Shared::kTilePitch + ng + 16 * j] = acc[i][j];
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int rows = BM / static_cast<int>(gridDim.z), row0 = rows * blockIdx.z;
    for (int index = tid; index < rows * (kF32Columns / 4); index += kF32Threads) {
        const int row = row0 + index / (kF32Columns / 4), column = 4 * (index % (kF32Columns / 4));
        const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(float32_memory + row * Shared::kTilePitch + column));
        float sum[4] = {};
        for (unsigned slice = 0; slice < gridDim.z; ++slice) {
            uint32_t address;
            float part[4];
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(address) : "r"(mine), "r"(slice));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(part[0]), "=f"(part[1]), "=f"(part[2]), "=f"(part[3]) : "r"(address) : "memory");
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[e] += part[e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (m0 + row < p.m && n0 + column + e < p.n) p.out[static_cast<size_t>(m0 + row) * p.n + n0 + column + e] = sum[e];
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // nobody's sums go away while they are read
}

template <int BM>
int launch_gemm_float32(const Float32Params& p, int slices, cudaStream_t stream) {
    static OncePerDevice once;
    auto kernel = gemm_float32_kernel<BM>;
    const cudaError_t allowed = allow_shared_memory(once, kernel, Float32Shared<BM>::kBytes);
    if (allowed != cudaSuccess) return static_cast<int>(allowed);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((p.n + kF32Columns - 1) / kF32Columns, (p.m + BM - 1) / BM, slices);
    config.blockDim = dim3(kF32Threads);
    config.dynamicSmemBytes = Float32Shared<BM>::kBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = 1;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = slices;
    // An early start (see launch_early_if) for more than 64 tokens: layers with one and without, attention of width 1024 300 tokens 125 and 129 us, a short convolution 100 57.6 and
    // 59.6, but of 64 tokens 54.9 and 49.2, of width 2048 8 tokens 70.9 and 55.5, a gated feed-forward 107 and 91.
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = p.m > 64 && overlap_launches() ? 1 : 0;
    config.attrs = attribute;
    config.numAttrs = 2;
    return static_cast<int>(cudaLaunchKernelEx(&config, kernel, p));
}

}  // namespace lb

extern "C" {

// out [m, n] = x [m, k] w [n, k]^T in float32; rows of x x_stride elements apart.  k and x_stride multiples of 4, x and w 16-byte aligned: -2 otherwise.
// slices: CTAs of a cluster that share out k (1, 2, 4 or 8), 0: chosen by the sizes.  Measured, ours and cuBLAS: 8 x 2048 x 1024 8 and 19 us, 20 x 2048 x 2048 15 and 37,
// 64 x 1024 x 4608 37 and 70, 300 x 1024 x 1024 24 and 31, 300 x 2048 x 1024 42 and 47; one row 7 and 5, 256 x 16384 x 2048 383 and 311 (its larger tiles
// do 78 % of the multiply-adds' rate, these 54 %).  Errors against 64 bits 2.1e-7 and 5.7e-7 (1,024 columns).  Which sizes come here: ops.float32_product_supported.
int lb_gemm_float32(const float* x, const float* w, float* out, int m, int n, int k, int x_stride, int slices, cudaStream_t stream) {
    if (m == 0 || n == 0) return 0;
    if (m < 1 || n < 1 || k < 4 || k % 4 != 0 || x_stride < k || x_stride % 4 != 0 || (slices != 0 && slices != 1 && slices != 2 && slices != 4 && slices != 8) ||
        ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
        return -2;
    const int rows = m <= 16 ? 16 : m <= 32 ? 32 : 64;
    const long long tiles = static_cast<long long>((n + lb::kF32Columns - 1) / lb::kF32Columns) * ((m + rows - 1) / rows);
    if ((m + rows - 1) / rows > 65535) return -2;
    const int blocks = (k + lb::kF32Block - 1) / lb::kF32Block, sms = lb::multiprocessor_count();
    if (slices == 0) {
        // Blocks of columns that the busiest multiprocessor works off, a start for every CTA; one CTA of 64 rows by itself takes a quarter longer than beside
        // another, and smaller ones share a multiprocessor without slowing each other.
        const long long room = static_cast<long long>(sms) * 64 / rows;
        long long least = -1;
        for (int s = 1; s <= 8; s *= 2) {
            if (s > 1 && blocks < 4 * s) break;
            const long long together = (tiles * s + room - 1) / room, cost = together * ((blocks + s - 1) / s + 1) * (rows == 64 && together == 1 ? 5 : 4);
            if (least < 0 || cost < least) least = cost, slices = s;
        }
    }
    const lb::Float32Params p{x, w, out, m, n, k, x_stride};
    return rows == 16 ? lb::launch_gemm_float32<16>(p, slices, stream) : rows == 32 ? lb::launch_gemm_float32<32>(p, slices, stream) : lb::launch_gemm_float32<64>(p, slices, stream);
}

}  // extern "C"
