// Tensor-core product for sm_100a of 32-bit operands: out[M, N] = x[M, K] * w[N, K]^T + bias, with the accuracy of 32-bit sums.
//
// A float is the sum of three bfloat16 numbers: its first eight significant bits, the next eight and the last eight (cut off, not rounded, so the
// three add up to it exactly), for numbers from about 2^-110 on: of smaller ones the last piece and then the middle one fall below bfloat16's smallest number, 2^-133, and such
// an operand keeps what lies above that.  Six of the nine piece products reach 2^-24 of a product:
//   x w = x0 w0 + (x0 w1 + x1 w0) + (x0 w2 + x1 w1 + x2 w0) + what is left out (2^-25 of it on average).
// bfloat16 products are exact in the tensor core's 32-bit accumulator, but its additions cut off instead of rounding, so no chain on it is long:
// each 64 columns of K get an accumulator of their own, the five small products enter it first and the large one last (four additions at full
// size), and the accumulators are read back and added by ordinary 32-bit additions.  Against 64 bits this is nearer than the chain of K
// multiply-adds of the plain kernel (gemm_simt.cu).
//
// What bounds it: shared memory and the products.  A block holds a tile of 128 features (lanes of tensor memory) by BN tokens (its columns) in five roles.  One
// thread asks for the 32-bit tiles of a step of 64 columns of K by TMA (128-byte swizzled rows of 32 columns); four warps cut the weights' and put the
// pieces into tensor memory, from where they are the A operand; four cut the activations' into swizzled rows of shared memory, the B operand;
// one warp issues the step's products; eight warps add its accumulator to their sums.  Where tiles are few, a tile's K is cut into ranges, one for each
// block of a cluster, whose sums meet in the blocks' shared memory.  With loads through registers, and loading, cutting and adding
// in the same eight warps, a step of 128 x 128 took 2.15 us (the load/store pipe takes one thing after another); in roles, with a single thread that computed its own
// descriptors as issuer, 1.55; with a whole warp that issues 1.17 (24 products of 64 clocks each are 0.8): 777 x 6144 x 1024 103 -> 85 -> 75 us, by multiply-adds
// 308 us.  Twice the warps for the weights, with fewer registers each, were slower, and activations cut ahead by a kernel of their own, so that all eight cut
// weights, no faster (79 us).
//
// A result that is not finite is computed again by plain multiply-adds: an infinite or very large operand has pieces whose products are
// NaN (inf - inf) where the plain sum is infinite.
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128;              // features of a tile
constexpr int BK = 64;               // K columns of a step: 128 bytes of pieces, one swizzle row
constexpr int kPieces = 3;
constexpr int kCutWarps = 4, kAddWarps = 8;      // warps that cut each operand, and that add
constexpr int kThreads = (2 * kCutWarps + kAddWarps + 2) * 32;
constexpr uint32_t kWeightRaw = BM * BK * 4;
constexpr int kMostStages = 3, kMostSplits = 8;
constexpr uint32_t kWeightColumns = kPieces * 32;      // tensor memory that a step's weight pieces take

struct Shared {
    uint64_t raw_full[kMostStages], raw_free[kMostStages];      // a step's 32-bit tiles have landed; they have been read
    uint64_t full[2];      // pieces of a step are in their places
    uint64_t done[2];      // its products are done: the accumulator is complete, the pieces are free
    uint64_t added[2];     // its accumulator has been read
    uint32_t tensor_memory_base;
    int abort_flag;
};

// Cuts two floats: a word of two bfloat16 numbers for each piece.
__device__ __forceinline__ void cut_pair(float x, float y, uint32_t (&pieces)[kPieces]) {
#pragma unroll
    for (int piece = 0; piece < kPieces; ++piece) {
        pieces[piece] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
        x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
        y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
    }
}
__device__ __forceinline__ float4 shared_load_4(uint32_t address) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address) : "memory");
    return v;
}
__device__ __forceinline__ void tensor_store_16(uint32_t address, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(address),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                 "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// The product's A operand from tensor memory (lane = row, a column holds two neighbouring bfloat16 of K).
__device__ __forceinline__ void mma_issue_from_tensor(uint32_t accumulator, uint32_t a, uint64_t b, uint32_t descriptor, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(accumulator), "r"(a), "l"(b), "r"(descriptor), "r"(accumulate)
        : "memory");
}

__device__ __noinline__ float plain_sum(const float* row, const float* column, int K) {
    float sum = 0.0f;
    for (int k = 0; k < K; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(row + k), b = *reinterpret_cast<const float4*>(column + k);
        sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
    }
    return sum;
}

template <int BN> constexpr int kStages = BN == 128 ? 2 : 3;      // of 32-bit tiles
template <int BN> constexpr int shared_bytes() {
    return static_cast<int>(sizeof(Shared)) + 1024 + kStages<BN> * (BM + BN) * BK * 4 + 2 * kPieces * BN * BK * 2;
}
static_assert(alone_on_an_sm(shared_bytes<64>()) && alone_on_an_sm(shared_bytes<128>()), "a block holds all 512 columns of tensor memory");

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap weight_map, const __grid_constant__ CUtensorMap input_map, const float* __restrict__ x, const float* __restrict__ w,
                   const float* __restrict__ bias, float* __restrict__ out, int M, int N, int K, long long x_stride, long long w_stride, long long out_stride,
                   int splits) {
    extern __shared__ uint8_t shared_raw[];
    Shared* shared = reinterpret_cast<Shared*>(shared_raw);
    uint8_t* const raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(shared_raw) + sizeof(Shared) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kInputRaw = BN * BK * 4, kRaw = kWeightRaw + kInputRaw, kInputPiece = BN * BK * 2;
    float* const partial = reinterpret_cast<float*>(raw);
    const uint32_t raw_tiles = smem_address(raw), input_pieces = raw_tiles + kStages<BN> * kRaw;
    constexpr uint32_t kAccumulators = 2 * kWeightColumns, kUsed = kAccumulators + 2 * BN, kColumns = kUsed <= 512 && kUsed > 256 ? 512 : 1024;
    static_assert(kColumns == 512, "a power of two that holds the pieces and two accumulators");
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    // A tile's ranges of K are the blocks of a cluster.
    const int split = splits > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int feature0 = blockIdx.x / splits * BM, token0 = blockIdx.y * BN;
    const int all_steps = (K + BK - 1) / BK, first_step = all_steps * split / splits, steps = all_steps * (split + 1) / splits - first_step;
    volatile int* abort_flag = &shared->abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages<BN>; ++s) {
            barrier_init(&shared->raw_full[s], 1);
            barrier_init(&shared->raw_free[s], 2 * kCutWarps);
        }
        for (int s = 0; s < 2; ++s) {
            barrier_init(&shared->full[s], 2 * kCutWarps);
            barrier_init(&shared->done[s], 1);
            barrier_init(&shared->added[s], kAddWarps);
        }
        shared->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(&shared->tensor_memory_base)), "r"(kColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tensor_fence_before_sync();
    __syncthreads();
    tensor_fence_after_sync();
    const uint32_t tensor_base = shared->tensor_memory_base;
    grid_dependents_launch();      // only now that this block has its tensor memory (see gemm_tc_kernel)

    // The whole warp waits; false if the block is giving up.
    auto warp_wait = [&](uint64_t* barrier, uint32_t parity) { return __all_sync(0xffffffffu, barrier_wait(barrier, parity, abort_flag)) != 0; };
    if (warp < kCutWarps) {
        // ---- the weights: a thread owns a row, its pieces go to its lane of tensor memory ----
        const uint32_t lane_base = tensor_base + (static_cast<uint32_t>(warp * 32) << 16);
        const int row = warp * 32 + lane;
        int stage = 0, phase = 0;
        for (int step = 0; step < steps; ++step) {
            if (!warp_wait(&shared->raw_full[stage], phase)) break;
            if (step >= 2 && !warp_wait(&shared->done[step & 1], ((step >> 1) - 1) & 1)) break;      // the pieces of the step before last are read
            tensor_fence_after_sync();
            const uint32_t source = raw_tiles + stage * kRaw + row * 128;
#pragma unroll
            for (int half = 0; half < 2; ++half) {      // 32 columns of K
                uint32_t pieces[kPieces][16];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 v = shared_load_4(source + half * BM * 128 + ((j ^ (row & 7)) << 4));
                    uint32_t first[kPieces], second[kPieces];
                    cut_pair(v.x, v.y, first);
                    cut_pair(v.z, v.w, second);
#pragma unroll
                    for (int p = 0; p < kPieces; ++p) pieces[p][2 * j] = first[p], pieces[p][2 * j + 1] = second[p];
                }
#pragma unroll
                for (int p = 0; p < kPieces; ++p) tensor_store_16(lane_base + (step & 1) * kWeightColumns + p * 32 + half * 16, pieces[p]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tensor_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                barrier_arrive(&shared->raw_free[stage]);
                barrier_arrive(&shared->full[step & 1]);
            }
            if (++stage == kStages<BN>) stage = 0, phase ^= 1;
        }
    } else if (warp < 2 * kCutWarps) {
        // ---- the activations: a thread owns a row (of 64: half of one), its pieces go to swizzled rows of 128 bytes ----
        const int thread = threadIdx.x - kCutWarps * 32, row = thread % BN;
        constexpr int kHalves = BN == 128 ? 2 : 1;
        const int first_half = BN == 128 ? 0 : thread / BN;
        int stage = 0, phase = 0;
        for (int step = 0; step < steps; ++step) {
            if (!warp_wait(&shared->raw_full[stage], phase)) break;
            if (step >= 2 && !warp_wait(&shared->done[step & 1], ((step >> 1) - 1) & 1)) break;
            const uint32_t target = input_pieces + (step & 1) * kPieces * kInputPiece + row * 128;
#pragma unroll
            for (int i = 0; i < kHalves; ++i) {
                const int half = first_half + i;
                const uint32_t source = raw_tiles + stage * kRaw + kWeightRaw + half * BN * 128 + row * 128;
#pragma unroll
                for (int j = 0; j < 4; ++j) {      // eight columns of K
                    const float4 a = shared_load_4(source + (((2 * j) ^ (row & 7)) << 4)), b = shared_load_4(source + (((2 * j + 1) ^ (row & 7)) << 4));
                    uint32_t pieces[4][kPieces];
                    cut_pair(a.x, a.y, pieces[0]); cut_pair(a.z, a.w, pieces[1]); cut_pair(b.x, b.y, pieces[2]); cut_pair(b.z, b.w, pieces[3]);
#pragma unroll
                    for (int p = 0; p < kPieces; ++p)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(target + p * kInputPiece + (((half * 4 + j) ^ (row & 7)) << 4)), "r"(pieces[0][p]),
                                     "r"(pieces[1][p]), "r"(pieces[2][p]), "r"(pieces[3][p])
                                     : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                barrier_arrive(&shared->raw_free[stage]);
                barrier_arrive(&shared->full[step & 1]);
            }
            if (++stage == kStages<BN>) stage = 0, phase ^= 1;
        }
    } else if (warp < 2 * kCutWarps + kAddWarps) {
        // ---- add: a warp owns 32 features by half of the tokens ----
        constexpr int kOwn = BN / 2;
        const int quarter = warp & 3, first = (warp - 2 * kCutWarps) / 4 * kOwn;
        const uint32_t lane_base = tensor_base + (static_cast<uint32_t>(quarter * 32) << 16) + kAccumulators + first;
        float sums[kOwn];
#pragma unroll
        for (int j = 0; j < kOwn; ++j) sums[j] = 0.0f;
        bool alive = true;
        for (int step = 0; step < steps; ++step) {
            alive = warp_wait(&shared->done[step & 1], (step >> 1) & 1);
            if (!alive) break;
            tensor_fence_after_sync();
#pragma unroll
            for (int part = 0; part < kOwn; part += 16) {
                uint32_t v[16];
                tensor_load_16(lane_base + (step & 1) * BN + part, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) sums[part + j] += __uint_as_float(v[j]);
            }
            tensor_fence_before_sync();
            __syncwarp();
            if (lane == 0) barrier_arrive(&shared->added[step & 1]);
        }
        if (splits > 1) {
            // The range's sums go where the 32-bit tiles were (all have been cut), as [token][feature of the tile].
#pragma unroll
            for (int j = 0; j < kOwn; ++j) partial[(first + j) * BM + quarter * 32 + lane] = sums[j];
        } else {
            grid_dependency_wait();      // the output may still be in use by the kernel before
            const int feature = feature0 + quarter * 32 + lane;
            if (alive && feature < N) {
                const float offset = bias != nullptr ? bias[feature] : 0.0f;
#pragma unroll
                for (int j = 0; j < kOwn; ++j) {
                    const int token = token0 + first + j;
                    if (token >= M) break;
                    float value = sums[j];
                    if (!isfinite(value)) value = plain_sum(x + token * x_stride, w + feature * w_stride, K);
                    out[token * out_stride + feature] = value + offset;
                }
            }
        }
    } else if (warp == 2 * kCutWarps + kAddWarps) {
        // ---- ask for the 32-bit tiles; weights do not depend on the kernel before ----
        if (lane == 0) {
            int stage = 0, phase = 0, step = 0;
            for (; step < steps; ++step) {
                if (step >= kStages<BN> && !barrier_wait(&shared->raw_free[stage], phase ^ 1, abort_flag)) break;
                uint8_t* tile = raw + stage * kRaw;
                barrier_expect_bytes(&shared->raw_full[stage], kRaw);
                for (int half = 0; half < 2; ++half) tma_load_2d(tile + half * BM * 128, &weight_map, (first_step + step) * BK + half * 32, feature0, &shared->raw_full[stage]);
                if (step == 0) grid_dependency_wait();
                for (int half = 0; half < 2; ++half) tma_load_2d(tile + kWeightRaw + half * BN * 128, &input_map, (first_step + step) * BK + half * 32, token0, &shared->raw_full[stage]);
                if (++stage == kStages<BN>) stage = 0, phase ^= 1;
            }
            // A block that gives up does not leave before its copies either.
            for (int last = max(0, step - kStages<BN>); last < step; ++last) barrier_outlast(&shared->raw_full[last % kStages<BN>], last / kStages<BN> & 1);
        }
    } else {
        // ---- issue: the whole warp, so that the descriptors are uniform ----
        const uint32_t descriptor = instruction_descriptor(BM, BN), base = __shfl_sync(0xffffffffu, tensor_base, 0);
        const bool leader = elect_one();
        for (int step = 0; step < steps; ++step) {
            if (!warp_wait(&shared->full[step & 1], (step >> 1) & 1)) break;
            if (step >= 2 && !warp_wait(&shared->added[step & 1], ((step >> 1) - 1) & 1)) break;
            tensor_fence_after_sync();
            const uint32_t weight = base + (step & 1) * kWeightColumns, input = input_pieces + (step & 1) * kPieces * kInputPiece;
            const uint32_t accumulator = base + kAccumulators + (step & 1) * BN;
            constexpr int kOrder[6][2] = {{2, 0}, {1, 1}, {0, 2}, {1, 0}, {0, 1}, {0, 0}};      // piece of the weight, piece of the input
            if (leader) {
#pragma unroll
                for (int pair = 0; pair < 6; ++pair)
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        mma_issue_from_tensor(accumulator, weight + kOrder[pair][0] * 32 + k * 8, tile_descriptor(input + kOrder[pair][1] * kInputPiece + k * 32), descriptor,
                                              pair + k > 0 ? 1u : 0u);
                mma_commit(&shared->done[step & 1]);
            }
            __syncwarp();
        }
    }

    tensor_fence_before_sync();
    __syncthreads();
    if (splits > 1) {
        // Every thread of every block comes here, also after a wait that ran out, so the two meetings cannot be missed.  Between them each block adds the ranges of its share of the
        // tile's tokens, in their order.
        cluster_share_abort(&shared->abort_flag, splits);
        cluster_sync_all();
        if (*abort_flag == 0) {
            grid_dependency_wait();
            const int live = min(BN, M - token0), per = (live + splits - 1) / splits, last = min(live, (split + 1) * per);
            const uint32_t own = smem_address(partial);
            for (int token = split * per + warp; token < last; token += kThreads / 32) {
                float4 part[kMostSplits];
#pragma unroll
                for (int other = 0; other < kMostSplits; ++other)
                    part[other] = other < splits ? cluster_load_4(cluster_address_of(own + (token * BM + lane * 4) * 4, other)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                float value[4] = {};
#pragma unroll
                for (int other = 0; other < kMostSplits; ++other)
                    value[0] += part[other].x, value[1] += part[other].y, value[2] += part[other].z, value[3] += part[other].w;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int feature = feature0 + lane * 4 + i;
                    if (feature >= N) continue;
                    if (!isfinite(value[i])) value[i] = plain_sum(x + (token0 + token) * x_stride, w + feature * w_stride, K);
                    out[(token0 + token) * out_stride + feature] = value[i] + (bias != nullptr ? bias[feature] : 0.0f);
                }
            }
        }
        cluster_sync_all();      // nobody leaves while another still reads its sums
    }
    if (warp == 0) {
        tensor_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tensor_base), "r"(kColumns) : "memory");
    }
}

// A map over a row-major 32-bit matrix `[rows, K]`; boxes of `box_rows` x 32 (128 bytes), zeros outside.
bool make_map(CUtensorMap* map, const void* base, int rows, int K, long long stride, int box_rows) {
    EncodeTiled encode = encode_tiled();
    if (!encode) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(stride) * 4};
    const cuuint32_t box[2] = {32, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t element_strides[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
int configure() {
    static bool configured = false;
    if (!configured) {
        const cudaError_t status = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared_bytes<BN>());
        if (status != cudaSuccess) return static_cast<int>(status);
        configured = true;
    }
    return 0;
}

// Clusters of `splits` blocks that the device holds at once (a cluster lies inside one GPC, so fewer than its blocks alone); 0 if it does not say.
template <int BN>
int clusters_at_once(int splits) {
    static int known[kMostSplits + 1] = {};      // 0: not asked, -1: no answer
    if (known[splits] == 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(splits);
        config.blockDim = dim3(kThreads);
        config.dynamicSmemBytes = shared_bytes<BN>();
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = splits;
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        int clusters = 0;
        known[splits] = cudaOccupancyMaxActiveClusters(&clusters, gemm_f32_tc_kernel<BN>, &config) == cudaSuccess && clusters > 0 ? clusters : -1;
        if (known[splits] < 0) cudaGetLastError();
    }
    return known[splits] < 0 ? 0 : known[splits];
}

constexpr int kLeastSteps = 2;      // of a range

// Ranges of K for a token tile of BN and the time that they take, about, in us: rounds of the 148 SMs, 0.8 or 1.17 a step, 4 to begin and end and 3 more where ranges
// meet.  A tile alone on its SM is a chain of K / 64 steps; ranges take as many SMs as there are.  Left as one against the picked ranges: 777 x 1024 x 3072 62 -> 38 us
// (2 ranges), 300 x 1024 x 3072 60 -> 21 (5), 130 x 1024 x 3072 41 -> 15, 64 x 6144 x 1024 17 -> 13 (2), 256 x 1024 x 1024 17 -> 10 (4).
template <int BN>
float choose_splits(int M, int N, int K, int* splits) {
    const long long tiles = static_cast<long long>((N + BM - 1) / BM) * ((M + BN - 1) / BN);
    const int steps = (K + BK - 1) / BK;
    *splits = tiles > 74 ? 1 : static_cast<int>(148 / tiles);
    if (*splits > kMostSplits) *splits = kMostSplits;
    while (*splits > 1 && (steps / *splits < kLeastSteps || clusters_at_once<BN>(*splits) < tiles)) --*splits;
    return static_cast<float>((tiles * *splits + 147) / 148) * static_cast<float>((steps + *splits - 1) / *splits) * (BN == 64 ? 0.8f : 1.17f) + (*splits > 1 ? 7.0f : 4.0f);
}

template <int BN>
int launch(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, long long x_stride, long long w_stride, long long out_stride, int splits, cudaStream_t stream) {
    const int status = configure<BN>();
    if (status) return status;
    if (splits == 0) choose_splits<BN>(M, N, K, &splits);
    if (splits < 1 || splits > kMostSplits || splits > (K + BK - 1) / BK) return cudaErrorInvalidValue;
    CUtensorMap weight_map, input_map;
    if (!make_map(&weight_map, w, N, K, w_stride, BM) || !make_map(&input_map, x, M, K, x_stride, BN)) return cudaErrorInvalidValue;
    const dim3 grid((N + BM - 1) / BM * splits, (M + BN - 1) / BN);
    if (splits > 1)
        tau_launch_clusters(splits, gemm_f32_tc_kernel<BN>, grid, dim3(kThreads), shared_bytes<BN>(), stream, weight_map, input_map, x, w, bias, out, M, N, K, x_stride, w_stride, out_stride,
                            splits);
    else
        tau_launch(gemm_f32_tc_kernel<BN>, grid, dim3(kThreads), shared_bytes<BN>(), stream, weight_map, input_map, x, w, bias, out, M, N, K, x_stride, w_stride, out_stride, splits);
    return tau_launch_status();
}

}  // namespace

// 0 if no wait has run out since the library was loaded (synchronises the device).
TAU_EXPORT int tau_gemm_f32_tc_status() {
    int flag = 0;
    if (cudaMemcpyFromSymbol(&flag, wait_error, sizeof(int)) != cudaSuccess) return -1;
    return flag;
}

// Strides in elements; K and the strides multiples of 4, x and w on 16 bytes.  `token_box`: tokens of a tile, 64 or 128; `splits`: ranges of K, up to 8; 0 picks.
TAU_EXPORT int tau_gemm_f32_tc(const void* x, const void* w, const void* bias, void* out, int M, int N, int K, long long x_stride, long long w_stride,
                               long long out_stride, int token_box, int splits, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!x || !w || !out || K <= 0 || (K & 3) || (x_stride & 3) || (w_stride & 3) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) || splits < 0)
        return cudaErrorInvalidValue;
    int box = token_box;
    // Wide tiles cut the weights less often, narrow ones give more blocks (us, 64 against 128 tokens, each with its ranges: 777 x 1024 x 3072 44 against 38, 300 x 6144 x 1024
    // 35 against 27, 64 x 6144 x 1024 13 against 17, 130 x 1024 x 3072 15 against 18).
    if (box == 0) {
        int status = configure<64>(), narrow = 0, wide = 0;
        if (!status) status = configure<128>();
        if (status) return status;
        box = splits > 0 ? (M <= 64 ? 64 : 128) : M <= 64 || choose_splits<64>(M, N, K, &narrow) < choose_splits<128>(M, N, K, &wide) ? 64 : 128;
    }
    const auto* xf = static_cast<const float*>(x);
    const auto* wf = static_cast<const float*>(w);
    const auto* bf = static_cast<const float*>(bias);
    auto* of = static_cast<float*>(out);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (box) {
        case 64: return launch<64>(xf, wf, bf, of, M, N, K, x_stride, w_stride, out_stride, splits, s);
        case 128: return launch<128>(xf, wf, bf, of, M, N, K, x_stride, w_stride, out_stride, splits, s);
        default: return cudaErrorInvalidValue;
    }
}
