// Causal attention of runs of new tokens over the paged cache on the tensor cores, for 32-bit queries, keys and values (heads of 64 and 128), with the
// accuracy of 32-bit sums.  The reference materialises the scores (crates/models/src/components/gated_attention.rs:449-473).
//
// Every operand is cut into three bfloat16 pieces (the next eight significant bits each, cut off, so that the pieces add up exactly, but for numbers below 2^-110) and every product
// is the six piece products that reach 2^-24 of it, as in gemm_f32_tc.cu; the tensor core's additions cut off instead of rounding, so chains on it are short,
// with the small pieces' products first: scores in two accumulators of D / 2 elements (of 64 where D is 64: one), which the softmax adds, and the
// weighted values in an accumulator of its own for every 64 keys, which is added to sums in registers.
//
// A block owns 128 queries of a head, whose pieces stay in shared memory, and walks the pages of 64 keys in two groups of warps:
//   softmax: eight warps, two threads to a query, which both find the maximum over its scores in tensor memory and then take half of the keys (expf, the
//            sum, the weights' pieces to tensor memory, from where they are the A operand of the second product) and half of the D sums, to which the
//            values of the page before are added;
//   cutters: four warps bring the next page's keys and values into registers (16-byte loads) while this one's are in use, cut them into the 128-byte swizzled rows
//            that both products read (values as they lie, MN-major); one of their warps issues the products (a whole warp, see elect_one).
// Order of the products: scores 0, scores 1, values 0, scores 2, values 1, ...: the softmax of page i + 1 runs beside the values of page i and the
// scores of page i + 2.  The keys of a tile may be shared out among the blocks of a cluster, whose maxima and sums are joined through shared memory.  Bound by the products: at D 128 the scores read 288 KB of shared memory for 6.3 M multiply-adds, about 2,300 cycles a
// page, the values 1,536.  16 heads of 128 over 777 tokens: 65 us in two ranges, 89 in one, 6.5 us a page of the
// longest block (its two groups of warps issue some 3,000 instructions a page to each scheduler); with 64 queries to a block on the 32-bit pipes 234 us.
//
// A row that is not finite (an infinity's or a NaN's pieces, also those of a value that the query does not see, make NaN of a whole page) is computed
// again by plain sums over the keys that it does see.
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128;             // queries of a block: lanes of tensor memory
constexpr int BN = 64;              // keys of a page
constexpr int kPieces = 3;
constexpr int kSoftmax = 256, kCutters = 128, kThreads = kSoftmax + kCutters;      // eight softmax warps, four cutters
constexpr int kScoreColumns = 128;  // a page's two score accumulators
constexpr int kWeightColumn = 2 * kScoreColumns, kValueColumn = kWeightColumn + kPieces * 32, kColumns = 512;

constexpr int kMostRanges = 8;

struct Shared {
    uint64_t keys_full, values_full;   // a page's pieces are in shared memory
    uint64_t scores_done[2];           // the scores of even and of odd pages are complete (the keys may be written over)
    uint64_t weights_ready;            // a page's weights are in tensor memory, its scores and the values' accumulator have been read
    uint64_t values_done;              // the values' accumulator is complete (the values may be written over)
    float total[2][BM];                // of each half of a query's keys
    int finite[2][BM];
    float top[BM];                     // of a range of the keys
    uint32_t tensor_memory_base;
    int abort_flag;
};

template <int D> constexpr int kSliceCount = D / 64;
template <int D> constexpr uint32_t kQueryPiece = BM * D * 2;
template <int D> constexpr uint32_t kPagePiece = BN * D * 2;
// Heads of 64 need some 103 KB, but a block takes all columns of tensor memory.
template <int D> constexpr int shared_bytes() {
    constexpr int used = static_cast<int>(sizeof(Shared)) + 1024 + kPieces * static_cast<int>(kQueryPiece<D> + 2 * kPagePiece<D>);
    return used < 120 * 1024 ? 120 * 1024 : used;
}
static_assert(alone_on_an_sm(shared_bytes<64>()) && alone_on_an_sm(shared_bytes<128>()), "a block holds all 512 columns of tensor memory");

// Cuts four floats into pieces and stores eight bytes of each.
__device__ __forceinline__ void store_pieces(const float4& value, uint32_t address, uint32_t piece_bytes) {
    float rest[4] = {value.x, value.y, value.z, value.w};
#pragma unroll
    for (int piece = 0; piece < kPieces; ++piece) {
        uint32_t bits[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bits[i] = __float_as_uint(rest[i]);
            rest[i] -= __uint_as_float(bits[i] & 0xffff0000u);
        }
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(address + piece * piece_bytes), "r"(__byte_perm(bits[0], bits[1], 0x7632)),
                     "r"(__byte_perm(bits[2], bits[3], 0x7632))
                     : "memory");
    }
}

// Where four elements from `column` on of row `row` lie in a tile of `rows` rows: slices of 64 elements, rows of 128 bytes, their 16-byte columns swizzled.
__device__ __forceinline__ uint32_t tile_place(int row, int column, int rows) {
    return (column >> 6) * rows * 128 + row * 128 + ((((column & 63) >> 3) ^ (row & 7)) << 4) + ((column >> 2) & 1) * 8;
}

// MN-major tile (`[key][element]` as it lies): 128-byte rows hold 64 elements of a key; groups of 8 keys 1024 bytes apart, the next 64 elements a slice further.
__device__ __forceinline__ uint64_t mn_major_descriptor(uint32_t address) {
    return static_cast<uint64_t>((address >> 4) & 0x3fffu) | (static_cast<uint64_t>((BN * 128) >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_issue_from_tensor(uint32_t accumulator, uint32_t a, uint64_t b, uint32_t descriptor, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(accumulator), "r"(a), "l"(b), "r"(descriptor), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tensor_store_16(uint32_t address, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(address),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                 "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}

// The row of one query by plain sums, by a whole warp: 32 keys at a time, a lane scores one and owns every 32nd element of the result.
template <int D>
__device__ __noinline__ void plain_row(const float* __restrict__ query, const float* __restrict__ keys, const float* __restrict__ values, float* __restrict__ target,
                                       const int* __restrict__ pages, size_t head_offset, size_t page_floats, int position, int first_key, float scale) {
    const int lane = threadIdx.x & 31;
    float top = -INFINITY, total = 0.0f, acc[D / 32] = {};
    for (int base = first_key; base <= position; base += 32) {
        const int key = base + lane;
        size_t row = 0;
        float score = -INFINITY;
        if (key <= position) {
            row = pages[key / BN] * page_floats + head_offset + static_cast<size_t>(key % BN) * D;
            float dot = 0.0f;
            for (int e = 0; e < D; ++e) dot = fmaf(query[e], keys[row + e], dot);
            score = dot * scale;
        }
        const float new_top = fmaxf(top, warp_max(score)), correction = expf(top - new_top);
        const float weight = key <= position ? expf(score - new_top) : 0.0f;
        total = total * correction + warp_sum(weight);
        top = new_top;
        for (int e = 0; e < D / 32; ++e) acc[e] *= correction;
        for (int j = 0; j < min(32, position - base + 1); ++j) {
            const float mine = __shfl_sync(0xffffffffu, weight, j);
            const size_t value_row = __shfl_sync(0xffffffffu, static_cast<unsigned long long>(row), j);
            for (int e = 0; e < D / 32; ++e) acc[e] = fmaf(mine, values[value_row + lane + 32 * e], acc[e]);
        }
    }
    for (int e = 0; e < D / 32; ++e) target[lane + 32 * e] = acc[e] / total;
}

// Joins the ranges' sums of one query, `elements` of them from `own` on, in the ranges' order; false if one is not finite.
__device__ __noinline__ bool join_ranges(Shared* shared, const float* own, int row, int ranges, int elements, float* target) {
    float top = -INFINITY, total = 0.0f, factor[kMostRanges];
#pragma unroll
    for (int other = 0; other < kMostRanges; ++other)
        if (other < ranges) top = fmaxf(top, cluster_load(cluster_address(&shared->top[row], other)));
#pragma unroll
    for (int other = 0; other < kMostRanges; ++other) {
        if (other >= ranges) break;
        factor[other] = expf(cluster_load(cluster_address(&shared->top[row], other)) - top);
        total += factor[other] * (cluster_load(cluster_address(&shared->total[0][row], other)) + cluster_load(cluster_address(&shared->total[1][row], other)));
    }
    const float inverse = 1.0f / total;
    bool finite = true;
    for (int e = 0; e < elements; e += 4) {
        float value[4] = {};
#pragma unroll
        for (int other = 0; other < kMostRanges; ++other) {
            if (other >= ranges) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) value[i] = fmaf(factor[other], cluster_load(cluster_address(own + (e + i) * BM, other)), value[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            value[i] *= inverse;
            finite = finite && isfinite(value[i]);
        }
        if (target) *reinterpret_cast<float4*>(target + e) = make_float4(value[0], value[1], value[2], value[3]);
    }
    return finite;
}

// grid (heads x ranges, tiles of 128 queries): tiles of sequence s are numbered from cu_seqlens[s] / 128 + s on; those of later tokens, which see more keys, begin first.
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_tc_kernel(const float* __restrict__ queries, const float* __restrict__ keys, const float* __restrict__ values, float* __restrict__ out,
                        const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start, const int* __restrict__ page_rows, int page_stride, int n_seqs, int n_heads,
                        int n_kv_heads, float scale, int window, int ranges) {
    extern __shared__ uint8_t shared_raw[];
    Shared* shared = reinterpret_cast<Shared*>(shared_raw);
    const uint32_t query_tiles = (smem_address(shared_raw) + static_cast<uint32_t>(sizeof(Shared)) + 1023u) & ~1023u;
    const uint32_t key_tiles = query_tiles + kPieces * kQueryPiece<D>, value_tiles = key_tiles + kPieces * kPagePiece<D>;
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    volatile int* abort_flag = &shared->abort_flag;
    constexpr int kAccumulators = kSliceCount<D>;      // score accumulators of 64 elements each

    if (threadIdx.x == 0) {
        barrier_init(&shared->keys_full, kCutters);
        barrier_init(&shared->values_full, kCutters);
        barrier_init(&shared->scores_done[0], 1);
        barrier_init(&shared->scores_done[1], 1);
        barrier_init(&shared->weights_ready, kSoftmax / 32);
        barrier_init(&shared->values_done, 1);
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
    grid_dependents_launch();      // only now that this block has its tensor memory
    grid_dependency_wait();

    const int range = ranges > 1 ? static_cast<int>(cluster_rank()) : 0;      // of the keys, the blocks of a cluster
    const int number = gridDim.y - 1 - blockIdx.y, head = blockIdx.x / ranges, kv_head = head / (n_heads / n_kv_heads);
    int sequence = 0;
    while (sequence + 1 < n_seqs && cu_seqlens[sequence + 1] / BM + sequence + 1 <= number) ++sequence;
    const int begin = cu_seqlens[sequence], first = (number - begin / BM - sequence) * BM;      // of the run's tokens
    const int live = min(BM, cu_seqlens[sequence + 1] - begin - first);
    const int position0 = seq_start[sequence] + first, last = position0 + live - 1;
    const int seen_page = window > 0 && position0 - window + 1 > 0 ? (position0 - window + 1) / BN : 0, all_pages = last / BN - seen_page + 1;
    const int first_page = seen_page + all_pages * range / ranges, pages = seen_page + all_pages * (range + 1) / ranges - first_page;
    const int* page_row = page_rows + static_cast<size_t>(sequence) * page_stride;
    const size_t page_floats = static_cast<size_t>(n_kv_heads) * BN * D, head_offset = static_cast<size_t>(kv_head) * BN * D;
    float* const partial = reinterpret_cast<float*>(shared_raw + (query_tiles - smem_address(shared_raw)));      // a range's sums [element][query], where the queries were
    // A row whose result is not finite once more, by one warp.
    auto again_plainly = [&](int row) {
        const size_t place = (static_cast<size_t>(begin + first + row) * n_heads + head) * D;
        plain_row<D>(queries + place, keys, values, out + place, page_row, head_offset, page_floats, position0 + row,
                     window > 0 && position0 + row - window + 1 > 0 ? position0 + row - window + 1 : 0, scale);
    };
    if (live > 0 && pages == 0) {      // fewer pages than ranges: nothing seen
        if (threadIdx.x < BM) {
            shared->top[threadIdx.x] = -INFINITY;
            shared->total[0][threadIdx.x] = shared->total[1][threadIdx.x] = 0.0f;
        }
        for (int item = threadIdx.x; item < BM * D; item += kThreads) partial[item] = 0.0f;
    } else if (live > 0) {      // else a number that no tile has
        // The queries' pieces, by everyone; rows behind the last are zeros.
        for (int item = threadIdx.x; item < BM * D / 4; item += kThreads) {
            const int row = item / (D / 4), column = item % (D / 4) * 4;
            const float4 q = row < live ? *reinterpret_cast<const float4*>(queries + (static_cast<size_t>(begin + first + row) * n_heads + head) * D + column)
                                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            store_pieces(q, query_tiles + tile_place(row, column, BM), kQueryPiece<D>);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        bool alive = true;
        if (warp < kSoftmax / 32) {
            // ---- softmax ----
            constexpr int kOwnKeys = BN / 2, kOwn = D / 2;
            const int quarter = warp & 3, half = warp >> 2;
            const uint32_t lane_base = tensor_base + (static_cast<uint32_t>(quarter * 32) << 16);
            const int row = quarter * 32 + lane, position = position0 + row;
            float sums[kOwn], top = -INFINITY, total = 0.0f;      // `total`: over this thread's keys
#pragma unroll
            for (int e = 0; e < kOwn; ++e) sums[e] = 0.0f;
            // Adds the accumulator of page `page - 1`, whose weights were taken at the maximum `top`, and goes over to a new maximum.
            auto add_values = [&](int page, float correction) {
                if (!__all_sync(0xffffffffu, barrier_wait(&shared->values_done, (page - 1) & 1, abort_flag))) return false;
                tensor_fence_after_sync();
#pragma unroll
                for (int part = 0; part < kOwn; part += 32) {
                    uint32_t v[32];
                    tensor_load_32(lane_base + kValueColumn + half * kOwn + part, v);
                    tensor_load_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) sums[part + e] = (sums[part + e] + __uint_as_float(v[e])) * correction;
                }
                return true;
            };
            for (int page = 0; page < pages; ++page) {
                if (!__all_sync(0xffffffffu, barrier_wait(&shared->scores_done[page & 1], (page >> 1) & 1, abort_flag))) { alive = false; break; }
                tensor_fence_after_sync();
                const int key0 = (first_page + page) * BN;
                const int seen = position - key0, low = window > 0 ? seen - window : -1;      // keys of the page up to the first and after the second
                const bool whole = key0 + BN - 1 <= position0 + quarter * 32 && (window <= 0 || key0 > position0 + quarter * 32 + 31 - window);      // for all rows of the warp
                // The other half's keys for their maximum, then the own half's, which stay.
                float score[kOwnKeys], high = -INFINITY;
#pragma unroll
                for (int turn = 0; turn < 2; ++turn) {
                    const int key = (turn == 0 ? half ^ 1 : half) * kOwnKeys;
                    uint32_t v[32];
                    tensor_load_32(lane_base + (page & 1) * kScoreColumns + key, v);
                    if constexpr (kAccumulators == 2) {
                        uint32_t more[32];
                        tensor_load_32(lane_base + (page & 1) * kScoreColumns + BN + key, more);
                        tensor_load_wait();
#pragma unroll
                        for (int j = 0; j < kOwnKeys; ++j) score[j] = (__uint_as_float(v[j]) + __uint_as_float(more[j])) * scale;
                    } else {
                        tensor_load_wait();
#pragma unroll
                        for (int j = 0; j < kOwnKeys; ++j) score[j] = __uint_as_float(v[j]) * scale;
                    }
                    if (!whole) {
#pragma unroll
                        for (int j = 0; j < kOwnKeys; ++j) score[j] = key + j <= seen && key + j > low ? score[j] : -INFINITY;
                    }
                    float part[4] = {high, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int j = 0; j < kOwnKeys; ++j) part[j & 3] = fmaxf(part[j & 3], score[j]);
                    high = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
                }
                const float new_top = fmaxf(top, high), base = new_top == -INFINITY ? 0.0f : new_top;      // a row may see nothing of a page
                const float correction = expf(top - base);
                float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int j = 0; j < kOwnKeys; ++j) {
                    score[j] = expf(score[j] - base);
                    part[j & 3] += score[j];
                }
                total = total * correction + ((part[0] + part[1]) + (part[2] + part[3]));
                top = new_top;
                if (page > 0 && !add_values(page, correction)) { alive = false; break; }
                // The weights' pieces, 16 columns each: the products of the page before are done.
#pragma unroll
                for (int piece = 0; piece < kPieces; ++piece) {
                    uint32_t packed[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float& x = score[2 * j];
                        float& y = score[2 * j + 1];
                        packed[j] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
                        x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
                        y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
                    }
                    tensor_store_16(lane_base + kWeightColumn + piece * 32 + half * 16, packed);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tensor_fence_before_sync();
                __syncwarp();
                if (lane == 0) barrier_arrive(&shared->weights_ready);
            }
            alive = alive && add_values(pages, 1.0f);
            // Both threads of a query meet: the sum over all keys, and whether all of the row is finite.
            shared->total[half][row] = total;
            if (ranges > 1) {
                if (half == 0) shared->top[row] = top;
#pragma unroll
                for (int e = 0; e < kOwn; ++e) partial[(half * kOwn + e) * BM + row] = sums[e];
            } else {
                asm volatile("bar.sync 1, %0;" ::"n"(kSoftmax) : "memory");
                const float inverse = 1.0f / (shared->total[0][row] + shared->total[1][row]);
                bool finite = true;
#pragma unroll
                for (int e = 0; e < kOwn; ++e) {
                    sums[e] *= inverse;
                    finite = finite && isfinite(sums[e]);
                }
                shared->finite[half][row] = finite;
                asm volatile("bar.sync 1, %0;" ::"n"(kSoftmax) : "memory");
                finite = shared->finite[0][row] && shared->finite[1][row];
                if (alive) {
                    float* target = out + (static_cast<size_t>(begin + first + row) * n_heads + head) * D + half * kOwn;
                    if (row < live && finite) {
#pragma unroll
                        for (int e = 0; e < kOwn; e += 4) *reinterpret_cast<float4*>(target + e) = make_float4(sums[e], sums[e + 1], sums[e + 2], sums[e + 3]);
                    }
                    for (unsigned again = half == 0 ? __ballot_sync(0xffffffffu, row < live && !finite) : 0u; again; again &= again - 1) again_plainly(quarter * 32 + __ffs(again) - 1);
                }
            }
        } else {
            // ---- cutters ----
            constexpr int kLoads = BN * D / 4 / kCutters, kRowsApart = kCutters / (D / 4);      // 16 bytes of every kRowsApart-th row
            const int thread = threadIdx.x - kSoftmax, row0 = thread / (D / 4), column = thread % (D / 4) * 4;
            float4 next_keys[kLoads], next_values[kLoads];
            auto load = [&](const float* cache, int page, float4 (&target)[kLoads]) {
                const int key0 = (first_page + page) * BN;
                const float* source = cache + (page < pages ? page_row[first_page + page] : 0) * page_floats + head_offset + column;
#pragma unroll
                for (int i = 0; i < kLoads; ++i) {      // positions behind the last query may hold anything
                    const int row = row0 + i * kRowsApart;
                    target[i] = page < pages && key0 + row <= last ? *reinterpret_cast<const float4*>(source + row * D) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            };
            auto cut = [&](const float4 (&source)[kLoads], uint32_t tiles, uint64_t* full) {
#pragma unroll
                for (int i = 0; i < kLoads; ++i) store_pieces(source[i], tiles + tile_place(row0 + i * kRowsApart, column, BN), kPagePiece<D>);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (!operands_lost()) barrier_arrive(full);
            };
            constexpr int kOrder[6][2] = {{2, 0}, {1, 1}, {0, 2}, {1, 0}, {0, 1}, {0, 0}};      // piece of A, piece of B: the small products first
            // The first cutter warp issues, one lane of it.
            const bool leader = elect_one();
            const uint32_t base = __shfl_sync(0xffffffffu, tensor_base, 0);
            auto warp_wait = [&](uint64_t* barrier, uint32_t parity) { return __all_sync(0xffffffffu, barrier_wait(barrier, parity, abort_flag)) != 0; };
            auto issue_scores = [&](int page) {
                if (!warp_wait(&shared->keys_full, page & 1)) return false;
                tensor_fence_after_sync();
                const uint32_t descriptor = instruction_descriptor(BM, BN);
                if (leader) {
#pragma unroll
                    for (int part = 0; part < kAccumulators; ++part) {
                        const uint32_t accumulator = base + (page & 1) * kScoreColumns + part * BN;
#pragma unroll
                        for (int pair = 0; pair < 6; ++pair) {
                            const uint32_t query = query_tiles + kOrder[pair][0] * kQueryPiece<D> + part * BM * 128, key = key_tiles + kOrder[pair][1] * kPagePiece<D> + part * BN * 128;
#pragma unroll
                            for (int k = 0; k < 4; ++k) mma_issue(accumulator, tile_descriptor(query + k * 32), tile_descriptor(key + k * 32), descriptor, pair + k > 0 ? 1u : 0u);
                        }
                    }
                    mma_commit(&shared->scores_done[page & 1]);
                }
                __syncwarp();
                return true;
            };
            auto issue_values = [&](int page) {
                if (!warp_wait(&shared->values_full, page & 1) || !warp_wait(&shared->weights_ready, page & 1)) return false;
                tensor_fence_after_sync();
                const uint32_t descriptor = instruction_descriptor(BM, D) | (1u << 16);      // B is MN-major
                if (leader) {
#pragma unroll
                    for (int pair = 0; pair < 6; ++pair)
#pragma unroll
                        for (int k = 0; k < BN / 16; ++k)
                            mma_issue_from_tensor(base + kValueColumn, base + kWeightColumn + kOrder[pair][0] * 32 + k * 8,
                                                  mn_major_descriptor(value_tiles + kOrder[pair][1] * kPagePiece<D> + k * 2048), descriptor, pair + k > 0 ? 1u : 0u);
                    mma_commit(&shared->values_done);
                }
                __syncwarp();
                return true;
            };
            auto by_one = [&](auto issue, int page) {
                if (warp == kSoftmax / 32) alive = issue(page);
            };
            auto all_wait = [&](uint64_t* barrier, int parity) {
                alive = __all_sync(0xffffffffu, barrier_wait(barrier, parity, abort_flag));
            };
            load(keys, 0, next_keys);
            load(values, 0, next_values);
            cut(next_keys, key_tiles, &shared->keys_full);
            load(keys, 1, next_keys);
            by_one(issue_scores, 0);
            cut(next_values, value_tiles, &shared->values_full);
            load(values, 1, next_values);
            // The next keys, once the scores before have read theirs: their accumulators were read by the softmax of two pages before, whose weights have been
            // waited for.
            auto next_scores = [&](int page) {
                if (page >= pages || !alive) return;
                all_wait(&shared->scores_done[(page - 1) & 1], ((page - 1) >> 1) & 1);
                if (!alive) return;
                cut(next_keys, key_tiles, &shared->keys_full);
                load(keys, page + 1, next_keys);
                by_one(issue_scores, page);
            };
            next_scores(1);
            for (int page = 0; page < pages && alive; ++page) {
                by_one(issue_values, page);
                next_scores(page + 2);
                if (page + 1 < pages && alive) {
                    all_wait(&shared->values_done, page & 1);
                    if (!alive) break;
                    cut(next_values, value_tiles, &shared->values_full);
                    load(values, page + 2, next_values);
                }
            }
        }
    }

    tensor_fence_before_sync();
    __syncthreads();
    if (ranges > 1) {
        // Every thread of every block comes here, also after a wait that ran out, so the two meetings cannot be missed.  Between them each block joins the ranges of its share
        // of the queries, in their order: several threads to a query.
        cluster_share_abort(&shared->abort_flag, ranges);
        cluster_sync_all();
        const int rows_here = BM / ranges, own_part = threadIdx.x / rows_here, row = range * rows_here + threadIdx.x % rows_here, elements = D * rows_here / kSoftmax;
        if (warp < kSoftmax / 32 && live > 0 && *abort_flag == 0) {
            float* target = out + (static_cast<size_t>(begin + first + row) * n_heads + head) * D + own_part * elements;
            const bool finite = join_ranges(shared, partial + own_part * elements * BM + row, row, ranges, elements, row < live ? target : nullptr);
            if (threadIdx.x < BM) shared->finite[0][threadIdx.x] = 1;
            asm volatile("bar.sync 1, %0;" ::"n"(kSoftmax) : "memory");      // also: the row's parts are stored
            if (!finite) shared->finite[0][row] = 0;
            asm volatile("bar.sync 1, %0;" ::"n"(kSoftmax) : "memory");
            for (int mine = range * rows_here + warp; mine < (range + 1) * rows_here && mine < live; mine += kSoftmax / 32)
                if (!shared->finite[0][mine]) again_plainly(mine);
        }
        cluster_sync_all();      // nobody leaves while another still reads its sums
    }
    if (warp == 0) {
        tensor_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tensor_base), "r"(kColumns) : "memory");
    }
}

// Clusters of `ranges` blocks that the device holds at once (a cluster lies inside one GPC, so fewer than its blocks alone); 0 if it does not say.
template <int D>
int clusters_at_once(int ranges) {
    static int known[kMostRanges + 1] = {};      // 0: not asked, -1: no answer
    if (known[ranges] == 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(ranges);
        config.blockDim = dim3(kThreads);
        config.dynamicSmemBytes = shared_bytes<D>();
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = ranges;
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        int clusters = 0;
        known[ranges] = cudaOccupancyMaxActiveClusters(&clusters, attention_f32_tc_kernel<D>, &config) == cudaSuccess && clusters > 0 ? clusters : -1;
        if (known[ranges] < 0) cudaGetLastError();
    }
    return known[ranges] < 0 ? 0 : known[ranges];
}

template <int D>
int launch(const float* queries, const float* keys, const float* values, float* out, const int* cu_seqlens, const int* seq_start, const int* page_rows, int page_stride,
           int n_tokens, int n_seqs, int n_heads, int n_kv_heads, float scale, int window, int ranges, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t status = cudaFuncSetAttribute(attention_f32_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared_bytes<D>());
        if (status != cudaSuccess) return static_cast<int>(status);
        configured = true;
    }
    const int tiles = n_tokens / BM + n_seqs;
    const long long blocks = static_cast<long long>(n_heads) * tiles;
    if (ranges <= 0) {
        // As many ranges as are resident at once (us, 16 heads of 128: 100 tokens behind 3,000 322 alone, 173 in two, 96 in four; 300 tokens 39 -> 31, 70 tokens 21 -> 19); two also
        // where the blocks of whole tiles would fill the SMs, but the tiles' lengths lie far apart: a block's time is its pages', and the longest of 777 tokens sees 13, the
        // average 8 (93 -> 65; tiles of one length, 160 blocks of 17 pages, 131 -> 144).
        const bool uneven = ranges < 0;
        ranges = kMostRanges;
        while (ranges > 1 && (blocks * ranges > 148 || clusters_at_once<D>(ranges) < blocks)) ranges /= 2;
        if (ranges == 1 && uneven && blocks <= 148) ranges = 2;
    }
    if (ranges != 1 && ranges != 2 && ranges != 4 && ranges != 8) return cudaErrorInvalidValue;
    if (ranges > 1)
        tau_launch_clusters(ranges, attention_f32_tc_kernel<D>, dim3(n_heads * ranges, tiles), dim3(kThreads), shared_bytes<D>(), stream, queries, keys, values, out, cu_seqlens, seq_start,
                            page_rows, page_stride, n_seqs, n_heads, n_kv_heads, scale, window, ranges);
    else
        tau_launch(attention_f32_tc_kernel<D>, dim3(n_heads, tiles), dim3(kThreads), shared_bytes<D>(), stream, queries, keys, values, out, cu_seqlens, seq_start, page_rows, page_stride,
                   n_seqs, n_heads, n_kv_heads, scale, window, ranges);
    return tau_launch_status();
}

}  // namespace

// 0 if no wait has run out since the library was loaded (synchronises the device).
TAU_EXPORT int tau_attention_f32_tc_status() {
    int flag = 0;
    if (cudaMemcpyFromSymbol(&flag, wait_error, sizeof(int)) != cudaSuccess) return -1;
    return flag;
}

// `ranges`: blocks that share the keys of 128 queries (1, 2, 4, 8); 0 picks, -1 picks for tiles that see very different numbers of keys.
// `cu_seqlens` bounds the runs, `seq_start` positions were cached before; heads of 64 or 128 elements, pages of 64, everything on 16 bytes.
TAU_EXPORT int tau_attention_f32_tc(const float* queries, const float* keys, const float* values, float* out, const int* cu_seqlens, const int* seq_start,
                                    const int* page_rows, int page_stride, int n_tokens, int n_seqs, int n_heads, int n_kv_heads, int head_dim, float scale, int window,
                                    int ranges, void* stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (!queries || !keys || !values || !out || !cu_seqlens || !seq_start || !page_rows || (head_dim != 64 && head_dim != 128) || n_heads <= 0 || n_kv_heads <= 0
        || n_heads % n_kv_heads != 0 || window < 0 || n_tokens / BM + n_seqs > 65535
        || ((reinterpret_cast<uintptr_t>(queries) | reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(values) | reinterpret_cast<uintptr_t>(out)) & 15) != 0)
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (head_dim == 64) return launch<64>(queries, keys, values, out, cu_seqlens, seq_start, page_rows, page_stride, n_tokens, n_seqs, n_heads, n_kv_heads, scale, window, ranges, s);
    return launch<128>(queries, keys, values, out, cu_seqlens, seq_start, page_rows, page_stride, n_tokens, n_seqs, n_heads, n_kv_heads, scale, window, ranges, s);
}
