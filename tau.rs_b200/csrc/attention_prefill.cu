// Prefill attention in bfloat16: runs of new tokens of many sequences, causal, over the paged cache.
//
// Compiled for one head size (-DTAU_HEAD_DIM=...).  The reference materialises `repeat_kv`, the score matrix
// `[B, nq, T, S]` and an additive mask (crates/models/src/components/gated_attention.rs:449-473); this kernel
// keeps scores in registers with an online softmax (32-bit statistics, `key <= query position`,
// crates/models/src/qwen3_5_common/model.rs:154) and never writes them.
//
// A warp owns 16 consecutive query positions of one head; the 4 warps of a block take the query heads of one
// KV group (or neighbouring query tiles when the group is small) and share the key and value tiles, which
// cp.async brings into shared memory a few tiles ahead.  Products are mma.sync m16n8k16 with fragments read
// as 16-byte vectors: a thread's 16 bytes of a key row feed two score products (the head dimension is permuted
// inside chunks of 32, identically for queries and keys), probabilities go from the score fragments into the
// A operand of the second product, whose other operand ldmatrix turns on the way out of shared memory.  The softmax
// moves on by a whole tile of 64 keys: by 16 keys, with value fragments put together by byte permutes, every product
// of the sums came with four multiplications of the rescaling (16 heads of 192 over 2,048 tokens: 223 us, 184 us now).
//
// The keys of the step's own tokens are in the cache already (the prepare kernel wrote them), so a run that
// continues a cached prefix, a whole prompt and a single token are the same case.
#include "chunk_mma.cuh"

#ifndef TAU_HEAD_DIM
#error "compile with -DTAU_HEAD_DIM=<multiple of 16 up to 256>"
#endif

namespace {

constexpr int D = TAU_HEAD_DIM;
static_assert(D % 16 == 0 && D >= 16 && D <= 256, "head_dim must be a multiple of 16 between 16 and 256");
constexpr int kWarps = 4;
constexpr int kTile = 16;                  // query positions per warp
constexpr int kQkChunks = (D + 31) / 32;
constexpr int kPairs = D / 16;             // pairs of eight columns of the result

__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned pack_bf16(float low, float high) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const unsigned*>(&pair);
}

constexpr int kKeyTile = 64;                       // keys per shared-memory tile: one cache page
constexpr int kChunksPerRow = D / 8;               // 16-byte chunks in a row of D bfloat16
constexpr bool kSwizzle = (kChunksPerRow % 8) == 0;
constexpr int kTileBytes = kKeyTile * D * 2;       // one tile of keys, or of values
// Two blocks to an SM up to heads of 192, one above.  Eight warps to a block with twice the stages read a tile for twice the rows, but leave one block where runs are
// short (us, 16 heads of 192: 2,048 tokens 191 so, 156 with four warps; 60 single tokens and one run of 64 behind 1,000: 346, 211; 8 heads of 256, 2,048
// tokens 189, 192; portions of 120 to 45 behind 1,500: 154, 109).
constexpr int kStages = D <= 128 ? 3 : 2;
// Above 192 elements the queries' fragments do not fit the registers beside the sums (48 bytes spilled, and no room to ask ahead): they lie in shared memory, a lane's
// own where it wrote them (8 heads of 256, portions of 120 to 45 tokens behind 1,500: 127 us with them in registers, 109 so).
constexpr bool kQueriesInShared = D > 192;
constexpr int kBarrierBytes = (kStages * 8 + 8 + 15) / 16 * 16;      // of the stages, and two numbers
constexpr int kSharedBytes = kStages * 2 * kTileBytes + kBarrierBytes + (kQueriesInShared ? kWarps * kQkChunks * 1024 : 0);
#if TAU_HEAD_DIM > 192
#define TAU_PREFILL_BOUNDS __launch_bounds__(kWarps * 32, 1)
#elif TAU_HEAD_DIM > 128
#define TAU_PREFILL_BOUNDS __launch_bounds__(kWarps * 32, 2)
#else
#define TAU_PREFILL_BOUNDS __launch_bounds__(kWarps * 32)
#endif

// Chunk `chunk` of row `row` lies at this byte offset of a tile.  Rows are 2 D bytes apart; the chunk number is
// XORed with the row's low bits so that 8 rows read at the same chunk fall into 8 different bank groups.
__device__ __forceinline__ int tile_offset(int row, int chunk) {
    return row * (D * 2) + ((kSwizzle ? (chunk ^ (row & 7)) : chunk) << 4);
}

__device__ __forceinline__ void copy_async_16(void* destination, const void* source, bool real) {
    const unsigned address = static_cast<unsigned>(__cvta_generic_to_shared(destination));
    const int bytes = real ? 16 : 0;   // 0 source bytes: the 16 destination bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(address), "l"(source), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Block `blockIdx.x` serves `tiles_per_block` neighbouring query tiles of one sequence and `heads_per_block`
// heads of KV head `blockIdx.y / passes`; warp w takes tile w / heads_per_block and head w % heads_per_block.
// Keys and values pass through shared memory in tiles of 64 (one cache page), `kStages` deep, copied with
// cp.async by all threads and read by every warp of the block.
// `kValuePairs`: pairs of eight value columns that are computed, at least those of `value_columns`.
template <int kValuePairs>
__global__ void TAU_PREFILL_BOUNDS
attention_prefill_kernel(const bf16* __restrict__ queries, const bf16* __restrict__ keys, const bf16* __restrict__ values,
                         bf16* __restrict__ out, const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start,
                         const int* __restrict__ page_rows, int page_stride, int page_tokens, int n_seqs, int n_heads, int n_kv_heads,
                         int heads_per_block, int passes, float scale, int window, const float* __restrict__ sinks, int value_columns, int swizzled) {
    if (!swizzled) grid_dependents_launch();      // with bulk copies in flight no other kernel's blocks beside this one's (see the launch)
    grid_dependency_wait();
    extern __shared__ __align__(128) uint8_t tiles[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int tiles_per_block = kWarps / heads_per_block;
    const int group = n_heads / n_kv_heads;
    // Which sequence does this block belong to?  Blocks are numbered sequence by sequence; a block index beyond
    // the last sequence has nothing to do.
    int block = blockIdx.x, seq = 0, row0 = 0, n_new = 0;
    for (; seq < n_seqs; ++seq) {
        row0 = cu_seqlens[seq];
        n_new = cu_seqlens[seq + 1] - row0;
        const int blocks_here = (n_new + kTile * tiles_per_block - 1) / (kTile * tiles_per_block);
        if (block < blocks_here) {
            block = blocks_here - 1 - block;   // the last tiles have the most keys: they start first
            break;
        }
        block -= blocks_here;
    }
    if (seq >= n_seqs) return;   // the whole block leaves
    const int kv_head = blockIdx.y / passes, pass = blockIdx.y % passes;
    const int start = seq_start[seq];                                   // positions cached before this step
    const int tile = block * tiles_per_block + warp / heads_per_block;  // this warp's query tile within the sequence
    const int head_in_group = pass * heads_per_block + warp % heads_per_block;
    const bool active = tile * kTile < n_new && head_in_group < group;   // an idle warp still copies and synchronises
    const int head = kv_head * group + (active ? head_in_group : 0);
    const int position0 = start + tile * kTile;
    const int rows_here = active ? min(kTile, n_new - tile * kTile) : 0;
    const int last_position = position0 + rows_here - 1;               // of this warp
    // The block's range of keys: from the first key that its first tile may see to the last position of its last tile.
    const int block_position0 = start + block * tiles_per_block * kTile;
    const int block_last = start + min(n_new, (block + 1) * tiles_per_block * kTile) - 1;
    int block_first_key = 0;
    if (window > 0 && block_position0 - window + 1 > 0) block_first_key = block_position0 - window + 1;
    const int first_tile = block_first_key / kKeyTile, last_tile = block_last / kKeyTile;
    const int n_key_tiles = last_tile - first_tile + 1;
    const int* pages = page_rows + static_cast<size_t>(seq) * page_stride;
    const size_t head_stride = static_cast<size_t>(page_tokens) * D;

    // Pages whose rows lie as `tile_offset` wants them come as one bulk copy for the keys and one for the values; a page that is not full comes row by row, with
    // zeros behind the last one.  (Row by row, 48 KB a tile, the copies of two blocks of 64 queries took an SM's load/store pipe most of the time.)
    uint64_t* barriers = reinterpret_cast<uint64_t*>(tiles + kStages * 2 * kTileBytes);
    auto whole = [&](int index) { return swizzled && (first_tile + index) * kKeyTile + kKeyTile - 1 <= block_last; };
    volatile int* gone = reinterpret_cast<volatile int*>(barriers + kStages);      // see chunk::barrier_wait; then the tiles up to the last one asked for by bulk copies
    if (swizzled) {
        if (threadIdx.x < kStages) chunk::barrier_init(barriers + threadIdx.x);
        if (threadIdx.x < 2) gone[threadIdx.x] = 0;
        chunk::barriers_ready();
        __syncthreads();
    }
    auto issue_tile = [&](int index) {   // copies key tile `first_tile + index` into stage `index % kStages`
        if (index < n_key_tiles) {
            const int key_tile = first_tile + index;
            const size_t base = (static_cast<size_t>(pages[key_tile * kKeyTile / page_tokens]) * n_kv_heads + kv_head) * head_stride +
                                static_cast<size_t>((key_tile * kKeyTile) % page_tokens) * D;
            uint8_t* stage = tiles + (index % kStages) * 2 * kTileBytes;
            if (whole(index)) {
                if (threadIdx.x == 0 && !gone[0]) {
                    gone[1] = index + 1;
                    uint64_t* barrier = barriers + index % kStages;
                    chunk::barrier_expect(barrier, 2 * kTileBytes);
                    chunk::bulk_copy(stage, keys + base, kTileBytes, barrier);
                    chunk::bulk_copy(stage + kTileBytes, values + base, kTileBytes, barrier);
                }
            } else {
                for (int item = threadIdx.x; item < kKeyTile * kChunksPerRow; item += kWarps * 32) {
                    const int row = item / kChunksPerRow, piece = item % kChunksPerRow;
                    const bool real = key_tile * kKeyTile + row <= block_last;   // rows beyond the block's last position become zero
                    const int place = swizzled ? tile_offset(row, piece) - row * (D * 2) : piece * 16;      // of the piece in its row in memory
                    const size_t source = base + static_cast<size_t>(row) * D + place / 2;
                    copy_async_16(stage + tile_offset(row, piece), keys + (real ? source : base), real);
                    copy_async_16(stage + kTileBytes + tile_offset(row, piece), values + (real ? source : base), real);
                }
            }
        }
        copy_async_commit();   // an empty group keeps the count of groups in step with the tiles
    };

    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
    uint4 q_lo[kQueriesInShared ? 1 : kQkChunks], q_hi[kQueriesInShared ? 1 : kQkChunks];
    uint4* own_queries = reinterpret_cast<uint4*>(tiles + kStages * 2 * kTileBytes + kBarrierBytes) + warp * kQkChunks * 64 + lane;      // [chunk][rows g or g + 8][lane]
    {
        const bool lo_live = g < rows_here, hi_live = g + 8 < rows_here;
        const bf16* base = queries + (static_cast<size_t>(row0 + (active ? tile * kTile : 0)) * n_heads + head) * D;
        const size_t row_stride = static_cast<size_t>(n_heads) * D;
#pragma unroll
        for (int c = 0; c < kQkChunks; ++c) {
            const int e = 32 * c + 8 * t;
            const bool inside = e + 8 <= D;
            const uint4 lo = (lo_live && inside) ? *reinterpret_cast<const uint4*>(base + g * row_stride + e) : zero4;
            const uint4 hi = (hi_live && inside) ? *reinterpret_cast<const uint4*>(base + (g + 8) * row_stride + e) : zero4;
            if constexpr (kQueriesInShared) {
                own_queries[c * 64] = lo;
                own_queries[c * 64 + 32] = hi;
            } else {
                q_lo[c] = lo;
                q_hi[c] = hi;
            }
        }
    }
    const float scale_log2 = scale * 1.4426950408889634f;
    const int position_lo = position0 + g, position_hi = position0 + g + 8;
    float max_lo = -INFINITY, max_hi = -INFINITY, sum_lo = 0.0f, sum_hi = 0.0f;
    float acc[kValuePairs][2][4] = {};
    int warp_first_key = 0;
    if (window > 0 && position0 - window + 1 > 0) warp_first_key = position0 - window + 1;

#pragma unroll
    for (int index = 0; index < kStages - 1; ++index) issue_tile(index);

    for (int index = 0; index < n_key_tiles; ++index) {
        copy_async_wait<kStages - 2>();   // this thread's copies of tile `index` have landed
        if (whole(index)) chunk::barrier_wait(barriers + index % kStages, index / kStages & 1, gone);
        __syncthreads();                  // ... and everyone's; and everyone is done with the stage refilled next
        issue_tile(index + kStages - 1);
        const uint8_t* key_tile = tiles + (index % kStages) * 2 * kTileBytes;
        const uint8_t* value_tile = key_tile + kTileBytes;
        const int tile_key0 = (first_tile + index) * kKeyTile;
        if (!active || tile_key0 > last_position || tile_key0 + kKeyTile <= warp_first_key) continue;   // nothing for this warp here
        // The 16-key steps of the tile that this warp sees anything of.
        const int first_step = max(0, warp_first_key - tile_key0) / 16, steps = min(kKeyTile / 16, (last_position - tile_key0) / 16 + 1);
        const bool edge = tile_key0 + kKeyTile - 1 > position0 || window > 0;      // some query may not see some key
        // All eight column tiles side by side and no branch among them: a product waits for the one before it on the same scores, some 30 cycles, and a tile
        // after the other left the tensor cores idle four fifths of the time.  Keys that nobody sees are masked below.
        float score[kKeyTile / 8][4] = {};
        float block_lo = -INFINITY, block_hi = -INFINITY;
#pragma unroll
        for (int c = 0; c < kQkChunks; ++c) {
            const uint4 lo = kQueriesInShared ? own_queries[c * 64] : q_lo[kQueriesInShared ? 0 : c], hi = kQueriesInShared ? own_queries[c * 64 + 32] : q_hi[kQueriesInShared ? 0 : c];
#pragma unroll
            for (int nt = 0; nt < kKeyTile / 8; ++nt) {
                // Every thread takes part in every product; a chunk beyond the head contributes zeros.
                const uint4 k = (32 * c + 8 * t + 8 <= D) ? *reinterpret_cast<const uint4*>(key_tile + tile_offset(8 * nt + g, 4 * c + t)) : zero4;
                mma_bf16(score[nt], lo.x, hi.x, lo.y, hi.y, k.x, k.y);
                mma_bf16(score[nt], lo.z, hi.z, lo.w, hi.w, k.z, k.w);
            }
        }
#pragma unroll
        for (int nt = 0; nt < kKeyTile / 8; ++nt) {
            // score[nt][0..1]: row g, keys 8 nt + 2t + {0, 1} of the tile; score[nt][2..3]: row g + 8, the same keys.
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int key = tile_key0 + 8 * nt + 2 * t + e;
                const bool lo_ok = !edge || (key <= position_lo && (window == 0 || key > position_lo - window));
                const bool hi_ok = !edge || (key <= position_hi && (window == 0 || key > position_hi - window));
                score[nt][e] = lo_ok ? score[nt][e] * scale_log2 : -INFINITY;
                score[nt][2 + e] = hi_ok ? score[nt][2 + e] * scale_log2 : -INFINITY;
                block_lo = fmaxf(block_lo, score[nt][e]);
                block_hi = fmaxf(block_hi, score[nt][2 + e]);
            }
        }
        block_lo = fmaxf(block_lo, __shfl_xor_sync(0xffffffffu, block_lo, 1));
        block_lo = fmaxf(block_lo, __shfl_xor_sync(0xffffffffu, block_lo, 2));
        block_hi = fmaxf(block_hi, __shfl_xor_sync(0xffffffffu, block_hi, 1));
        block_hi = fmaxf(block_hi, __shfl_xor_sync(0xffffffffu, block_hi, 2));
        // A row that has seen no key yet keeps its maximum at -inf; subtract 0 then, so that nothing becomes NaN.
        const float new_lo = fmaxf(max_lo, block_lo), new_hi = fmaxf(max_hi, block_hi);
        const float shift_lo = new_lo == -INFINITY ? 0.0f : new_lo, shift_hi = new_hi == -INFINITY ? 0.0f : new_hi;
        const float correction_lo = exp2f(max_lo - shift_lo), correction_hi = exp2f(max_hi - shift_hi);
        max_lo = new_lo;
        max_hi = new_hi;
        float share_lo = 0.0f, share_hi = 0.0f;
#pragma unroll
        for (int nt = 0; nt < kKeyTile / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                score[nt][e] = exp2f(score[nt][e] - shift_lo);
                score[nt][2 + e] = exp2f(score[nt][2 + e] - shift_hi);
                share_lo += score[nt][e];
                share_hi += score[nt][2 + e];
            }
        sum_lo = sum_lo * correction_lo + share_lo;
        sum_hi = sum_hi * correction_hi + share_hi;
#pragma unroll
        for (int pair = 0; pair < kValuePairs; ++pair)
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                acc[pair][n][0] *= correction_lo;
                acc[pair][n][1] *= correction_lo;
                acc[pair][n][2] *= correction_hi;
                acc[pair][n][3] *= correction_hi;
            }
#pragma unroll
        for (int step = 0; step < kKeyTile / 16; ++step) {
            if (step < first_step || step >= steps) continue;
            const unsigned pa0 = pack_bf16(score[2 * step][0], score[2 * step][1]), pa1 = pack_bf16(score[2 * step][2], score[2 * step][3]);
            const unsigned pa2 = pack_bf16(score[2 * step + 1][0], score[2 * step + 1][1]), pa3 = pack_bf16(score[2 * step + 1][2], score[2 * step + 1][3]);
#pragma unroll
            for (int pair = 0; pair < kValuePairs; ++pair) {
                const unsigned address = static_cast<unsigned>(__cvta_generic_to_shared(value_tile + tile_offset(16 * step + lane % 16, 2 * pair + lane / 16)));
                unsigned v0, v1, v2, v3;      // keys 0-7 and 8-15 of eight columns, then of the next eight
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v0), "=r"(v1), "=r"(v2), "=r"(v3) : "r"(address) : "memory");
                mma_bf16(acc[pair][0], pa0, pa1, pa2, pa3, v0, v1);
                mma_bf16(acc[pair][1], pa0, pa1, pa2, pa3, v2, v3);
            }
        }
    }
    copy_async_wait<0>();
    if (swizzled && __syncthreads_or(gone[0] != 0)) {   // a wait ran out: no result, and the block ends when the copies in flight have
        const int asked = gone[1];
        for (int index = max(0, asked - (kStages - 1)); index < asked; ++index)
            if (whole(index)) chunk::barrier_wait(barriers + index % kStages, index / kStages & 1, nullptr);
        return;
    }
    if (!active) return;
    sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, 1);
    sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, 2);
    sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, 1);
    sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, 2);
    if (sinks) {   // a sink per head: exp(sink) joins the denominator with no key or value behind it (the maxima are in powers of two)
        const float sink = sinks[head] * 1.4426950408889634f;
        sum_lo += exp2f(sink - max_lo);
        sum_hi += exp2f(sink - max_hi);
    }
    const float inverse_lo = 1.0f / sum_lo, inverse_hi = 1.0f / sum_hi;
    bf16* out_base = out + (static_cast<size_t>(row0 + tile * kTile) * n_heads + head) * D;
    const size_t row_stride = static_cast<size_t>(n_heads) * D;
    const bool in_fours = (reinterpret_cast<uintptr_t>(out) & 3) == 0;      // rows are an even number of elements: all of them start on 4 bytes, or none
    auto store_two = [&](bf16* target, unsigned two) {
        if (in_fours) {
            *reinterpret_cast<unsigned*>(target) = two;
        } else {
            reinterpret_cast<unsigned short*>(target)[0] = static_cast<unsigned short>(two);
            reinterpret_cast<unsigned short*>(target)[1] = static_cast<unsigned short>(two >> 16);
        }
    };
    // acc[pair][n][0], [1]: row g, columns 16 pair + 8 n + 2t + {0, 1}; [2], [3]: row g + 8, the same columns.
#pragma unroll
    for (int pair = 0; pair < kValuePairs; ++pair) {
        if (pair >= value_columns / 16) break;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int column = 16 * pair + 8 * n + 2 * t;
            if (g < rows_here) store_two(out_base + g * row_stride + column, pack_bf16(acc[pair][n][0] * inverse_lo, acc[pair][n][1] * inverse_lo));
            if (g + 8 < rows_here) store_two(out_base + (g + 8) * row_stride + column, pack_bf16(acc[pair][n][2] * inverse_hi, acc[pair][n][3] * inverse_hi));
        }
    }
}

}  // namespace

TAU_EXPORT int tau_attention_prefill_head_dim() { return D; }
// 1 if a bounded wait ran out since the library was loaded (synchronises the device).
TAU_EXPORT int tau_attention_prefill_status() { return chunk::wait_status(); }

// `swizzled`: the pieces of eight elements of row r of a page lie in the order piece ^ (r & 7) (pages of 64 rows, heads of a multiple of 64).
// `value_columns`: only that many columns of the values are read and of the result written (a multiple of 16).
TAU_EXPORT int tau_attention_prefill(const void* queries, const void* keys, const void* values, void* out, const int* cu_seqlens,
                                     const int* seq_start, const int* page_rows, int page_stride, int page_tokens, int n_seqs,
                                     int n_tokens, int n_heads, int n_kv_heads, float scale, int window, const float* sinks, int value_columns,
                                     int swizzled, void* stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (!queries || !keys || !values || !out || !cu_seqlens || !seq_start || !page_rows || n_heads <= 0 || n_kv_heads <= 0 ||
        n_heads % n_kv_heads != 0 || page_tokens <= 0 || window < 0 || value_columns <= 0 || value_columns > D || value_columns % 16 != 0 ||
        (swizzled && (!kSwizzle || page_tokens != kKeyTile || ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(values)) & 15) != 0)))
        return cudaErrorInvalidValue;
    const int group = n_heads / n_kv_heads;
    const int heads_per_block = group >= 4 ? 4 : group == 3 ? 2 : group;     // 1, 2 or 4: divides the 4 warps
    const int passes = (group + heads_per_block - 1) / heads_per_block;
    const int tiles_per_block = kWarps / heads_per_block;
    const int rows_per_block = kTile * tiles_per_block;
    const int blocks = (n_tokens + rows_per_block - 1) / rows_per_block + n_seqs;   // every sequence may leave a ragged block
    const dim3 grid(blocks, n_kv_heads * passes);
    // Values that are narrower than the keys by a third or more have a kernel of their own.
    constexpr int kFewer = kPairs >= 3 ? kPairs * 2 / 3 : kPairs;
    auto* kernel = value_columns <= kFewer * 16 ? attention_prefill_kernel<kFewer> : attention_prefill_kernel<kPairs>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes) != cudaSuccess) return cudaErrorInvalidValue;
    // Kernels that wait for bulk copies start when the kernel before them has finished (the chunks of the delta rule say why).
    tau_launch_as(!swizzled, kernel, dim3(grid), dim3(kWarps * 32), kSharedBytes, static_cast<cudaStream_t>(stream), 
        static_cast<const bf16*>(queries), static_cast<const bf16*>(keys), static_cast<const bf16*>(values), static_cast<bf16*>(out),
        cu_seqlens, seq_start, page_rows, page_stride, page_tokens, n_seqs, n_heads, n_kv_heads, heads_per_block, passes, scale, window, sinks, value_columns, swizzled);
    return tau_launch_status();
}
