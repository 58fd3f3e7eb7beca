// Attention over the paged cache, for every head size, head count and dtype: the prepare step (per-head
// q/k RMSNorm, rotation, cache write) and a plain attention kernel with an online softmax.
//
// Reference counterparts: crates/cuda-kernels/src/kernels/decode_attention.cu:120-181 (`attention_prepare`:
// one block per query or key head of one token: norm, rotate, write Q / append K and V) and :186-250
// (`attention`: 32-bit dot per key, `* rsqrt(d)`, max, exp, sum, probabilities times V).  Here a launch
// covers every token of a step, each with its own sequence, position and page list.
//
// Cache layout of one layer: keys[page][kv_head][slot_in_page][d], the same for values; position `p` of
// sequence `s` lies in page `page_rows[s * page_stride + p / page_tokens]` at `p % page_tokens`.
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int kMaxPerLane = 8;  // head_dim <= 256

template <typename T>
__global__ void attention_prepare_kernel(
    const T* __restrict__ projected, long long projected_stride, T* __restrict__ queries, T* __restrict__ keys,
    T* __restrict__ values, const float* __restrict__ q_weight, const float* __restrict__ k_weight, float eps,
    const float* __restrict__ cos_table, const float* __restrict__ sin_table, int rotary_dim,
    const int* __restrict__ positions, const int* __restrict__ token_seq, const int* __restrict__ page_rows,
    int page_stride, int page_tokens, int n_heads, int n_kv_heads, int head_dim, int write_cache) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int token = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int position = positions[token];
    const int heads_total = write_cache ? n_heads + 2 * n_kv_heads : n_heads;
    const T* row = projected + static_cast<size_t>(token) * projected_stride;
    const int half = rotary_dim / 2;
    size_t cache_base = 0;
    if (write_cache) {
        const int page = page_rows[static_cast<size_t>(token_seq[token]) * page_stride + position / page_tokens];
        cache_base = (static_cast<size_t>(page) * n_kv_heads * page_tokens + position % page_tokens) * head_dim;
    }
    for (int head = warp; head < heads_total; head += warps) {
        const T* source = row + static_cast<size_t>(head) * head_dim;
        T* target;
        const float* weight;
        bool rotate = true;
        if (head < n_heads) {
            target = queries + (static_cast<size_t>(token) * n_heads + head) * head_dim;
            weight = q_weight;
        } else {
            const int kv_head = (head - n_heads) % n_kv_heads;
            const bool is_key = head < n_heads + n_kv_heads;
            target = (is_key ? keys : values) + cache_base + static_cast<size_t>(kv_head) * page_tokens * head_dim;
            weight = is_key ? k_weight : nullptr;
            rotate = is_key;
            if (!is_key) {  // values are stored as projected
                for (int e = lane; e < head_dim; e += 32) target[e] = source[e];
                continue;
            }
        }
        float inverse = 1.0f;
        if (weight) {
            float squares = 0.0f;
            for (int e = lane; e < head_dim; e += 32) {
                const float value = to_float(source[e]);
                squares += value * value;
            }
            inverse = rsqrtf(warp_sum(squares) / static_cast<float>(head_dim) + eps);
        }
        // Normalised values are rounded to the storage type, rotated in 32-bit and rounded once more.
        auto normalized = [&](int e) {
            const float value = to_float(source[e]);
            return weight ? round_through<T>(value * inverse * weight[e]) : value;
        };
        if (rotate && half > 0) {
            const float* cos_row = cos_table + static_cast<size_t>(position) * half;
            const float* sin_row = sin_table + static_cast<size_t>(position) * half;
            for (int j = lane; j < half; j += 32) {
                const float first = normalized(j), second = normalized(j + half);
                const float c = cos_row[j], s = sin_row[j];
                target[j] = from_float<T>(first * c - second * s);
                target[j + half] = from_float<T>(second * c + first * s);
            }
            for (int e = rotary_dim + lane; e < head_dim; e += 32) target[e] = from_float<T>(normalized(e));
        } else {
            for (int e = lane; e < head_dim; e += 32) target[e] = from_float<T>(normalized(e));
        }
    }
}

// The same for head sizes of 32 * PER elements that are rotated whole (or not at all): a lane holds PER neighbouring
// elements, loaded and stored as one vector; the element it is paired with by the rotation lies in lane ^ 16.
template <typename T, int PER> struct alignas(sizeof(T) * PER) HeadVector { T v[PER]; };

template <typename T, int PER>
__global__ void attention_prepare_vec_kernel(
    const T* __restrict__ projected, long long projected_stride, T* __restrict__ queries, T* __restrict__ keys,
    T* __restrict__ values, const float* __restrict__ q_weight, const float* __restrict__ k_weight, float eps,
    const float* __restrict__ cos_table, const float* __restrict__ sin_table, int rotary_dim,
    const int* __restrict__ positions, const int* __restrict__ token_seq, const int* __restrict__ page_rows,
    int page_stride, int page_tokens, int n_heads, int n_kv_heads, int write_cache) {
    grid_dependents_launch();
    grid_dependency_wait();
    constexpr int head_dim = 32 * PER;
    typedef HeadVector<T, PER> Vector;
    const int token = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int position = positions[token];
    const int heads_total = write_cache ? n_heads + 2 * n_kv_heads : n_heads;
    const T* row = projected + static_cast<size_t>(token) * projected_stride;
    size_t cache_base = 0;
    if (write_cache) {
        const int page = page_rows[static_cast<size_t>(token_seq[token]) * page_stride + position / page_tokens];
        cache_base = (static_cast<size_t>(page) * n_kv_heads * page_tokens + position % page_tokens) * head_dim;
    }
    // This lane's rotation coefficients: elements PER * (lane % 16) + i of the half-width tables.
    float cosines[PER], sines[PER];
    if (rotary_dim) {
        const size_t table = static_cast<size_t>(position) * (head_dim / 2) + PER * (lane & 15);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            cosines[i] = cos_table[table + i];
            sines[i] = lane < 16 ? -sin_table[table + i] : sin_table[table + i];   // first half: x cos - partner sin; second half: x cos + partner sin
        }
    }
    // A warp takes the heads warp, warp + warps, ...; their vectors are asked for several at a time, so that the loads of
    // one token's heads travel together instead of one after another.
    constexpr int kBatch = 6;
    for (int first = warp; first < heads_total; first += warps * kBatch) {
        Vector loaded[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const int head = first + b * warps;
            if (head < heads_total) loaded[b] = *reinterpret_cast<const Vector*>(row + static_cast<size_t>(head) * head_dim + PER * lane);
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const int head = first + b * warps;
            if (head >= heads_total) break;
            T* target;
            const float* weight;
            if (head < n_heads) {
                target = queries + (static_cast<size_t>(token) * n_heads + head) * head_dim;
                weight = q_weight;
            } else {
                const bool is_key = head < n_heads + n_kv_heads;
                const int kv_head = head - n_heads - (is_key ? 0 : n_kv_heads);
                target = (is_key ? keys : values) + cache_base + static_cast<size_t>(kv_head) * page_tokens * head_dim;
                weight = k_weight;
                if (!is_key) {  // values are stored as projected
                    *reinterpret_cast<Vector*>(target + PER * lane) = loaded[b];
                    continue;
                }
            }
            float value[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) value[i] = to_float(loaded[b].v[i]);
            if (weight) {
                float squares = 0.0f;
#pragma unroll
                for (int i = 0; i < PER; ++i) squares += value[i] * value[i];
                const float inverse = rsqrtf(warp_sum(squares) / static_cast<float>(head_dim) + eps);
#pragma unroll
                for (int i = 0; i < PER; ++i) value[i] = round_through<T>(value[i] * inverse * weight[PER * lane + i]);
            }
            Vector result;
            if (rotary_dim) {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const float partner = __shfl_xor_sync(0xffffffffu, value[i], 16);
                    result.v[i] = from_float<T>(value[i] * cosines[i] + partner * sines[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < PER; ++i) result.v[i] = from_float<T>(value[i]);
            }
            *reinterpret_cast<Vector*>(target + PER * lane) = result;
        }
    }
}

// One warp per (token, query head).  Keys are taken 32 at a time: lane `l` scores key `l` of the chunk
// with a full dot product, the chunk's maximum and sum are found by shuffles, and the values are
// accumulated with each lane owning elements `lane, lane + 32, ...` of the head.
template <typename T>
__global__ void attention_generic_kernel(
    const T* __restrict__ queries, const T* __restrict__ keys, const T* __restrict__ values, T* __restrict__ out,
    const int* __restrict__ positions, const int* __restrict__ token_seq, const int* __restrict__ page_rows,
    int page_stride, int page_tokens, int n_tokens, int n_heads, int n_kv_heads, int head_dim, float scale, int window) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ float query_shared[];  // [warps][head_dim]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const long long pair = static_cast<long long>(blockIdx.x) * warps + warp;
    if (pair >= static_cast<long long>(n_tokens) * n_heads) return;  // whole warps leave; no block-wide sync follows
    const int token = static_cast<int>(pair / n_heads), head = static_cast<int>(pair % n_heads);
    const int kv_head = head / (n_heads / n_kv_heads);
    const int position = positions[token];
    const int* pages = page_rows + static_cast<size_t>(token_seq[token]) * page_stride;
    float* query = query_shared + warp * head_dim;
    const T* query_row = queries + (static_cast<size_t>(token) * n_heads + head) * head_dim;
    for (int e = lane; e < head_dim; e += 32) query[e] = to_float(query_row[e]);
    __syncwarp();

    const int first_key = (window > 0 && position - window + 1 > 0) ? position - window + 1 : 0;
    float running_max = -INFINITY, running_sum = 0.0f;
    float acc[kMaxPerLane];
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) acc[i] = 0.0f;
    const size_t head_stride = static_cast<size_t>(page_tokens) * head_dim;

    for (int chunk = first_key; chunk <= position; chunk += 32) {
        const int key = chunk + lane;
        const bool live = key <= position;
        float score = -INFINITY;
        size_t offset = 0;
        if (live) {
            const int page = pages[key / page_tokens];
            offset = (static_cast<size_t>(page) * n_kv_heads + kv_head) * head_stride +
                     static_cast<size_t>(key % page_tokens) * head_dim;
            const T* key_row = keys + offset;
            float dot = 0.0f;
            for (int e = 0; e < head_dim; ++e) dot = fmaf(query[e], to_float(key_row[e]), dot);
            score = dot * scale;
        }
        const float chunk_max = warp_max(score);
        const float new_max = fmaxf(running_max, chunk_max);  // finite: lane 0 of every chunk is live
        const float correction = expf(running_max - new_max);
        const float weight = live ? expf(score - new_max) : 0.0f;
        running_sum = running_sum * correction + warp_sum(weight);
        running_max = new_max;
#pragma unroll
        for (int i = 0; i < kMaxPerLane; ++i) acc[i] *= correction;
        const int in_chunk = min(32, position - chunk + 1);
        for (int j = 0; j < in_chunk; ++j) {
            const float w = __shfl_sync(0xffffffffu, weight, j);
            const size_t value_offset = __shfl_sync(0xffffffffu, static_cast<unsigned long long>(offset), j);
            const T* value_row = values + value_offset;
#pragma unroll
            for (int i = 0; i < kMaxPerLane; ++i) {
                const int e = lane + 32 * i;
                if (e < head_dim) acc[i] = fmaf(w, to_float(value_row[e]), acc[i]);
            }
        }
    }
    T* target = out + (static_cast<size_t>(token) * n_heads + head) * head_dim;
    const float inverse = 1.0f / running_sum;
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
        const int e = lane + 32 * i;
        if (e < head_dim) target[e] = from_float<T>(acc[i] * inverse);
    }
}

// Causal 32-bit attention of runs of new tokens, tile by tile.  The kernel above reads every key once per query and head (777 tokens, 16 heads of 128:
// 2.6 ms, bound by those reads); here a block owns 64 queries of a head and reads a page of 64 keys and values once for all of them.  Scores: 4 x 4
// a thread, queries and keys turned in shared memory so that both are read 16 bytes at a time; weights go through shared memory (over the keys,
// which are done with) to the sums, 4 queries by kDim / 16 elements a thread.  100 KB of shared memory at kDim 128: two blocks to an SM.
// 16 heads of 128 over 777 tokens: 227 us, 2,647 us by a warp to a token and head.
// grid (tiles of 64 queries, heads): tiles of sequence s are numbered from cu_seqlens[s] / 64 + s on; block 256.
constexpr int kTileTokens = 64, kTilePitch = 68;      // floats of a turned row: 16-byte aligned, rows 4 banks apart
template <int kDim> constexpr int tiled_bytes() { return (2 * kDim * kTilePitch + kTileTokens * kDim) * 4; }

template <int kDim>
__global__ void __launch_bounds__(256)
attention_tiled_kernel(const float* __restrict__ queries, const float* __restrict__ keys, const float* __restrict__ values, float* __restrict__ out,
                       const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start, const int* __restrict__ page_rows, int page_stride, int n_seqs, int n_heads,
                       int n_kv_heads, float scale, int window) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ __align__(16) float shared[];
    float* qs = shared;                              // [kDim][kTilePitch]
    float* ks = qs + kDim * kTilePitch;              // [kDim][kTilePitch], then the weights [key][kTilePitch]
    float* vs = ks + kDim * kTilePitch;              // [key][kDim]
    constexpr int kPer = kDim / 16;
    const int head = blockIdx.y, kv_head = head / (n_heads / n_kv_heads), tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    int sequence = 0;
    while (sequence + 1 < n_seqs && cu_seqlens[sequence + 1] / kTileTokens + sequence + 1 <= static_cast<int>(blockIdx.x)) ++sequence;
    const int begin = cu_seqlens[sequence], first = (static_cast<int>(blockIdx.x) - begin / kTileTokens - sequence) * kTileTokens;      // of the run's tokens
    const int live = min(kTileTokens, cu_seqlens[sequence + 1] - begin - first);
    if (live <= 0) return;                           // a number that no tile has
    const int position0 = seq_start[sequence] + first, last = position0 + live - 1;
    for (int item = threadIdx.x; item < kTileTokens * kDim / 4; item += 256) {
        const int row = item % kTileTokens, column = item / kTileTokens * 4;
        const float4 q = row < live ? *reinterpret_cast<const float4*>(queries + (static_cast<size_t>(begin + first + row) * n_heads + head) * kDim + column) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        qs[column * kTilePitch + row] = q.x; qs[(column + 1) * kTilePitch + row] = q.y; qs[(column + 2) * kTilePitch + row] = q.z; qs[(column + 3) * kTilePitch + row] = q.w;
    }
    float acc[4][kPer] = {}, top[4], total[4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) top[i] = -INFINITY;
    const int first_key = window > 0 && position0 - window + 1 > 0 ? position0 - window + 1 : 0;
    for (int page = first_key / kTileTokens; page * kTileTokens <= last; ++page) {
        const size_t source = (static_cast<size_t>(page_rows[sequence * page_stride + page]) * n_kv_heads + kv_head) * kTileTokens * kDim;
        __syncthreads();                             // the weights and values before are read
        for (int item = threadIdx.x; item < kTileTokens * kDim / 4; item += 256) {
            const int row = item % kTileTokens, column = item / kTileTokens * 4;
            const bool written = page * kTileTokens + row <= last;      // positions behind the last query may hold anything
            const float4 k = written ? *reinterpret_cast<const float4*>(keys + source + row * kDim + column) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            ks[column * kTilePitch + row] = k.x; ks[(column + 1) * kTilePitch + row] = k.y; ks[(column + 2) * kTilePitch + row] = k.z; ks[(column + 3) * kTilePitch + row] = k.w;
            const int value_row = item / (kDim / 4);
            *reinterpret_cast<float4*>(vs + item * 4) = page * kTileTokens + value_row <= last ? *reinterpret_cast<const float4*>(values + source + item * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncthreads();
        float scores[4][4] = {};
#pragma unroll 8
        for (int e = 0; e < kDim; ++e) {
            const float4 q = *reinterpret_cast<const float4*>(qs + e * kTilePitch + ty * 4), k = *reinterpret_cast<const float4*>(ks + e * kTilePitch + tx * 4);
            const float a[4] = {q.x, q.y, q.z, q.w}, b[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) scores[i][j] = fmaf(a[i], b[j], scores[i][j]);
        }
        __syncthreads();                             // the keys are done with
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int position = position0 + ty * 4 + i;
            float high = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = page * kTileTokens + tx * 4 + j;
                scores[i][j] = key <= position && (window <= 0 || key > position - window) ? scores[i][j] * scale : -INFINITY;
                high = fmaxf(high, scores[i][j]);
            }
#pragma unroll
            for (int offset = 8; offset > 0; offset >>= 1) high = fmaxf(high, __shfl_xor_sync(0xffffffffu, high, offset));
            const float new_top = fmaxf(top[i], high), base = new_top == -INFINITY ? 0.0f : new_top;      // a row may see nothing of a page
            const float correction = expf(top[i] - base);
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                scores[i][j] = expf(scores[i][j] - base);
                sum += scores[i][j];
            }
#pragma unroll
            for (int offset = 8; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
            total[i] = total[i] * correction + sum;
            top[i] = new_top;
#pragma unroll
            for (int e = 0; e < kPer; ++e) acc[i][e] *= correction;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(ks + (tx * 4 + j) * kTilePitch + ty * 4) = make_float4(scores[0][j], scores[1][j], scores[2][j], scores[3][j]);
        __syncthreads();
        const int seen = min(kTileTokens, last - page * kTileTokens + 1);
        // Where some query of the tile does not see some key of the page, a value meets its own query's weight only (zero times an infinity is not zero).
        const bool careful = page * kTileTokens + kTileTokens - 1 > position0 || (window > 0 && page * kTileTokens <= last - window);
        auto add = [&](int key, auto checked) {
            const float4 weight = *reinterpret_cast<const float4*>(ks + key * kTilePitch + ty * 4);
            const float a[4] = {weight.x, weight.y, weight.z, weight.w};
#pragma unroll
            for (int e = 0; e < kPer; e += 4) {      // a thread's elements lie 64 apart in fours
                const float4 v = *reinterpret_cast<const float4*>(vs + key * kDim + e / 4 * 64 + tx * 4);
                const float b[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (!checked || a[i] != 0.0f) acc[i][e + j] = fmaf(a[i], b[j], acc[i][e + j]);
            }
        };
        if (careful) {
#pragma unroll 2
            for (int key = 0; key < seen; ++key) add(key, std::true_type{});
        } else {
#pragma unroll 4
            for (int key = 0; key < seen; ++key) add(key, std::false_type{});
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (ty * 4 + i >= live) continue;
        const float inverse = 1.0f / total[i];
        float* target = out + (static_cast<size_t>(begin + first + ty * 4 + i) * n_heads + head) * kDim;
#pragma unroll
        for (int e = 0; e < kPer; e += 4)
            *reinterpret_cast<float4*>(target + e / 4 * 64 + tx * 4) = make_float4(acc[i][e] * inverse, acc[i][e + 1] * inverse, acc[i][e + 2] * inverse, acc[i][e + 3] * inverse);
    }
}

}  // namespace

TAU_EXPORT int tau_attention_prepare(
    int dtype, const void* projected, long long projected_stride, void* queries, void* keys, void* values,
    const float* q_weight, const float* k_weight, float eps, const float* cos_table, const float* sin_table,
    int rotary_dim, const int* positions, const int* token_seq, const int* page_rows, int page_stride, int page_tokens,
    int n_tokens, int n_heads, int n_kv_heads, int head_dim, int write_cache, void* stream) {
    if (n_tokens <= 0) return 0;
    if (!projected || !queries || !positions || head_dim <= 0 || head_dim > 32 * kMaxPerLane || n_heads <= 0 ||
        n_kv_heads <= 0 || rotary_dim < 0 || rotary_dim > head_dim || (rotary_dim & 1) ||
        (rotary_dim > 0 && (!cos_table || !sin_table)) ||
        (write_cache && (!keys || !values || !token_seq || !page_rows || page_tokens <= 0)))
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int heads_total = write_cache ? n_heads + 2 * n_kv_heads : n_heads;
    const int threads = 32 * (heads_total < 8 ? heads_total : 8);
    // The vector form: heads of 64, 128 or 256 elements rotated whole or not at all, rows aligned to a vector.
    const bool whole = (rotary_dim == 0 || rotary_dim == head_dim) && (head_dim == 64 || head_dim == 128 || head_dim == 256) &&
                       projected_stride % (head_dim / 32) == 0;
#define TAU_PREPARE_VEC(T, PER)                                                                                                     \
    tau_launch(attention_prepare_vec_kernel<T, PER>, dim3(n_tokens), dim3(threads), 0, s, static_cast<const T*>(projected),          \
               projected_stride, static_cast<T*>(queries), static_cast<T*>(keys), static_cast<T*>(values), q_weight, k_weight, eps,  \
               cos_table, sin_table, rotary_dim, positions, token_seq, page_rows, page_stride, page_tokens, n_heads, n_kv_heads,     \
               write_cache)
    if (whole && dtype == TAU_BF16) {
        if (head_dim == 64) TAU_PREPARE_VEC(bf16, 2);
        else if (head_dim == 128) TAU_PREPARE_VEC(bf16, 4);
        else TAU_PREPARE_VEC(bf16, 8);
        return tau_launch_status();
    }
    if (whole && dtype == TAU_F32) {
        if (head_dim == 64) TAU_PREPARE_VEC(float, 2);
        else if (head_dim == 128) TAU_PREPARE_VEC(float, 4);
        else TAU_PREPARE_VEC(float, 8);
        return tau_launch_status();
    }
#undef TAU_PREPARE_VEC
    if (dtype == TAU_F32)
        tau_launch(attention_prepare_kernel<float>, dim3(n_tokens), dim3(threads), 0, s, 
            static_cast<const float*>(projected), projected_stride, static_cast<float*>(queries), static_cast<float*>(keys),
            static_cast<float*>(values), q_weight, k_weight, eps, cos_table, sin_table, rotary_dim, positions, token_seq,
            page_rows, page_stride, page_tokens, n_heads, n_kv_heads, head_dim, write_cache);
    else if (dtype == TAU_BF16)
        tau_launch(attention_prepare_kernel<bf16>, dim3(n_tokens), dim3(threads), 0, s, 
            static_cast<const bf16*>(projected), projected_stride, static_cast<bf16*>(queries), static_cast<bf16*>(keys),
            static_cast<bf16*>(values), q_weight, k_weight, eps, cos_table, sin_table, rotary_dim, positions, token_seq,
            page_rows, page_stride, page_tokens, n_heads, n_kv_heads, head_dim, write_cache);
    else
        return cudaErrorInvalidValue;
    return tau_launch_status();
}

TAU_EXPORT int tau_attention_generic(
    int dtype, const void* queries, const void* keys, const void* values, void* out, const int* positions,
    const int* token_seq, const int* page_rows, int page_stride, int page_tokens, int n_tokens, int n_heads,
    int n_kv_heads, int head_dim, float scale, int window, void* stream) {
    if (n_tokens <= 0) return 0;
    if (!queries || !keys || !values || !out || !positions || !token_seq || !page_rows || head_dim <= 0 ||
        head_dim > 32 * kMaxPerLane || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0 || page_tokens <= 0 ||
        window < 0)
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    constexpr int warps = 4;
    const long long pairs = static_cast<long long>(n_tokens) * n_heads;
    const unsigned blocks = static_cast<unsigned>((pairs + warps - 1) / warps);
    const size_t shared = warps * head_dim * sizeof(float);
    if (dtype == TAU_F32)
        tau_launch(attention_generic_kernel<float>, dim3(blocks), dim3(warps * 32), shared, s, 
            static_cast<const float*>(queries), static_cast<const float*>(keys), static_cast<const float*>(values),
            static_cast<float*>(out), positions, token_seq, page_rows, page_stride, page_tokens, n_tokens, n_heads,
            n_kv_heads, head_dim, scale, window);
    else if (dtype == TAU_BF16)
        tau_launch(attention_generic_kernel<bf16>, dim3(blocks), dim3(warps * 32), shared, s, 
            static_cast<const bf16*>(queries), static_cast<const bf16*>(keys), static_cast<const bf16*>(values),
            static_cast<bf16*>(out), positions, token_seq, page_rows, page_stride, page_tokens, n_tokens, n_heads,
            n_kv_heads, head_dim, scale, window);
    else
        return cudaErrorInvalidValue;
    return tau_launch_status();
}

// 32-bit attention of runs of new tokens (`cu_seqlens` bounds them, `seq_start` positions were cached before), heads of 64 or 128 elements, pages of 64.
TAU_EXPORT int tau_attention_tiled(const float* queries, const float* keys, const float* values, float* out, const int* cu_seqlens, const int* seq_start,
                                   const int* page_rows, int page_stride, int n_tokens, int n_seqs, int n_heads, int n_kv_heads, int head_dim, float scale, int window,
                                   void* stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return 0;
    if (!queries || !keys || !values || !out || !cu_seqlens || !seq_start || !page_rows || (head_dim != 64 && head_dim != 128) || n_heads <= 0 || n_heads > 65535
        || n_kv_heads <= 0 || n_heads % n_kv_heads != 0 || window < 0
        || ((reinterpret_cast<uintptr_t>(queries) | reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(values) | reinterpret_cast<uintptr_t>(out)) & 15) != 0)
        return cudaErrorInvalidValue;
    auto* kernel = head_dim == 64 ? attention_tiled_kernel<64> : attention_tiled_kernel<128>;
    const int bytes = head_dim == 64 ? tiled_bytes<64>() : tiled_bytes<128>();
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return cudaErrorInvalidValue;
    tau_launch(kernel, dim3(n_tokens / kTileTokens + n_seqs, n_heads), dim3(256), bytes, static_cast<cudaStream_t>(stream), queries, keys, values, out, cu_seqlens, seq_start,
               page_rows, page_stride, n_seqs, n_heads, n_kv_heads, scale, window);
    return tau_launch_status();
}
