// The gated delta rule: a matrix state S (key_dim x value_dim) per head that decays, is corrected towards the token's value along
// the token's key, and is read with the token's query:
//
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q            (the read-out sees the token's own write)
//
// `q` and `k` belong to key heads (value head h reads key head h / (heads / key_heads)); q and k are unit vectors per head
// (x / sqrt(sum x^2 + 1e-6)), q also times key_dim^-1/2; beta = sigmoid(b); g = exp(-exp(A_log) softplus(a + dt_bias)).
//
//   prepare:  per token, in 32-bit and in place on [q | k | v] rows: the two unit norms and the query's scale, k . q per key head,
//             and (g, beta) per value head from the pre-activations.
//   walk:     one block owns (sequence, head, tile of value columns) and walks the run's tokens in order; what the next few tokens
//             bring (q, k, the tile's values, g, beta, k . q) is on its way into a ring in shared memory meanwhile (cp.async), so that
//             a token waits for shared memory and one barrier, not for a round trip to memory.  A column of S is shared by
//             kSplit threads, each with kRows key rows in registers.  With a = S_old^T k and b = S_old^T q (both from the state
//             before the token, one pass and one barrier) the token's result is u = beta (v - g a), o = g b + u (k . q),
//             S = g S_old + k u^T: the equations above with the decay pulled out of the sums.
//
// A decay per head and key channel (`channel`: g is a vector over the rows of S, from pre-activations [tokens, heads * key_dim]) walks the
// same way with the vector inside the sums: a = S_old^T (g * k), b = S_old^T (g * q), u = beta (v - a), o = b + u (k . q),
// S = g * S_old + k u^T.
//
// The state is 32-bit and lives in the cache, [heads, value_dim, key_dim] per slot.  TAU_KEY_DIM fixes key_dim.
#include "chunk_mma.cuh"

#ifndef TAU_KEY_DIM
#error "compile with -DTAU_KEY_DIM=<key elements per head>"
#endif

namespace {

constexpr int kDim = TAU_KEY_DIM;
constexpr int kSplit = kDim <= 16 ? 1 : kDim <= 32 ? 2 : kDim <= 64 ? 4 : kDim <= 128 ? 8 : kDim <= 256 ? 16 : 32;   // threads that share a column
constexpr int kRows = (kDim + kSplit - 1) / kSplit;
constexpr bool kExact = kDim % kSplit == 0;      // every thread's rows exist

// grid: tokens; block: 128.  rows [tokens, stride] float: q at q_offset (key_heads * kDim), k at k_offset.  pre [tokens, pre_stride]:
// the pre-activations of beta, then (without `channel`) of the decay's step.  gates [tokens, heads, 2] = (g, beta); kq [tokens, key_heads].
// `channel` [tokens, heads * kDim]: the pre-activations of a decay per head and key channel (dt_bias is then as wide), replaced by the
// decays themselves; g of `gates` is then 1.
__global__ void __launch_bounds__(128)
delta_prepare_kernel(float* __restrict__ rows, long long stride, int q_offset, int k_offset, const float* __restrict__ pre, int pre_stride,
                     const float* __restrict__ a_log, const float* __restrict__ dt_bias, float* __restrict__ gates, float* __restrict__ kq,
                     float* __restrict__ channel, int heads, int key_heads, float query_scale) {
    grid_dependents_launch();
    grid_dependency_wait();
    constexpr int kOwn = (kDim + 31) / 32;      // elements of a lane
    const int token = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    float* row = rows + static_cast<size_t>(token) * stride;
    for (int head = warp; head < key_heads; head += warps) {
        float* q = row + q_offset + head * kDim;
        float* k = row + k_offset + head * kDim;
        float own_q[kOwn], own_k[kOwn], qq = 0.0f, kk = 0.0f;      // one round trip to memory, not one for the sums and one for the results
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const bool there = lane + 32 * i < kDim;
            own_q[i] = there ? q[lane + 32 * i] : 0.0f;
            own_k[i] = there ? k[lane + 32 * i] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            qq = fmaf(own_q[i], own_q[i], qq);
            kk = fmaf(own_k[i], own_k[i], kk);
        }
        const float q_factor = query_scale / sqrtf(warp_sum(qq) + 1e-6f), k_factor = 1.0f / sqrtf(warp_sum(kk) + 1e-6f);
        float dot = 0.0f;
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const float a = own_q[i] * q_factor, b = own_k[i] * k_factor;
            if (lane + 32 * i < kDim) {
                q[lane + 32 * i] = a;
                k[lane + 32 * i] = b;
            }
            dot = fmaf(a, b, dot);
        }
        dot = warp_sum(dot);
        if (lane == 0) kq[static_cast<size_t>(token) * key_heads + head] = dot;
    }
    for (int head = threadIdx.x; head < heads; head += blockDim.x) {
        const float b = pre[static_cast<size_t>(token) * pre_stride + head];
        float decay = 1.0f;
        if (!channel) {
            const float z = pre[static_cast<size_t>(token) * pre_stride + heads + head] + dt_bias[head];
            const float soft = z > 20.0f ? z : log1pf(expf(z));
            decay = expf(-expf(a_log[head]) * soft);
        }
        gates[(static_cast<size_t>(token) * heads + head) * 2] = decay;
        gates[(static_cast<size_t>(token) * heads + head) * 2 + 1] = 1.0f / (1.0f + expf(-b));
    }
    if (channel) {
        float* steps = channel + static_cast<size_t>(token) * heads * kDim;
        for (int index = threadIdx.x; index < heads * kDim; index += blockDim.x) {
            const float z = steps[index] + dt_bias[index];
            const float soft = z > 20.0f ? z : log1pf(expf(z));
            steps[index] = expf(-expf(a_log[index / kDim]) * soft);
        }
    }
}

// Four bytes from global to shared memory without passing a register; complete after `copy_wait` and a barrier.
__device__ __forceinline__ void copy_float(float* target, const float* source) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(target))), "l"(source) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int kRing = kDim <= 256 ? 8 : 4;      // tokens whose q, k, values and gates are in shared memory or on their way there

template <int kColumns, bool kChannel>
__global__ void __launch_bounds__(kColumns * kSplit)
delta_rule_kernel(const float* __restrict__ rows, long long stride, int q_offset, int k_offset, int v_offset, const float* __restrict__ gates,
                  const float* __restrict__ kq, const float* __restrict__ channel, float* __restrict__ state, long long slot_stride,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, float* __restrict__ out, int heads, int key_heads, int value_dim,
                  int below) {
    grid_dependents_launch();
    grid_dependency_wait();
    __shared__ __align__(16) float qs[kRing][kDim], ks[kRing][kDim];      // a thread's rows start on 16 bytes where kRows is a multiple of 4
    __shared__ __align__(16) float gs[kRing][kChannel ? kDim : 1];        // the head's decay per key channel
    __shared__ float vs[kRing][kColumns], scalars[kRing][4], part_a[2][kSplit][kColumns], part_b[2][kSplit][kColumns];
    const int head = blockIdx.x, sequence = blockIdx.y, key_head = head / (heads / key_heads);
    const int local = threadIdx.x % kColumns, part = threadIdx.x / kColumns, row0 = part * kRows;
    const int column = blockIdx.z * kColumns + local;
    const bool live = column < value_dim;
    float* record = state + static_cast<size_t>(seq_slot[sequence]) * slot_stride + (static_cast<size_t>(head) * value_dim + (live ? column : 0)) * kDim;
    float S[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) S[r] = (live && row0 + r < kDim) ? record[row0 + r] : 0.0f;
    const int begin = cu_seqlens[sequence], end = cu_seqlens[sequence + 1];
    if (end - begin >= below) return;      // the chunk kernels' run
    constexpr int kStage = (kDim + kColumns * kSplit - 1) / (kColumns * kSplit);
    // Asks for token `begin + index` (if the run has it) in its place of the ring; one group of copies per token, empty ones too, so
    // that the count of groups in flight says which tokens have arrived.
    auto stage = [&](int index) {
        const int token = begin + index, place = index % kRing;
        if (token < end) {
            const float* row = rows + static_cast<size_t>(token) * stride;
#pragma unroll
            for (int i = 0; i < kStage; ++i) {
                const int d = threadIdx.x + i * kColumns * kSplit;
                if (d < kDim) {
                    copy_float(&qs[place][d], row + q_offset + key_head * kDim + d);
                    copy_float(&ks[place][d], row + k_offset + key_head * kDim + d);
                    if (kChannel) copy_float(&gs[place][d], channel + (static_cast<size_t>(token) * heads + head) * kDim + d);
                }
            }
            if (part == 0 && live) copy_float(&vs[place][local], row + v_offset + head * value_dim + column);
            if (threadIdx.x < 2) copy_float(&scalars[place][threadIdx.x], gates + (static_cast<size_t>(token) * heads + head) * 2 + threadIdx.x);
            if (threadIdx.x == 2) copy_float(&scalars[place][2], kq + static_cast<size_t>(token) * key_heads + key_head);
        }
        copy_commit();
    };
#pragma unroll
    for (int index = 0; index < kRing - 1; ++index) stage(index);
    copy_wait<kRing - 2>();      // the first token has arrived
    __syncthreads();
    for (int token = begin; token < end; ++token) {
        const int index = token - begin, place = index % kRing, half = index & 1;
        const float value = live ? vs[place][local] : 0.0f;
        const float decay = scalars[place][0], beta = scalars[place][1], key_query = scalars[place][2];
        float key[kRows], keep[kChannel ? kRows : 1];
        float a[2] = {0.0f, 0.0f}, b[2] = {0.0f, 0.0f};
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            key[r] = (kExact || row0 + r < kDim) ? ks[place][row0 + r] : 0.0f;
            const float query = (kExact || row0 + r < kDim) ? qs[place][row0 + r] : 0.0f;
            if (kChannel) {
                keep[r] = (kExact || row0 + r < kDim) ? gs[place][row0 + r] : 0.0f;
                const float kept = keep[r] * S[r];
                a[r & 1] = fmaf(kept, key[r], a[r & 1]);
                b[r & 1] = fmaf(kept, query, b[r & 1]);
            } else {
                a[r & 1] = fmaf(S[r], key[r], a[r & 1]);
                b[r & 1] = fmaf(S[r], query, b[r & 1]);
            }
        }
        part_a[half][part][local] = a[0] + a[1];
        part_b[half][part][local] = b[0] + b[1];
        // The place of the token before this one is free: everybody has passed that token's barrier, and read its place before it.
        stage(index + kRing - 1);
        copy_wait<kRing - 2>();      // this thread's copies of the next token are done; the barrier shows everybody's
        __syncthreads();
        float sum_a = 0.0f, sum_b = 0.0f;
#pragma unroll
        for (int p = 0; p < kSplit; ++p) {
            sum_a += part_a[half][p][local];
            sum_b += part_b[half][p][local];
        }
        const float update = beta * (value - decay * sum_a);
#pragma unroll
        for (int r = 0; r < kRows; ++r) S[r] = fmaf(kChannel ? keep[r] : decay, S[r], key[r] * update);
        if (part == 0 && live) out[(static_cast<size_t>(token) * heads + head) * value_dim + column] = fmaf(decay, sum_b, update * key_query);
    }
    copy_wait<0>();
    if (live) {
#pragma unroll
        for (int r = 0; r < kRows; ++r)
            if (row0 + r < kDim) record[row0 + r] = S[r];
    }
}

// ---- runs of tokens in chunks -------------------------------------------------------------------------------------------------
// Inside a chunk of 32 tokens, with S the state before it, G_i the sum of log g up to token i and e(i, j) = exp(G_i - G_j):
//
//     u_i = beta_i (v_i - exp(G_i) S^T k_i - sum over j < i of e(i, j) (k_j . k_i) u_j)        o_i = exp(G_i) S^T q_i + sum over j <= i of e(i, j) (k_j . q_i) u_j
//     S <- exp(G_last) S + sum over j of e(last, j) k_j u_j^T
//
// The u of a chunk solve a unit lower triangular system that does not depend on S; with T its inverse, U = T (beta v) - W S, W = T diag(beta exp(G)) K.
//
//   delta_chunk:   one block per (chunk, head), no chunk waiting for another: q, k and W in three bfloat16 pieces (chunk_mma.cuh), the weights
//                  e(i, j) (k_j . q_i), and U_0 = T (beta v).  T by forward substitution, a column to a lane.
//   delta_state:   one block per (sequence, head, 16 value columns) walks the chunks: W S and q S from the state in the accumulators' registers, U = U_0 - W S,
//                  then the read-outs and the state.
//
// The token walk is a chain of T steps of about 0.4 us; the chunks are a chain of T / 32 steps.  Nothing is rounded to 16 bits on the way.
constexpr bool kChunked = kDim % 16 == 0 && kDim <= 128;
constexpr int kTokens = 32, kTile = 16, kPitch = kDim + 8, kScorePitch = kTokens + 8, kWalkers = 512, kChunkThreads = 256;
constexpr int kKeySteps = kDim / 16 > 0 ? kDim / 16 : 1;
constexpr int kGroups = kKeySteps >= 8 ? 8 : kKeySteps >= 4 ? 4 : kKeySteps >= 2 ? 2 : 1;      // warps that share the key elements out
constexpr int kKeyBytes = chunk::kPieces * kTokens * kPitch * 2, kScoreBytes = chunk::kPieces * kTokens * kScorePitch * 2;
constexpr int kScalars = 2 * kTokens + 4;                                    // exp(G), e(last, .), exp(G_last)
constexpr int kBlockBytes = 3 * kKeyBytes + kScoreBytes + kScalars * 4;      // what delta_state reads of a (chunk, head), as it lies in shared memory: W, q, k, weights, scalars
constexpr int kLowerPitch = kTokens + 4, kValueColumns = 64, kValuePitch = kValueColumns + 8;           // of delta_chunk, at a time
constexpr int kPrepareBytes = kBlockBytes + kScoreBytes + chunk::kPieces * kTokens * kValuePitch * 2 + kTokens * 12;
constexpr int kSumBytes = 2 * kGroups * kTokens * kTile * 4;
constexpr int kStateBytes = 2 * kBlockBytes + kSumBytes + chunk::kPieces * (kTokens * 24 + kTile * kScorePitch) * 2 + 2 * kTokens * kTile * 4 + 32;

// grid (chunk numbers, heads); block kChunkThreads: two blocks of eight warps to an SM, which shared memory allows (with four warps each most of a block's time was
// the latency of its own chain: 2,048 tokens of 16 heads of 128 74 us, here 60; a delta layer 316 -> 301).
// Narrow keys leave shared memory for more blocks, and the registers follow (four runs of 300 tokens of 8 heads of 64 43.5 us with two blocks to an SM, 37 with three).
__global__ void __launch_bounds__(kChunkThreads, kDim <= 32 ? 4 : kDim <= 64 ? 3 : 2)
delta_chunk_kernel(const float* __restrict__ rows, long long stride, int q_offset, int k_offset, int v_offset, const float* __restrict__ gates,
                   const int* __restrict__ cu_seqlens, int n_seqs, unsigned char* __restrict__ blocks, float* __restrict__ first_updates, int heads, int key_heads, int value_dim,
                   int chunks_from) {
    if constexpr (kChunked) {
        grid_dependency_wait();
        extern __shared__ __align__(128) unsigned char shared[];
        bf16* Ws = reinterpret_cast<bf16*>(shared);                              // [piece][token][kPitch], as are q and k
        bf16* qs = Ws + kKeyBytes / 2;
        bf16* ks = qs + kKeyBytes / 2;
        bf16* ps = ks + kKeyBytes / 2;                                           // weights [piece][token][kScorePitch]
        float* scalars = reinterpret_cast<float*>(ps + kScoreBytes / 2);
        bf16* Ts = reinterpret_cast<bf16*>(shared + kBlockBytes);                // T with its columns weighted [piece][token][kScorePitch]
        bf16* vs = Ts + kScoreBytes / 2;                                         // values [piece][token][kValuePitch]
        float* lower = reinterpret_cast<float*>(vs);                             // beta_i e(i, j) (k_i . k_j) below the diagonal [token][kLowerPitch], before the values
        double* G = reinterpret_cast<double*>(vs + chunk::kPieces * kTokens * kValuePitch);
        float* betas = reinterpret_cast<float*>(G + kTokens);
        const int number = blockIdx.x, head = blockIdx.y, key_head = head / (heads / key_heads), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const chunk::Run run = chunk::find_run<true>(cu_seqlens, n_seqs, chunks_from, kTokens, number);
        if (run.sequence < 0) return;                                            // a number that no chunk has
        const int start = cu_seqlens[run.sequence] + (number - run.first) * kTokens, live = min(kTokens, cu_seqlens[run.sequence + 1] - start);
        // A key or gate that is no number must not reach the tokens before it, as weights of zero times it would: from such a token on keys are taken as
        // zero here, and exp(G) as NaN, which makes NaN of these tokens' results and of the state, as the walk does.
        int bad = kTokens;
        constexpr int kVectors = kDim / 4;
        // Loads are asked for eight at a time: one after the other they were a third of this kernel (a block alone took 29 us).
        constexpr int kLoads = kChunked ? 2 * kTokens * kVectors / kChunkThreads : 1, kBatch = kLoads % 8 == 0 ? 8 : kLoads % 4 == 0 ? 4 : kLoads % 2 == 0 ? 2 : 1;
        const bool whole = ((reinterpret_cast<uintptr_t>(rows) & 15) | (stride & 3) | (q_offset & 3) | (k_offset & 3)) == 0;      // 16 bytes at a time
#pragma unroll 1
        for (int done = 0; done < kLoads; done += kBatch) {
            float4 x[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int item = threadIdx.x + (done + i) * kChunkThreads, which = item / (kTokens * kVectors), token = item / kVectors % kTokens, column = item % kVectors * 4;
                const float* source = rows + static_cast<size_t>(start + min(token, live - 1)) * stride + (which ? k_offset : q_offset) + key_head * kDim + column;
                x[i] = whole ? *reinterpret_cast<const float4*>(source) : make_float4(source[0], source[1], source[2], source[3]);
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int item = threadIdx.x + (done + i) * kChunkThreads, which = item / (kTokens * kVectors), token = item / kVectors % kTokens, column = item % kVectors * 4;
                if (token >= live) x[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (which && !(fabsf(x[i].x) < INFINITY && fabsf(x[i].y) < INFINITY && fabsf(x[i].z) < INFINITY && fabsf(x[i].w) < INFINITY)) bad = min(bad, token);
                uint32_t low[chunk::kPieces], high[chunk::kPieces];
                chunk::split_pair(x[i].x, x[i].y, low);
                chunk::split_pair(x[i].z, x[i].w, high);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p)
                    *reinterpret_cast<uint2*>((which ? ks : qs) + (p * kTokens + token) * kPitch + column) = make_uint2(low[p], high[p]);
            }
        }
        if (warp == 0) {
            const float2 gate = *reinterpret_cast<const float2*>(gates + (static_cast<size_t>(start + min(lane, live - 1)) * heads + head) * 2);
            const bool odd = !(fabsf(gate.x) < INFINITY) || !(fabsf(gate.y) < INFINITY);
            if (odd && lane < live) bad = min(bad, lane);
            // A decay that vanished in 32 bits is below exp(-104); taken as that, a product with it vanishes again, and differences of sums stay finite.
            // Nothing says that a decay is positive: G is the logarithm of the products' sizes, and a bit a token says whether the product up to it is below zero.
            double sum = lane < live && !odd ? fmax(log(fabs(static_cast<double>(gate.x))), -104.0) : 0.0;
            const unsigned below_zero = __ballot_sync(0xffffffffu, lane < live && !odd && gate.x < 0.0f);
            const unsigned turned = __ballot_sync(0xffffffffu, __popc(below_zero & (0xffffffffu >> (31 - lane))) & 1);
            if (lane == 0) scalars[2 * kTokens + 1] = __uint_as_float(turned);
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const double before = __shfl_up_sync(0xffffffffu, sum, offset);
                if (lane >= offset) sum += before;
            }
            G[lane] = sum;
            betas[lane] = lane < live && !odd ? gate.y : 0.0f;
        }
        bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, 16)); bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, 8)); bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, 4));
        bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, 2)); bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, 1));
        if (threadIdx.x == 0) scalars[0] = __int_as_float(kTokens);
        __syncthreads();
        if (lane == 0 && bad < kTokens) atomicMin(reinterpret_cast<int*>(scalars), bad);
        __syncthreads();
        bad = __float_as_int(scalars[0]);
        __syncthreads();
        if (bad < kTokens)
            for (int item = threadIdx.x; item < chunk::kPieces * kTokens * kDim; item += kChunkThreads)
                if (item / kDim % kTokens >= bad) ks[item / kDim * kPitch + item % kDim] = __float2bfloat16_rn(0.0f);
        const unsigned turned = __float_as_uint(scalars[2 * kTokens + 1]);
        auto signed_by = [&](float size, unsigned bit) { return __uint_as_float(__float_as_uint(size) ^ (bit & 1u) << 31); };
        if (warp == 0) {
            const bool gone = lane >= bad;
            scalars[lane] = gone ? __int_as_float(0x7fffffff) : signed_by(expf(static_cast<float>(G[lane])), turned >> lane);
            scalars[kTokens + lane] = lane < live && !gone ? signed_by(expf(static_cast<float>(G[live - 1] - G[lane])), turned >> (live - 1) ^ turned >> lane) : 0.0f;
            if (lane == live - 1) scalars[2 * kTokens] = bad < live ? __int_as_float(0x7fffffff) : signed_by(expf(static_cast<float>(G[lane])), turned >> lane);
            if (gone) betas[lane] = 0.0f;
        }
        __syncthreads();
        // k k^T by the first four warps, q k^T by the others: 16 rows by 16 columns to a warp.
        const int strip = warp % 2, half = warp / 2 % 2, quarter = warp / 2;
        {
            const bool of_queries = warp >= 4;
            float sums[2][4] = {};      // [columns 0-7 or 8-15]
#pragma unroll 1
            for (int from = 0; from < kKeySteps; from += 2) {
                float large[2][4] = {}, small[2][4] = {};
#pragma unroll
                for (int ahead = 0; ahead < 2; ++ahead) {
                    const int step = from + ahead;
                    if (step >= kKeySteps) break;
                    uint32_t b[chunk::kPieces][4];
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p)
                        chunk::load_matrices(b[p], ks + (p * kTokens + half * 16 + lane % 8 + lane / 16 * 8) * kPitch + step * 16 + lane / 8 % 2 * 8);
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p) {
                        uint32_t a[4];
                        chunk::load_matrices(a, (of_queries ? qs : ks) + (p * kTokens + strip * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
#pragma unroll
                        for (int other = 0; other + p < chunk::kPieces; ++other) {
                            chunk::multiply(p + other ? small[0] : large[0], a, b[other][0], b[other][1]);
                            chunk::multiply(p + other ? small[1] : large[1], a, b[other][2], b[other][3]);
                        }
                    }
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sums[n][e] += large[n][e] + small[n][e];
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int down = 0; down < 2; ++down) {
                    const int i = strip * 16 + lane / 4 + down * 8, j = half * 16 + n * 8 + lane % 4 * 2;
                    float weights[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float kept = j + e <= i ? signed_by(expf(static_cast<float>(G[i] - G[j + e])), turned >> i ^ turned >> (j + e)) : 0.0f;
                        if (!of_queries) lower[i * kLowerPitch + j + e] = j + e < i ? betas[i] * (kept * sums[n][down * 2 + e]) : 0.0f;
                        weights[e] = j + e <= i && i < live ? kept * sums[n][down * 2 + e] : 0.0f;
                    }
                    if (!of_queries) continue;
                    uint32_t pieces[chunk::kPieces];
                    chunk::split_pair(weights[0], weights[1], pieces);
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p) *reinterpret_cast<uint32_t*>(ps + (p * kTokens + i) * kScorePitch + j) = pieces[p];
                }
        }
        __syncthreads();
        // The values' columns are on their way while the first warp solves for T, and the next while these are multiplied.
        constexpr int kValueLoads = kTokens * kValueColumns / 2 / kChunkThreads;
        float2 x[kValueLoads];
        auto fetch = [&](int base) {
#pragma unroll
            for (int i = 0; i < kValueLoads; ++i) {
                const int item = threadIdx.x + i * kChunkThreads, token = item / (kValueColumns / 2), at = item % (kValueColumns / 2) * 2;
                const float* source = rows + static_cast<size_t>(start + min(token, live - 1)) * stride + v_offset + head * value_dim + base + at;
                x[i].x = token < live && base + at < value_dim ? source[0] : 0.0f;
                x[i].y = token < live && base + at + 1 < value_dim ? source[1] : 0.0f;
            }
        };
        fetch(0);
        float column[kTokens];      // T's column `lane`, in the first warp
        auto lay_out = [&](float factor) {
#pragma unroll
            for (int i = 0; i < kTokens; ++i) {
                bf16 pieces[chunk::kPieces];
                chunk::split_one(i >= lane ? column[i] * factor : 0.0f, pieces);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) Ts[(p * kTokens + i) * kScorePitch + lane] = pieces[p];
            }
        };
        if (warp == 0) {
#pragma unroll
            for (int i = 0; i < kTokens; ++i) {
                float sums[4] = {i == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int j = 0; j < i; j += 4) {
                    const float4 row = *reinterpret_cast<const float4*>(lower + i * kLowerPitch + j);
                    sums[0] = fmaf(-row.x, column[j], sums[0]);
                    if (j + 1 < i) sums[1] = fmaf(-row.y, column[j + 1], sums[1]);
                    if (j + 2 < i) sums[2] = fmaf(-row.z, column[j + 2], sums[2]);
                    if (j + 3 < i) sums[3] = fmaf(-row.w, column[j + 3], sums[3]);
                }
                column[i] = (sums[0] + sums[1]) + (sums[2] + sums[3]);
            }
            lay_out(lane < bad ? betas[lane] * scalars[lane] : 0.0f);
        }
        __syncthreads();
        // W: 16 rows by a quarter of the key elements to a warp.
#pragma unroll 1
        for (int step = quarter; step < kKeySteps; step += 4) {
            float large[2][4] = {}, small[2][4] = {};
#pragma unroll
            for (int deep = 0; deep < 2; ++deep) {
                uint32_t b[chunk::kPieces][4];
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) chunk::load_matrices_turned(b[p], ks + (p * kTokens + deep * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) {
                    uint32_t a[4];
                    chunk::load_matrices(a, Ts + (p * kTokens + strip * 16 + lane % 16) * kScorePitch + deep * 16 + lane / 16 * 8);
#pragma unroll
                    for (int other = 0; other + p < chunk::kPieces; ++other) {
                        chunk::multiply(p + other ? small[0] : large[0], a, b[other][0], b[other][1]);
                        chunk::multiply(p + other ? small[1] : large[1], a, b[other][2], b[other][3]);
                    }
                }
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int down = 0; down < 2; ++down) {
                    uint32_t pieces[chunk::kPieces];
                    chunk::split_pair(large[n][down * 2] + small[n][down * 2], large[n][down * 2 + 1] + small[n][down * 2 + 1], pieces);
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p)
                        *reinterpret_cast<uint32_t*>(Ws + (p * kTokens + strip * 16 + lane / 4 + down * 8) * kPitch + step * 16 + n * 8 + lane % 4 * 2) = pieces[p];
                }
        }
        chunk::shared_writes_ready();
        __syncthreads();
        if (threadIdx.x == 0) chunk::bulk_store(blocks + (static_cast<size_t>(number) * heads + head) * kBlockBytes, shared, kBlockBytes);
        if (warp == 0) lay_out(betas[lane]);
        // U_0, 64 value columns at a time.
        for (int base = 0; base < value_dim; base += kValueColumns) {
            bool odd = false;
#pragma unroll
            for (int i = 0; i < kValueLoads; ++i) {
                const int item = threadIdx.x + i * kChunkThreads, token = item / (kValueColumns / 2), at = item % (kValueColumns / 2) * 2;
                odd |= !(fabsf(x[i].x) < INFINITY) || !(fabsf(x[i].y) < INFINITY);
                uint32_t pieces[chunk::kPieces];
                chunk::split_pair(x[i].x, x[i].y, pieces);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) *reinterpret_cast<uint32_t*>(vs + (p * kTokens + token) * kValuePitch + at) = pieces[p];
            }
            if (base + kValueColumns < value_dim) fetch(base + kValueColumns);
            odd = __syncthreads_or(odd);
            {
                const int column0 = quarter * 16;
                float large[2][4] = {}, small[2][4] = {};
#pragma unroll
                for (int deep = 0; deep < 2; ++deep) {
                    uint32_t b[chunk::kPieces][4];
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p) chunk::load_matrices_turned(b[p], vs + (p * kTokens + deep * 16 + lane % 16) * kValuePitch + column0 + lane / 16 * 8);
#pragma unroll
                    for (int p = 0; p < chunk::kPieces; ++p) {
                        uint32_t a[4];
                        chunk::load_matrices(a, Ts + (p * kTokens + strip * 16 + lane % 16) * kScorePitch + deep * 16 + lane / 16 * 8);
#pragma unroll
                        for (int other = 0; other + p < chunk::kPieces; ++other) {
                            chunk::multiply(p + other ? small[0] : large[0], a, b[other][0], b[other][1]);
                            chunk::multiply(p + other ? small[1] : large[1], a, b[other][2], b[other][3]);
                        }
                    }
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = strip * 16 + lane / 4 + e / 2 * 8, at = column0 + n * 8 + lane % 4 * 2 + e % 2;
                        float update = large[n][e] + small[n][e];
                        if (odd) {      // an infinity or NaN reaches the tokens from its own on
                            update = 0.0f;
                            for (int j = 0; j <= i; ++j) {
                                float weight = 0.0f, value = __bfloat162float(vs[j * kValuePitch + at]);
                                for (int p = chunk::kPieces - 1; p >= 0; --p) weight += __bfloat162float(Ts[(p * kTokens + i) * kScorePitch + j]);
                                for (int p = 1; p < chunk::kPieces; ++p)
                                    if (fabsf(value) < INFINITY) value += __bfloat162float(vs[(p * kTokens + j) * kValuePitch + at]);
                                update = fmaf(weight, value, update);
                            }
                        }
                        if (i < live && base + at < value_dim) first_updates[(static_cast<size_t>(start + i) * heads + head) * value_dim + base + at] = update;
                    }
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) chunk::bulk_stored();      // no early start of the next kernel: see the launch
    }
}

// grid (heads, runs, tiles of 16 value columns); block kWalkers.  A group of key elements belongs to a warp as S^T tiles of 16 columns by 16 elements
// in the accumulators' layout, in which they are the right operand of W S and q S; the warps of a group keep the same state and share W, q and their
// tokens out.  Two barriers a chunk: behind the first the groups' sums become U, behind the second U becomes read-outs and state.
// One block to an SM, which its shared memory says anyway: told so, the compiler takes 112 registers and not 64 with a spill (both kernels over 2,048 tokens
// of 16 heads: 202 against 214 us).
__global__ void __launch_bounds__(kWalkers, 1)
delta_state_kernel(const unsigned char* __restrict__ blocks, const float* __restrict__ first_updates, float* __restrict__ state, long long slot_stride,
                   const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, float* __restrict__ out, int heads, int value_dim, int n_seqs,
                   int chunks_from) {
    if constexpr (kChunked) {
        constexpr int kStrips = kTokens / 16, kParts = kWalkers / 32 / kGroups, kMyStrips = kParts >= 4 ? 1 : 2, kMine = (kKeySteps + kGroups - 1) / kGroups;
        grid_dependency_wait();
        extern __shared__ __align__(128) unsigned char shared[];
        float* partial = reinterpret_cast<float*>(shared + 2 * kBlockBytes);     // [W or q][group][token][kTile]
        bf16* us = reinterpret_cast<bf16*>(partial + kSumBytes / 4);             // U [piece][token][24]
        bf16* ws = us + chunk::kPieces * kTokens * 24;                           // e(last, .) U, turned [piece][column][kScorePitch]
        float* updates = reinterpret_cast<float*>(ws + chunk::kPieces * kTile * kScorePitch);      // U_0 of even and odd chunks [token][kTile]
        uint64_t* barriers = reinterpret_cast<uint64_t*>(updates + 2 * kTokens * kTile);
        const int head = blockIdx.x, column0 = blockIdx.z * kTile, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const chunk::Run run = chunk::find_run<false>(cu_seqlens, n_seqs, chunks_from, kTokens, blockIdx.y);
        if (run.sequence < 0) return;
        const int sequence = run.sequence, first = run.first;
        const int group = warp % kGroups, part = warp / kGroups, which = part % 2, strip0 = part / 2 * kMyStrips;
        const int begin = cu_seqlens[sequence], end = cu_seqlens[sequence + 1];
        float* record = state + static_cast<size_t>(seq_slot[sequence]) * slot_stride + static_cast<size_t>(head) * value_dim * kDim;
        float S[kMine][2][4];
#pragma unroll
        for (int mine = 0; mine < kMine; ++mine)
#pragma unroll
            for (int side = 0; side < 2; ++side)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int column = column0 + lane / 4 + e / 2 * 8, element = (group + mine * kGroups) * 16 + side * 8 + lane % 4 * 2 + e % 2;
                    S[mine][side][e] = column < value_dim && element < kDim ? record[static_cast<size_t>(column) * kDim + element] : 0.0f;
                }
        const int chunks = (end - begin + kTokens - 1) / kTokens;
        volatile int* gone = reinterpret_cast<volatile int*>(barriers + 2);      // see barrier_wait; then the chunks asked for
        auto ask = [&](int chunk_index) {
            if (gone[0]) return;
            gone[1] = chunk_index + 1;
            uint64_t* barrier = barriers + (chunk_index & 1);
            chunk::barrier_expect(barrier, kBlockBytes);
            chunk::bulk_copy(shared + (chunk_index & 1) * kBlockBytes, blocks + (static_cast<size_t>(first + chunk_index) * heads + head) * kBlockBytes, kBlockBytes, barrier);
        };
        // U_0: a thread's token and column.
        const int my_token = threadIdx.x / kTile, my_column = column0 + threadIdx.x % kTile;
        auto fetch = [&](int chunk_index) {
            const int at = begin + chunk_index * kTokens + my_token;
            return at < end && my_column < value_dim ? first_updates[(static_cast<size_t>(at) * heads + head) * value_dim + my_column] : 0.0f;
        };
        if (threadIdx.x < 2) {
            chunk::barrier_init(barriers + threadIdx.x);
            gone[threadIdx.x] = 0;
        }
        chunk::barriers_ready();
        __syncthreads();
        if (threadIdx.x == 0) ask(0);
        float next_update = fetch(0);
        for (int chunk_index = 0; chunk_index < chunks; ++chunk_index) {
            const unsigned char* block = shared + (chunk_index & 1) * kBlockBytes;
            const bf16* rows = reinterpret_cast<const bf16*>(block) + which * (kKeyBytes / 2);      // W or q
            const bf16* ks = reinterpret_cast<const bf16*>(block) + kKeyBytes;
            const bf16* ps = ks + kKeyBytes / 2;
            const float* scalars = reinterpret_cast<const float*>(ps + kScoreBytes / 2);
            float* update = updates + (chunk_index & 1) * kTokens * kTile;
            update[threadIdx.x] = next_update;
            chunk::barrier_wait(barriers + (chunk_index & 1), chunk_index / 2 & 1, gone);
            if (strip0 < kStrips) {
                float sums[kMyStrips][2][4] = {};
#pragma unroll
                for (int mine = 0; mine < kMine; ++mine) {
                    const int step = group + mine * kGroups;
                    if (step < kKeySteps) {
                        uint32_t pieces[2][2][chunk::kPieces];      // [columns 0-7 or 8-15][key elements 0-7 or 8-15]
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            chunk::split_pair(S[mine][side][0], S[mine][side][1], pieces[0][side]);
                            chunk::split_pair(S[mine][side][2], S[mine][side][3], pieces[1][side]);
                        }
#pragma unroll
                        for (int p = chunk::kPieces - 1; p >= 0; --p) {      // the small products first
                            uint32_t a[kMyStrips][4];
#pragma unroll
                            for (int strip = 0; strip < kMyStrips; ++strip)
                                chunk::load_matrices(a[strip], rows + (p * kTokens + (strip0 + strip) * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
#pragma unroll
                            for (int other = chunk::kPieces - 1 - p; other >= 0; --other)
#pragma unroll
                                for (int strip = 0; strip < kMyStrips; ++strip)
#pragma unroll
                                    for (int n = 0; n < 2; ++n) chunk::multiply(sums[strip][n], a[strip], pieces[n][0][other], pieces[n][1][other]);
                        }
                    }
                }
#pragma unroll
                for (int strip = 0; strip < kMyStrips; ++strip)
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int down = 0; down < 2; ++down)      // columns 8-15 first in every other pair of rows, so that four rows meet all banks
                            *reinterpret_cast<float2*>(partial + ((which * kGroups + group) * kTokens + (strip0 + strip) * 16 + lane / 4 + down * 8) * kTile + (n ^ lane / 8 % 2) * 8 + lane % 4 * 2) =
                                make_float2(sums[strip][n][down * 2], sums[strip][n][down * 2 + 1]);
            }
            __syncthreads();      // the groups' sums are there; the other half's block was last read before this barrier
            if (chunk_index + 1 < chunks) {
                if (threadIdx.x == 0) ask(chunk_index + 1);
                next_update = fetch(chunk_index + 1);
            }
            // 16 tokens by 8 columns to a warp: U by the first four warps, what the state gives the read-outs by the next four.
            const int strip = warp / 2 % 2, n = warp % 2, row = strip * 16 + lane / 4, local = n * 8 + lane % 4 * 2;
            float inside[4];
            bool odd = false;
            if (warp < 8) {
#pragma unroll
                for (int down = 0; down < 2; ++down) {
                    float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int from = 0; from < kGroups; ++from) {
                        const float2 part_sum = *reinterpret_cast<const float2*>(partial + ((warp / 4 * kGroups + from) * kTokens + row + down * 8) * kTile + (n ^ lane / 8 % 2) * 8 + lane % 4 * 2);
                        sum.x += part_sum.x;
                        sum.y += part_sum.y;
                    }
                    if (warp < 4) {
                        const float2 own = *reinterpret_cast<const float2*>(update + (row + down * 8) * kTile + local);
                        const float x = own.x - sum.x, y = own.y - sum.y, left = scalars[kTokens + row + down * 8];
                        odd |= !(fabsf(x) < INFINITY) || !(fabsf(y) < INFINITY);
                        uint32_t pieces[chunk::kPieces];
                        chunk::split_pair(x, y, pieces);
                        bf16 first_pieces[chunk::kPieces], second_pieces[chunk::kPieces];
                        chunk::split_one(x * left, first_pieces);
                        chunk::split_one(y * left, second_pieces);
#pragma unroll
                        for (int p = 0; p < chunk::kPieces; ++p) {
                            *reinterpret_cast<uint32_t*>(us + (p * kTokens + row + down * 8) * 24 + local) = pieces[p];
                            ws[(p * kTile + local) * kScorePitch + row + down * 8] = first_pieces[p];
                            ws[(p * kTile + local + 1) * kScorePitch + row + down * 8] = second_pieces[p];
                        }
                    } else {
                        inside[down * 2] = scalars[row + down * 8] * sum.x;
                        inside[down * 2 + 1] = scalars[row + down * 8] * sum.y;
                    }
                }
            }
            odd = __syncthreads_or(odd || gone[0] != 0);      // U is there
            if (odd && __syncthreads_or(gone[0] != 0)) {      // ... or a wait ran out: the state stays as it was, and the block ends when its copies have
                const int asked = gone[1];
                if (asked > 1) chunk::barrier_wait(barriers + (asked & 1), (asked - 2) / 2 & 1, nullptr);
                chunk::barrier_wait(barriers + ((asked - 1) & 1), (asked - 1) / 2 & 1, nullptr);
                return;
            }
            if (warp >= 4 && warp < 8) {
                if (!odd) {
                    float large[4] = {}, small[4] = {};
#pragma unroll
                    for (int step = 0; step < kStrips; ++step) {
                        if (step > strip) break;
                        uint32_t b[chunk::kPieces][2];
#pragma unroll
                        for (int p = 0; p < chunk::kPieces; ++p) chunk::load_pair_turned(b[p], us + (p * kTokens + step * 16 + lane % 16) * 24 + n * 8);
#pragma unroll
                        for (int p = 0; p < chunk::kPieces; ++p) {
                            uint32_t a[4];
                            chunk::load_matrices(a, ps + (p * kTokens + strip * 16 + lane % 16) * kScorePitch + step * 16 + lane / 16 * 8);
#pragma unroll
                            for (int other = 0; other + p < chunk::kPieces; ++other) chunk::multiply(p + other == 0 ? large : small, a, b[other][0], b[other][1]);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) inside[e] += large[e] + small[e];
                } else {      // an infinity or NaN must not reach the tokens before it
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = row + e / 2 * 8;
                        for (int j = 0; j <= i; ++j) {
                            float weight = 0.0f, value = __bfloat162float(us[j * 24 + local + e % 2]);
                            for (int p = chunk::kPieces - 1; p >= 0; --p) weight += __bfloat162float(ps[(p * kTokens + i) * kScorePitch + j]);
                            for (int p = 1; p < chunk::kPieces; ++p)
                                if (fabsf(value) < INFINITY) value += __bfloat162float(us[(p * kTokens + j) * 24 + local + e % 2]);
                            inside[e] = fmaf(weight, value, inside[e]);
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int token = begin + chunk_index * kTokens + row + e / 2 * 8, column = column0 + local + e % 2;
                    if (token < end && column < value_dim) out[(static_cast<size_t>(token) * heads + head) * value_dim + column] = inside[e];
                }
            }
            const float keep = scalars[2 * kTokens];
            float large[kMine][2][4] = {}, small[kMine][2][2][4] = {};
#pragma unroll
            for (int deep = 0; deep < kStrips; ++deep) {
                uint32_t a[chunk::kPieces][4];
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) chunk::load_matrices(a[p], ws + (p * kTile + lane % 16) * kScorePitch + deep * 16 + lane / 16 * 8);
#pragma unroll
                for (int mine = 0; mine < kMine; ++mine) {
                    const int step = group + mine * kGroups;
                    if (step < kKeySteps) {
#pragma unroll
                        for (int p = 0; p < chunk::kPieces; ++p) {
                            uint32_t b[4];
                            chunk::load_matrices_turned(b, ks + (p * kTokens + deep * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
#pragma unroll
                            for (int other = 0; other + p < chunk::kPieces; ++other)
#pragma unroll
                                for (int side = 0; side < 2; ++side)
                                    chunk::multiply(p + other == 0 ? large[mine][side] : small[mine][side][(p + other) % 2], a[other], b[side * 2], b[side * 2 + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int mine = 0; mine < kMine; ++mine)
#pragma unroll
                for (int side = 0; side < 2; ++side)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[mine][side][e] = fmaf(keep, S[mine][side][e], large[mine][side][e] + (small[mine][side][0][e] + small[mine][side][1][e]));
        }
        if (part == 0) {
#pragma unroll
            for (int mine = 0; mine < kMine; ++mine)
#pragma unroll
                for (int side = 0; side < 2; ++side)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int column = column0 + lane / 4 + e / 2 * 8, element = (group + mine * kGroups) * 16 + side * 8 + lane % 4 * 2 + e % 2;
                        if (column < value_dim && element < kDim) record[static_cast<size_t>(column) * kDim + element] = S[mine][side][e];
                    }
        }
    }
}

}  // namespace

TAU_EXPORT int tau_delta_key_dim() { return kDim; }

// 1 if a bounded wait ran out since the library was loaded (synchronises the device).
TAU_EXPORT int tau_delta_status() { return chunk::wait_status(); }

// Bytes of workspace with which `tau_delta_rule` walks runs of `chunks` tokens and more in chunks (one decay per head); 0: these key widths are not walked in chunks.
TAU_EXPORT long long tau_delta_workspace(int tokens, int n_seqs, int heads, int value_dim, int chunks) {
    if (!kChunked || tokens <= 0 || n_seqs <= 0 || heads <= 0 || value_dim <= 0 || chunks <= 0) return 0;
    return static_cast<long long>(chunk::most_chunks(tokens, n_seqs, chunks, kTokens)) * heads * kBlockBytes + static_cast<long long>(tokens) * heads * value_dim * 4;
}

TAU_EXPORT int tau_delta_prepare(float* rows, long long stride, int q_offset, int k_offset, const float* pre, int pre_stride, const float* a_log,
                                 const float* dt_bias, float* gates, float* kq, float* channel, int tokens, int heads, int key_heads, float query_scale,
                                 void* stream) {
    if (tokens <= 0) return 0;
    if (!rows || !pre || !a_log || !dt_bias || !gates || !kq || heads <= 0 || key_heads <= 0 || heads % key_heads != 0 || pre_stride < (channel ? heads : 2 * heads))
        return cudaErrorInvalidValue;
    tau_launch(delta_prepare_kernel, dim3(tokens), dim3(128), 0, static_cast<cudaStream_t>(stream), rows, stride, q_offset, k_offset, pre, pre_stride, a_log,
               dt_bias, gates, kq, channel, heads, key_heads, query_scale);
    return tau_launch_status();
}

// rows [tokens, stride] float with q, k (key_heads * key_dim each) and v (heads * value_dim) at their offsets, prepared as above.
// state: [heads, value_dim, key_dim] floats per slot, slots `slot_stride` apart.  out [tokens, heads * value_dim].
// `channel` (or null): [tokens, heads * key_dim], a decay per head and key channel as `tau_delta_prepare` left it.
// `workspace` (or null; 16-byte aligned, `tau_delta_workspace` bytes): runs of `chunks` tokens and more go in chunks, without `channel`, and with `shorter`
// the others token by token (without it there are none).
TAU_EXPORT int tau_delta_rule(const float* rows, long long stride, int q_offset, int k_offset, int v_offset, const float* gates, const float* kq,
                              const float* channel, float* state, long long slot_stride, const int* cu_seqlens, const int* seq_slot, float* out, int n_seqs, int heads,
                              int key_heads, int value_dim, int tokens, int chunks, int shorter, void* workspace, long long workspace_bytes, void* stream) {
    if (n_seqs <= 0) return 0;
    if (!rows || !gates || !kq || !state || !cu_seqlens || !seq_slot || !out || heads <= 0 || key_heads <= 0 || heads % key_heads != 0 || value_dim <= 0)
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (workspace) {
        if (channel || !kChunked || chunks <= 0 || (reinterpret_cast<uintptr_t>(workspace) & 15) != 0 || (reinterpret_cast<uintptr_t>(gates) & 7) != 0
            || workspace_bytes < tau_delta_workspace(tokens, n_seqs, heads, value_dim, chunks) || tau_delta_workspace(tokens, n_seqs, heads, value_dim, chunks) == 0)
            return cudaErrorInvalidValue;
        if (cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrepareBytes) != cudaSuccess
            || cudaFuncSetAttribute(delta_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStateBytes) != cudaSuccess)
            return cudaErrorInvalidValue;
        const int numbers = chunk::most_chunks(tokens, n_seqs, chunks, kTokens), runs = chunk::most_runs(tokens, n_seqs, chunks);
        unsigned char* blocks = static_cast<unsigned char*>(workspace);
        float* first_updates = reinterpret_cast<float*>(blocks + static_cast<size_t>(numbers) * heads * kBlockBytes);
        // Each starts when the kernel before it has finished, and lets the next start when it is done itself: with blocks of their neighbours resident beside
        // them (programmatic launch) one pass in some hundreds did not end, for a cause that is not known; 12,000 passes without that did.  It costs about 3 us
        // of 200.  Kernels that move tiles through the bulk copies of chunk_mma.cuh are all launched so; it orders the kernels of one stream, no more.
        if (runs > 0) {
            tau_launch_as(false, delta_chunk_kernel, dim3(numbers, heads), dim3(kChunkThreads), kPrepareBytes, s, rows, stride, q_offset, k_offset, v_offset, gates, cu_seqlens, n_seqs, blocks,
                       first_updates, heads, key_heads, value_dim, chunks);
            tau_launch_as(false, delta_state_kernel, dim3(heads, runs, (value_dim + kTile - 1) / kTile), dim3(kWalkers), kStateBytes, s, static_cast<const unsigned char*>(blocks),
                       static_cast<const float*>(first_updates), state, slot_stride, cu_seqlens, seq_slot, out, heads, value_dim, n_seqs, chunks);
        }
        const int status = tau_launch_status();
        if (status != 0 || !shorter) return status;
    }
    const int below = workspace ? chunks : 0x7fffffff;
    const bool narrow = heads * n_seqs * ((value_dim + 31) / 32) < 148 && kSplit <= 16;     // blocks of 16 columns reach more SMs
    const int tile = narrow ? 16 : 32;
    dim3 grid(heads, n_seqs, (value_dim + tile - 1) / tile), block(tile * kSplit);
    // A walk over runs of tokens starts when the kernel before it has finished: started earlier, its few long blocks pile up on the SMs that fall free first
    // (2,048 tokens, 16 heads of 128 x 128 behind the kernels of a layer: 2.4 to 5.8 ms a layer that way, 1.1 ms so).
    const bool dependent = workspace || tokens <= 4 * n_seqs;
#define TAU_DELTA(COLUMNS, CHANNEL)                                                                                                               \
    tau_launch_as(dependent, delta_rule_kernel<COLUMNS, CHANNEL>, grid, block, 0, s, rows, stride, q_offset, k_offset, v_offset, gates, kq, channel, state, slot_stride, \
               cu_seqlens, seq_slot, out, heads, key_heads, value_dim, below)
    if (narrow) {
        if (channel) TAU_DELTA(16, true); else TAU_DELTA(16, false);
    } else {
        if (channel) TAU_DELTA(32, true); else TAU_DELTA(32, false);
    }
#undef TAU_DELTA
    return tau_launch_status();
}
