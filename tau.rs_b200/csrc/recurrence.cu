// Linear recurrences with a matrix state per head, for runs of new tokens and for single tokens alike:
//
//     S_t = a_t S_(t-1) + b_t k_t v_t^T          o_t = S_t^T q_t            (S is key_dim x value_dim)
//
// Two gatings.  Decay: a_t is a constant of the head, b_t = 1 (linear attention with a decay per head).
// Exponential: a log input gate i_t and a log forget gate f_t per head and token, both from soft-capped
// pre-activations (i = cap tanh(x / cap), f = logsigmoid(cap tanh(y / cap))), a running maximum
// m_t = max(f_t + m_(t-1), i_t) that starts at 0, a_t = exp(f_t + m_(t-1) - m_t), b_t = exp(i_t - m_t), a normaliser
// n_t = a_t n_(t-1) + b_t k_t, and o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6).
//
// The state is 32-bit and lives in the cache, one record per (slot, head): value_dim (+1) columns of key_dim
// numbers each, the extra column being n (which obeys the recurrence of a value that is always 1), then m.
// One block owns a (sequence, head, tile of columns) and walks the sequence's new tokens in order; a thread keeps
// its share of one column in registers, so a token costs one pass over key_dim per thread and two barriers.
// Everything is computed in 32-bit; q, k, v arrive in the activations' dtype.  TAU_KEY_DIM fixes key_dim.
//
// Runs of bfloat16 tokens take the same recurrence in chunks of tokens on the tensor cores.  Inside a chunk, with w(i, j) what is left at
// token i of the write of token j (a product of gates, at most 1 with the running maximum) and g(i) what is left of the state S before the chunk:
//
//     o_i = g(i) S^T q_i + sum over j <= i of w(i, j) (q_i . k_j) v_j          S <- g(last) S + sum over j of w(last, j) k_j v_j^T
//
//   gate_scan:     running maximum and log forget sums of every (sequence, head), 32 pieces of the run at once.
//   chunk_scores:  one block per (chunk, head): the scores w(i, j) (q_i . k_j), which no chunk waits for another for.
//   chunk_state:   one block per (sequence, head, 16 columns of the state) walks the chunks; the state stays in the accumulators' registers.
//
// The token walk is a chain of T steps of about 1 us; the chunks are a chain of T / 64 (or T / 32) steps.  q, k and v are exact in bfloat16 (or are
// split into three pieces behind an activation); scores, state and weighted values are 32-bit numbers in three pieces (chunk_mma.cuh), so that
// nothing is rounded to 16 bits on the way.
#include "chunk_mma.cuh"

#ifndef TAU_KEY_DIM
#error "compile with -DTAU_KEY_DIM=<key elements per head>"
#endif

namespace {

constexpr int kDim = TAU_KEY_DIM;
constexpr int kSplit = kDim <= 16 ? 1 : kDim <= 32 ? 2 : kDim <= 64 ? 4 : kDim <= 128 ? 8 : kDim <= 256 ? 16 : 32;   // threads that share a column
constexpr int kRows = (kDim + kSplit - 1) / kSplit;                               // key rows per thread
// Columns of a block (n included): 32, or 16 where 32 would leave SMs without a block.

__device__ __forceinline__ float activate(float value, int activation) { return activation ? value / (1.0f + expf(-value)) : value; }

// The gates' pre-activations become log gates in place, for all tokens at once: what does not depend on the token before
// is not computed inside the walk.  gates [tokens, 2 heads]: inputs first, then forgets.  `start` [sequences, heads, kDim + 1] receives n and m as
// they are before the run: every block of a (sequence, head) reads them and one writes them, which may be done before another begins.
__global__ void log_gates_kernel(float* __restrict__ gates, long long count, int heads, float gate_cap, const float* __restrict__ state, long long slot_stride,
                                 const int* __restrict__ seq_slot, int n_seqs, int value_dim, float* __restrict__ start) {
    grid_dependents_launch();
    grid_dependency_wait();
    for (long long index = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; index < count; index += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float capped = gate_cap * tanhf(gates[index] / gate_cap);
        const bool forget = (index / heads) & 1;
        gates[index] = forget ? fminf(capped, 0.0f) - log1pf(expf(-fabsf(capped))) : capped;     // logsigmoid for the forget gate
    }
    const long long kept = static_cast<long long>(n_seqs) * heads * (kDim + 1);
    for (long long index = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; index < kept; index += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long pair = index / (kDim + 1);
        const size_t record = (static_cast<size_t>(value_dim) + 1) * kDim + 1;
        start[index] = state[static_cast<size_t>(seq_slot[pair / heads]) * slot_stride + static_cast<size_t>(pair % heads) * record + static_cast<size_t>(value_dim) * kDim + index % (kDim + 1)];
    }
}

long long start_floats(int n_seqs, int heads) { return static_cast<long long>(n_seqs) * heads * (kDim + 1); }

template <typename T, int kColumns>
__global__ void __launch_bounds__(kColumns * kSplit)
linear_recurrence_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long stride,
                         const float* __restrict__ gates, const float* __restrict__ decays, const float* __restrict__ start, float* __restrict__ state, long long slot_stride,
                         const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, float* __restrict__ out,
                         int heads, int value_dim, int exponential, float gate_cap, float query_scale, int activation, int below) {
    grid_dependents_launch();
    grid_dependency_wait();
    __shared__ float qs[2][kDim], ks[2][kDim], partial[2][kSplit][kColumns];
    const int head = blockIdx.x, sequence = blockIdx.y;
    const int columns = value_dim + (exponential ? 1 : 0);           // n rides as one more column of the state
    // A block serves a tile of value columns; with the exponential gating its last thread column serves n as well, in every
    // block (each needs n . q), and the first block alone writes n and m back.
    const int tile = exponential ? kColumns - 1 : kColumns;
    const int local = threadIdx.x % kColumns;
    const bool is_n = exponential && local == kColumns - 1;
    const int column = is_n ? value_dim : blockIdx.z * tile + local;
    const int part = threadIdx.x / kColumns, row0 = part * kRows;
    const bool live = is_n || column < value_dim;
    float* record = state + static_cast<size_t>(seq_slot[sequence]) * slot_stride + static_cast<size_t>(head) * (static_cast<size_t>(columns) * kDim + (exponential ? 1 : 0));
    const float* start_n = exponential ? start + (static_cast<size_t>(sequence) * heads + head) * (kDim + 1) : nullptr;
    float S[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) S[r] = (live && row0 + r < kDim) ? (is_n ? start_n : record + static_cast<size_t>(column) * kDim)[row0 + r] : 0.0f;
    float m = exponential ? start_n[kDim] : 0.0f;
    const float decay = exponential ? 1.0f : decays[head];
    const int begin = cu_seqlens[sequence], end = cu_seqlens[sequence + 1];
    if (end - begin >= below) return;      // the chunk kernels' run
    // Operands are asked for four tokens ahead, in four sets of registers that take turns: a token's q and k go into the free
    // half of qs/ks one token before they are used, its v and gates stay in their set until its turn, and the set is filled
    // again for the token four further on.  The walk then waits for memory at its start only.
    constexpr int kStage = (kDim + kColumns * kSplit - 1) / (kColumns * kSplit);
    constexpr int kAhead = 4;
    float next_q[kAhead][kStage], next_k[kAhead][kStage], next_v[kAhead], next_in[kAhead], next_forget[kAhead];
    auto fetch = [&](int set, int token) {
        if (token >= end) return;
        const size_t row = static_cast<size_t>(token) * stride;
#pragma unroll
        for (int i = 0; i < kStage; ++i) {
            const int d = threadIdx.x + i * kColumns * kSplit;
            if (d < kDim) {
                next_q[set][i] = to_float(q[row + head * kDim + d]);
                next_k[set][i] = to_float(k[row + head * kDim + d]);
            }
        }
        if (live && !is_n) next_v[set] = to_float(v[row + head * value_dim + column]);
        if (exponential) {
            next_in[set] = gates[static_cast<size_t>(token) * 2 * heads + head];
            next_forget[set] = gates[static_cast<size_t>(token) * 2 * heads + heads + head];
        }
    };
    auto publish = [&](int set, int half) {
#pragma unroll
        for (int i = 0; i < kStage; ++i) {
            const int d = threadIdx.x + i * kColumns * kSplit;
            if (d < kDim) {
                qs[half][d] = activate(next_q[set][i], activation) * query_scale;
                ks[half][d] = activate(next_k[set][i], activation);
            }
        }
    };
#pragma unroll
    for (int set = 0; set < kAhead; ++set) {
        next_v[set] = next_in[set] = next_forget[set] = 0.0f;
        fetch(set, begin + set);
    }
    if (begin < end) publish(0, 0);
    __syncthreads();
    for (int base = begin; base < end; base += kAhead) {
#pragma unroll
      for (int set = 0; set < kAhead; ++set) {
        const int token = base + set;
        if (token >= end) break;
        const int half = set & 1;                  // kAhead is even: the halves take turns with the tokens
        const float raw_value = next_v[set], raw_in = next_in[set], raw_forget = next_forget[set];
        float keep = decay, take = 1.0f;
        if (exponential) {
            const float log_in = raw_in, log_forget = raw_forget;     // made log gates by `log_gates_kernel`
            const float m_new = fmaxf(log_forget + m, log_in);
            keep = expf(log_forget + m - m_new);
            take = expf(log_in - m_new);
            m = m_new;
        }
        const float value = is_n ? 1.0f : live ? activate(raw_value, activation) : 0.0f;
        const float scaled = take * value;
        float sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};      // four chains, so that a sum does not wait for the one before it
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            if (row0 + r < kDim) {
                S[r] = fmaf(keep, S[r], ks[half][row0 + r] * scaled);
                sums[r & 3] = fmaf(S[r], qs[half][row0 + r], sums[r & 3]);
            }
        }
        // One barrier per token: partial sums and the next token's q and k go to the halves of shared memory that nobody reads
        // now; behind the barrier the first thread of each column adds the parts up, and n's as well for the denominator.
        partial[half][part][local] = (sums[0] + sums[1]) + (sums[2] + sums[3]);
        if (token + 1 < end) publish((set + 1) % kAhead, half ^ 1);
        fetch(set, token + kAhead);                 // this set's q and k were published a token ago, its v and gates just used
        __syncthreads();
        if (part == 0 && live && !is_n) {
            float sum = 0.0f;
#pragma unroll
            for (int p = 0; p < kSplit; ++p) sum += partial[half][p][local];
            if (exponential) {
                float normaliser = 0.0f;
#pragma unroll
                for (int p = 0; p < kSplit; ++p) normaliser += partial[half][p][kColumns - 1];
                sum /= fmaxf(fabsf(normaliser), expf(-m)) + 1e-6f;
            }
            out[static_cast<size_t>(token) * heads * value_dim + head * value_dim + column] = sum;
        }
      }
    }
    if (live && (!is_n || blockIdx.z == 0)) {
#pragma unroll
        for (int r = 0; r < kRows; ++r)
            if (row0 + r < kDim) record[static_cast<size_t>(column) * kDim + row0 + r] = S[r];
    }
    if (exponential && blockIdx.z == 0 && threadIdx.x == 0) record[static_cast<size_t>(columns) * kDim] = m;
}

// ---- runs of tokens in chunks -------------------------------------------------------------------------------------------------
constexpr bool kChunked = kDim % 16 == 0 && kDim <= 256;
constexpr int kTile = 16;             // state columns of a block
constexpr int kPitch = kDim + 8;      // elements of a row of q or k in shared memory: eight rows, 16 bytes beside a multiple of 32, meet different banks
constexpr int kWalkers = 512;         // threads of chunk_state: 16 warps, so that a scheduler has four to choose from
constexpr int kKeySteps = kDim / 16 > 0 ? kDim / 16 : 1;
constexpr int kGroups = kKeySteps >= 16 ? 16 : kKeySteps >= 8 ? 8 : kKeySteps >= 4 ? 4 : kKeySteps >= 2 ? 2 : 1;      // warps that share the key elements out

// Sizes by what q and k are: exact in bfloat16 (one piece each), or numbers behind an activation (three).
template <int kOperand> struct Chunk {
    static constexpr int kTokens = kOperand == 1 ? 64 : 32;      // three pieces of 64 tokens, twice buffered, would not fit shared memory
    static constexpr int kScorePitch = kTokens + 8;
    static constexpr int kKeyBytes = kOperand * kTokens * kPitch * 2;
    static constexpr int kScoreBytes = chunk::kPieces * kTokens * kScorePitch * 2;
    static constexpr int kValueBytes = kOperand * kTokens * 24 * 2;
    static constexpr int kWriteBytes = chunk::kPieces * kTile * kScorePitch * 2;
    static constexpr int kSumPitch = 16;                         // columns 8-15 first in every other pair of rows, so that four rows meet all banks
    static constexpr int kSumBytes = kGroups * kTokens * kSumPitch * 4;
    static constexpr int kScalars = 3 * kTokens + 4;             // per (chunk, head): g (times the query scale), w(last, .), exp(-m), then g(last) and m behind the chunk
    static constexpr int kBytes = 3 * kKeyBytes + kScoreBytes + 2 * kValueBytes + kWriteBytes + kSumBytes + 2 * kScalars * 4 + kTokens * 4 + 4 * 8 + 16;
};

// The chunks [first, behind) of a run of `length` tokens that lane `lane` of the scan goes over: every chunk belongs to one lane, and a lane that the run
// has no chunk for owns none (it must not write: the last chunk is another lane's).
__host__ __device__ inline void gate_piece(int length, int tokens, int lane, int* first, int* behind) {
    const int chunks = (length + tokens - 1) / tokens, per_lane = (chunks + 31) / 32;
    *first = lane * per_lane < chunks ? lane * per_lane : chunks;
    *behind = *first + per_lane < chunks ? *first + per_lane : chunks;
}

// Block: 256 threads per (head, run).  Forget sums F (64-bit, from the token's chunk's start) and the running maximum m of every token, and m before
// every chunk.  Max-plus is associative: eight threads, the scan's lane of `gate_piece`, go over a piece of the run, each over an eighth of a chunk at a time whose
// loads travel together, the pieces are joined, and each thread goes over its tokens again from the m that they start with.  Bound by the chains of additions: with one thread
// to a lane 2,048 tokens of 4 heads took 14 us, here 7 (an mLSTM layer 206 -> 198).
constexpr int kScanThreads = 256, kShare = 8;      // threads; those of a chunk

struct Step {      // what tokens do to the maximum before them: max(m + sum, high)
    double sum, high;
};
__device__ __forceinline__ Step then(const Step& first, const Step& second) { return {first.sum + second.sum, fmax(first.high + second.sum, second.high)}; }

template <int kTokens>
__global__ void __launch_bounds__(kScanThreads)
gate_scan_kernel(const float* __restrict__ gates, const float* __restrict__ state, long long slot_stride, const int* __restrict__ cu_seqlens,
                 const int* __restrict__ seq_slot, double* __restrict__ forget_sums, float* __restrict__ maxima, float* __restrict__ before, int heads, int value_dim,
                 int n_seqs, int chunks_from) {
    grid_dependents_launch();
    grid_dependency_wait();
    constexpr int kMine = kTokens / kShare;
    __shared__ Step pieces[kScanThreads / kShare];
    const int head = blockIdx.x, lane = threadIdx.x / kShare, share = threadIdx.x % kShare;
    const chunk::Run run = chunk::find_run<false>(cu_seqlens, n_seqs, chunks_from, kTokens, blockIdx.y);
    if (run.sequence < 0) return;
    const int begin = cu_seqlens[run.sequence], length = cu_seqlens[run.sequence + 1] - begin;
    int first, behind;
    gate_piece(length, kTokens, lane, &first, &behind);
    const float* forgets = gates + static_cast<size_t>(begin) * 2 * heads + heads + head;
    float forget[kMine], in[kMine];      // of this thread's tokens of a chunk; behind the run's end what changes nothing
    auto load = [&](int chunk_index) {
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int token = chunk_index * kTokens + share * kMine + i;
            forget[i] = token < length ? forgets[static_cast<size_t>(token) * 2 * heads] : 0.0f;
            in[i] = token < length ? forgets[static_cast<size_t>(token) * 2 * heads - heads] : -INFINITY;
        }
    };
    // This thread's tokens after those of the threads before it; `whole`: the chunk's.
    auto scan = [&](Step& whole) {
        Step mine = {0.0, -INFINITY};
#pragma unroll
        for (int i = 0; i < kMine; ++i) mine = then(mine, {forget[i], in[i]});
#pragma unroll
        for (int apart = 1; apart < kShare; apart <<= 1) {
            const Step other = {__shfl_up_sync(0xffffffffu, mine.sum, apart, kShare), __shfl_up_sync(0xffffffffu, mine.high, apart, kShare)};
            if (share >= apart) mine = then(other, mine);
        }
        whole = {__shfl_sync(0xffffffffu, mine.sum, kShare - 1, kShare), __shfl_sync(0xffffffffu, mine.high, kShare - 1, kShare)};
        const Step start = {__shfl_up_sync(0xffffffffu, mine.sum, 1, kShare), __shfl_up_sync(0xffffffffu, mine.high, 1, kShare)};
        return share > 0 ? start : Step{0.0, -INFINITY};
    };
    const int chunks = (length + kTokens - 1) / kTokens, turns = (chunks + kScanThreads / kShare - 1) / (kScanThreads / kShare);      // the same for all lanes of a warp
    Step piece = {0.0, -INFINITY}, start = piece, whole;
    for (int turn = 0; turn < turns; ++turn) {
        load(first + turn < behind ? first + turn : chunks);      // behind the last chunk: nothing
        start = scan(whole);
        piece = then(piece, whole);
    }
    if (share == 0) pieces[lane] = piece;
    __syncthreads();
    double mine = state[static_cast<size_t>(seq_slot[run.sequence]) * slot_stride + static_cast<size_t>(head + 1) * ((static_cast<size_t>(value_dim) + 1) * kDim + 1) - 1];
    for (int other = 0; other < lane; ++other) mine = fmax(mine + pieces[other].sum, pieces[other].high);
    float m = static_cast<float>(mine);
    const size_t row = static_cast<size_t>(head) * cu_seqlens[n_seqs] + begin;
    for (int turn = 0; turn < turns; ++turn) {
        const int chunk_index = first + turn < behind ? first + turn : chunks;
        if (turns > 1) {
            load(chunk_index);
            start = scan(whole);
        }
        if (chunk_index < chunks && share == 0) before[static_cast<size_t>(run.first + chunk_index) * heads + head] = m;
        double forgotten = start.sum;
        float high = static_cast<float>(fmax(static_cast<double>(m) + start.sum, start.high));
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int token = chunk_index * kTokens + share * kMine + i;
            forgotten += forget[i];
            high = fmaxf(forget[i] + high, in[i]);
            if (token < length) {
                forget_sums[row + token] = forgotten;
                maxima[row + token] = high;
            }
        }
        m = __shfl_sync(0xffffffffu, high, kShare - 1, kShare);
    }
}

// grid (chunk numbers, heads); block 128.  scores [chunk, head, piece, token, kScorePitch], scalars [chunk, head, Chunk::kScalars],
// tiles [chunk, head, q or k, piece, token, kPitch]: each as chunk_state lays it in shared memory, so that it takes one bulk copy.
template <int kOperand>
__global__ void __launch_bounds__(128)
chunk_scores_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, long long stride, const float* __restrict__ gates, const float* __restrict__ decays,
                    const double* __restrict__ forget_sums, const float* __restrict__ maxima, const float* __restrict__ before, const int* __restrict__ cu_seqlens,
                    int n_seqs, bf16* __restrict__ scores, float* __restrict__ scalars, bf16* __restrict__ tiles, int heads, int exponential, float query_scale,
                    int chunks_from) {
    if constexpr (kChunked) {
        using Sizes = Chunk<kOperand>;
        constexpr int kTokens = Sizes::kTokens;
        grid_dependency_wait();
        extern __shared__ __align__(128) unsigned char shared[];
        bf16* qs = reinterpret_cast<bf16*>(shared);                              // [pieces][tokens][kPitch]
        bf16* ks = qs + kOperand * kTokens * kPitch;
        double* row_part = reinterpret_cast<double*>(shared + 2 * Sizes::kKeyBytes);      // exponents: w(i, j) = exp(row_part[i] + column_part[j])
        double* column_part = row_part + kTokens;
        float* powers = reinterpret_cast<float*>(column_part + kTokens);         // decay^0 .. decay^tokens
        const int number = blockIdx.x, head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const chunk::Run run = chunk::find_run<true>(cu_seqlens, n_seqs, chunks_from, kTokens, number);
        if (run.sequence < 0) return;                                            // a number that no chunk has
        const int start = cu_seqlens[run.sequence] + (number - run.first) * kTokens, live = min(kTokens, cu_seqlens[run.sequence + 1] - start);
        const int tokens = cu_seqlens[n_seqs];
        constexpr int kVectors = kDim / 8;
        for (int item = threadIdx.x; item < 2 * kTokens * kVectors; item += 128) {
            const int which = item / (kTokens * kVectors), token = item / kVectors % kTokens, column = item % kVectors * 8;
            const bf16* source = (which ? k : q) + static_cast<size_t>(start + min(token, live - 1)) * stride + head * kDim + column;
            bf16* target = (which ? ks : qs) + token * kPitch + column;
            if (kOperand == 1) {
                chunk::copy16(target, source, token < live);
            } else {
                const uint4 raw = *reinterpret_cast<const uint4*>(source);
                const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
                uint32_t out[4][chunk::kPieces];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    chunk::split_pair(activate(__uint_as_float(words[i] << 16), 1), activate(__uint_as_float(words[i] & 0xffff0000u), 1), out[i]);
#pragma unroll
                for (int p = 0; p < kOperand; ++p) {
                    const uint4 piece = token < live ? make_uint4(out[0][p], out[1][p], out[2][p], out[3][p]) : make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4*>(target + p * kTokens * kPitch) = piece;
                }
            }
        }
        chunk::copies_commit();
        float* numbers = scalars + (static_cast<size_t>(number) * heads + head) * Sizes::kScalars;
        if (exponential) {
            const size_t row = static_cast<size_t>(head) * tokens + start;
            const double m_before = before[static_cast<size_t>(number) * heads + head];
            const double final_part = forget_sums[row + live - 1] - maxima[row + live - 1];
            for (int i = threadIdx.x; i < kTokens; i += 128) {
                const int at = min(i, live - 1);
                const double a = forget_sums[row + at] - maxima[row + at];
                const double b = gates[(static_cast<size_t>(start) + at) * 2 * heads + head] - forget_sums[row + at];
                row_part[i] = a;
                column_part[i] = b;
                numbers[i] = expf(static_cast<float>(a + m_before)) * query_scale;
                numbers[kTokens + i] = i < live ? expf(static_cast<float>(final_part + b)) : 0.0f;
                numbers[2 * kTokens + i] = expf(-maxima[row + at]);
                if (i == live - 1) {
                    numbers[3 * kTokens] = expf(static_cast<float>(a + m_before));
                    numbers[3 * kTokens + 1] = maxima[row + at];
                }
            }
        } else {
            for (int i = threadIdx.x; i <= kTokens; i += 128) {
                double power = 1.0, base = decays[head];
                for (int n = i; n > 0; n >>= 1, base *= base)
                    if (n & 1) power *= base;
                powers[i] = static_cast<float>(power);
            }
        }
        chunk::copies_wait<0>();
        chunk::shared_writes_ready();
        __syncthreads();
        if (threadIdx.x == 0) chunk::bulk_store(tiles + (static_cast<size_t>(number) * heads + head) * Sizes::kKeyBytes, shared, 2 * Sizes::kKeyBytes);
        if (!exponential) {
            for (int i = threadIdx.x; i < kTokens; i += 128) {
                numbers[i] = powers[min(i, live - 1) + 1] * query_scale;
                numbers[kTokens + i] = i < live ? powers[live - 1 - i] : 0.0f;
                numbers[2 * kTokens + i] = 0.0f;
                if (i == 0) numbers[3 * kTokens] = powers[live];
            }
        }
        // 16 rows of scores to a warp (or half of their columns, where there are two strips of rows for four warps).
        constexpr int kStrips = kTokens / 16, kPerStrip = 4 / kStrips, kColumns = kTokens / 8 / kPerStrip, kSmall = kOperand > 1 ? kColumns : 2;
        const int strip = warp % kStrips, column0 = warp / kStrips * kColumns;
        float sums[kColumns][4] = {};
        constexpr int kSteps = kDim / 16, kChain = kOperand == 1 ? 4 : 2;        // products onto one accumulator before it is added up
#pragma unroll 1
        for (int from = 0; from < kSteps; from += kChain) {
            float large[kColumns][4] = {}, small[kSmall][4] = {};
#pragma unroll
            for (int ahead = 0; ahead < kChain; ++ahead) {
                const int step = from + ahead;
                if (step >= kSteps) break;
#pragma unroll
                for (int p = 0; p < kOperand; ++p) {
                    uint32_t a[4];
                    chunk::load_matrices(a, qs + (p * kTokens + strip * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
#pragma unroll
                    for (int other = 0; other + p < kOperand; ++other)
#pragma unroll
                        for (int n = 0; n < kColumns; n += 2) {
                            uint32_t b[4];      // two tiles of eight keys, 16 elements each
                            chunk::load_matrices(b, ks + (other * kTokens + (column0 + n) * 8 + lane % 8 + lane / 16 * 8) * kPitch + step * 16 + lane / 8 % 2 * 8);
                            chunk::multiply(p + other > 0 ? small[n % kSmall] : large[n], a, b[0], b[1]);
                            chunk::multiply(p + other > 0 ? small[(n + 1) % kSmall] : large[n + 1], a, b[2], b[3]);
                        }
                }
            }
#pragma unroll
            for (int n = 0; n < kColumns; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) sums[n][e] += kOperand > 1 ? large[n][e] + small[n % kSmall][e] : large[n][e];
        }
        bf16* target = scores + (static_cast<size_t>(number) * heads + head) * (Sizes::kScoreBytes / 2);
#pragma unroll
        for (int n = 0; n < kColumns; ++n)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = strip * 16 + lane / 4 + half * 8, j = (column0 + n) * 8 + lane % 4 * 2;
                float pair[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool seen = j + e <= i && i < live;
                    const float weight = !seen ? 0.0f : exponential ? expf(static_cast<float>(row_part[i] + column_part[j + e])) : powers[i - j - e];
                    pair[e] = seen ? sums[n][half * 2 + e] * query_scale * weight : 0.0f;
                }
                uint32_t pieces[chunk::kPieces];
                chunk::split_pair(pair[0], pair[1], pieces);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) *reinterpret_cast<uint32_t*>(target + (p * kTokens + i) * Sizes::kScorePitch + j) = pieces[p];
            }
        if (threadIdx.x == 0) chunk::bulk_stored();
    }
}

// grid (heads, runs, tiles of state columns); block kWalkers.  A group of key elements belongs to a warp (to several, if there are fewer groups than
// warps: they share the tokens of q S out and each keep the state): S^T tiles of 16 columns by 16 key elements, as accumulators.  As such they are,
// split in pieces, the right operand of q S without passing memory; the groups' sums meet in shared memory.  Between the two barriers of a chunk
// every warp works on the state; behind them the first half of the warps finishes the chunk's read-outs while the second half lays out the next
// chunk's values and asks for its rows.
template <int kOperand>
__global__ void __launch_bounds__(kWalkers)
chunk_state_kernel(const bf16* __restrict__ tiles, const bf16* __restrict__ v, long long v_stride,
                   const bf16* __restrict__ scores, const float* __restrict__ scalars, const float* __restrict__ start, float* __restrict__ state, long long slot_stride,
                   const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, float* __restrict__ out, int heads, int value_dim, int exponential,
                   int n_seqs, int chunks_from) {
    if constexpr (kChunked) {
        using Sizes = Chunk<kOperand>;
        constexpr int kTokens = Sizes::kTokens, kStrips = kTokens / 16, kHalf = kWalkers / 2;
        constexpr int kMine = (kKeySteps + kGroups - 1) / kGroups, kParts = kWalkers / 32 / kGroups, kMyStrips = kParts >= kStrips ? 1 : kStrips / kParts;
        constexpr int kValues = kTokens * kTile / kHalf;         // value elements of a thread of the second half
        grid_dependency_wait();
        extern __shared__ __align__(128) unsigned char shared[];
        bf16* query_rows = reinterpret_cast<bf16*>(shared);                      // [2][pieces][tokens][kPitch]
        bf16* ks = reinterpret_cast<bf16*>(shared + 2 * Sizes::kKeyBytes);
        bf16* ps = reinterpret_cast<bf16*>(shared + 3 * Sizes::kKeyBytes);       // scores [piece][token][kScorePitch]
        bf16* value_rows = ps + Sizes::kScoreBytes / 2;                          // values [2][piece][token][24]
        bf16* ws = value_rows + Sizes::kValueBytes;                              // w(last, .) v, turned [piece][column][kScorePitch]
        float* partial = reinterpret_cast<float*>(ws + Sizes::kWriteBytes / 2);  // [group][token][kSumPitch]
        float* numbers = partial + Sizes::kSumBytes / 4;                         // [2][kScalars]
        float* denominators = numbers + 2 * Sizes::kScalars;                     // [tokens]
        uint64_t* barriers = reinterpret_cast<uint64_t*>(denominators + kTokens);      // queries of even and odd chunks, keys, scores
        const int head = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const chunk::Run run = chunk::find_run<false>(cu_seqlens, n_seqs, chunks_from, kTokens, blockIdx.y);
        if (run.sequence < 0) return;
        const int sequence = run.sequence, first = run.first;
        const int group = warp % kGroups, part = warp / kGroups;
        const bool second = threadIdx.x >= kHalf;
        const int helper = threadIdx.x - kHalf;                                  // number among the second half
        const int begin = cu_seqlens[sequence], end = cu_seqlens[sequence + 1];
        const int columns = value_dim + (exponential ? 1 : 0), tile = exponential ? kTile - 1 : kTile;
        // The state column of a column of the tile, or -1; the last one is n with the exponential gating.
        auto column_of = [&](int local) {
            const int column = exponential && local == kTile - 1 ? value_dim : static_cast<int>(blockIdx.z) * tile + local;
            return column < value_dim || (exponential && local == kTile - 1) ? column : -1;
        };
        float* record = state + static_cast<size_t>(seq_slot[sequence]) * slot_stride + static_cast<size_t>(head) * (static_cast<size_t>(columns) * kDim + (exponential ? 1 : 0));
        float S[kMine][2][4];
#pragma unroll
        for (int mine = 0; mine < kMine; ++mine)
#pragma unroll
            for (int side = 0; side < 2; ++side)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int column = column_of(lane / 4 + half * 8), element = (group + mine * kGroups) * 16 + side * 8 + lane % 4 * 2;
                    const bool there = column >= 0 && element < kDim;
                    const float* source = there && column == value_dim ? start + (static_cast<size_t>(sequence) * heads + head) * (kDim + 1) : record + static_cast<size_t>(there ? column : 0) * kDim;
                    S[mine][side][half * 2] = there ? source[element] : 0.0f;
                    S[mine][side][half * 2 + 1] = there ? source[element + 1] : 0.0f;
                }
        const int chunks = (end - begin + kTokens - 1) / kTokens;
        // The second half's work: a chunk's tiles of queries, keys and scores (one thread asks for them), its values and numbers.
        auto ask_tile = [&](int which, bf16* target, uint64_t* barrier, int chunk_index) {
            chunk::barrier_expect(barrier, Sizes::kKeyBytes);
            chunk::bulk_copy(target, tiles + ((static_cast<size_t>(first + chunk_index) * heads + head) * 2 + which) * (Sizes::kKeyBytes / 2), Sizes::kKeyBytes, barrier);
        };
        auto ask_scores = [&](int chunk_index) {
            chunk::barrier_expect(barriers + 3, Sizes::kScoreBytes);
            chunk::bulk_copy(ps, scores + (static_cast<size_t>(first + chunk_index) * heads + head) * (Sizes::kScoreBytes / 2), Sizes::kScoreBytes, barriers + 3);
        };
        const bool asks = helper == 0;
        // A thread's values: one column of neighbouring tokens, two by two.
        const int my_column = column_of(helper % kTile);
        const bool is_n = exponential && helper % kTile == kTile - 1;
        auto token_of = [&](int i) { return helper / kTile * 2 + i % 2 + i / 2 * (2 * kHalf / kTile); };
        float next_value[kValues], next_weight[kValues], next_number = 0.0f;
        auto fetch = [&](int chunk_index) {
            const float* source = scalars + (static_cast<size_t>(first + chunk_index) * heads + head) * Sizes::kScalars;
#pragma unroll
            for (int i = 0; i < kValues; ++i) {
                const int token = token_of(i), at = begin + chunk_index * kTokens + token;
                next_weight[i] = source[kTokens + token];
                next_value[i] = at >= end || my_column < 0 ? 0.0f : is_n ? 1.0f : __bfloat162float(v[static_cast<size_t>(at) * v_stride + head * value_dim + my_column]);
            }
            if (helper <= 3 * kTokens + 1) next_number = source[helper];
        };
        bool odd = false;      // an infinity or NaN among the values
        auto publish = [&](int chunk_index) {
            bf16* vs = value_rows + (chunk_index & 1) * (Sizes::kValueBytes / 2);
            odd = false;
#pragma unroll
            for (int i = 0; i < kValues; i += 2) {
                float value[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    value[e] = is_n || kOperand == 1 ? next_value[i + e] : activate(next_value[i + e], 1);
                    odd |= !(fabsf(value[e]) < INFINITY);
                    bf16 pieces[chunk::kPieces];
                    chunk::split_one(value[e], pieces);
#pragma unroll
                    for (int p = 0; p < kOperand; ++p) vs[(p * kTokens + token_of(i + e)) * 24 + helper % kTile] = pieces[p];
                }
                uint32_t pieces[chunk::kPieces];
                chunk::split_pair(value[0] * next_weight[i], value[1] * next_weight[i + 1], pieces);
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p) *reinterpret_cast<uint32_t*>(ws + (p * kTile + helper % kTile) * Sizes::kScorePitch + token_of(i)) = pieces[p];
            }
            if (helper <= 3 * kTokens + 1) numbers[(chunk_index & 1) * Sizes::kScalars + helper] = next_number;
        };
        volatile int* gone = reinterpret_cast<volatile int*>(barriers + 4);      // see barrier_wait; then the last chunk whose keys were asked for
        if (threadIdx.x < 4) chunk::barrier_init(barriers + threadIdx.x);
        if (threadIdx.x < 2) gone[threadIdx.x] = 0;
        chunk::barriers_ready();
        __syncthreads();
        if (second) {
            if (asks) {
                ask_tile(0, query_rows, barriers, 0);
                ask_tile(1, ks, barriers + 2, 0);
            }
            fetch(0);
            publish(0);
            if (chunks > 1) fetch(1);
        }
        // After a wait that ran out: the copies that may be in flight (those that are there cost nothing); then the block ends, the state as it was.
        auto settle = [&](int queries_of, int scores_of) {
            if (queries_of > 0) chunk::barrier_wait(barriers + ((queries_of - 1) & 1), (queries_of - 1) / 2 & 1, nullptr);
            chunk::barrier_wait(barriers + (queries_of & 1), queries_of / 2 & 1, nullptr);
            chunk::barrier_wait(barriers + 2, gone[1] & 1, nullptr);
            chunk::barrier_wait(barriers + 3, scores_of & 1, nullptr);
        };
        for (int chunk_index = 0; chunk_index < chunks; ++chunk_index) {
            const float* scalar = numbers + (chunk_index & 1) * Sizes::kScalars;
            const bf16* vs = value_rows + (chunk_index & 1) * (Sizes::kValueBytes / 2);
            const bf16* qs = query_rows + (chunk_index & 1) * kOperand * kTokens * kPitch;
            const bool careful = __syncthreads_or(odd || gone[0] != 0);      // the chunk's values and numbers are there
            if (careful && __syncthreads_or(gone[0] != 0)) {                 // ... or a wait of the chunk before ran out
                settle(chunk_index, chunk_index - 1);
                return;
            }
            if (asks) {
                ask_scores(chunk_index);
                if (chunk_index + 1 < chunks) ask_tile(0, query_rows + ((chunk_index + 1) & 1) * kOperand * kTokens * kPitch, barriers + ((chunk_index + 1) & 1), chunk_index + 1);
            }
            chunk::barrier_wait(barriers + (chunk_index & 1), chunk_index / 2 & 1, gone);
            // q S over this warp's key elements.  Loops run over independent accumulators inside and over the pieces outside, so that a product does
            // not wait for the one before it.
            if (part * kMyStrips < kStrips) {
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
                        for (int p = kOperand - 1; p >= 0; --p) {      // the small products first
                            uint32_t a[kMyStrips][4];
#pragma unroll
                            for (int strip = 0; strip < kMyStrips; ++strip)
                                chunk::load_matrices(a[strip], qs + (p * kTokens + (part * kMyStrips + strip) * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
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
                        for (int half = 0; half < 2; ++half)
                            *reinterpret_cast<float2*>(partial + (group * kTokens + (part * kMyStrips + strip) * 16 + lane / 4 + half * 8) * Sizes::kSumPitch + (n ^ lane / 8 % 2) * 8 + lane % 4 * 2) =
                                make_float2(sums[strip][n][half * 2], sums[strip][n][half * 2 + 1]);
            }
            // The state behind the chunk.  Its keys were asked for last, behind the barrier before: they travel beside q S.
            chunk::barrier_wait(barriers + 2, chunk_index & 1, gone);
            const float keep = scalar[3 * kTokens];
            float large[kMine][2][4] = {}, small[kMine][2][2][4] = {};
#pragma unroll
            for (int strip = 0; strip < kStrips; ++strip) {
                uint32_t a[chunk::kPieces][4];
#pragma unroll
                for (int p = 0; p < chunk::kPieces; ++p)
                    chunk::load_matrices(a[p], ws + (p * kTile + lane % 16) * Sizes::kScorePitch + strip * 16 + lane / 16 * 8);
#pragma unroll
                for (int mine = 0; mine < kMine; ++mine) {
                    const int step = group + mine * kGroups;
                    if (step < kKeySteps) {
#pragma unroll
                        for (int p = 0; p < kOperand; ++p) {
                            uint32_t b[4];
                            chunk::load_matrices_turned(b, ks + (p * kTokens + strip * 16 + lane % 16) * kPitch + step * 16 + lane / 16 * 8);
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
            __syncthreads();      // the groups' sums are there, the keys and weighted values are done with
            if (second) {
                if (chunk_index + 1 < chunks) {
                    if (asks && !gone[0]) {
                        ask_tile(1, ks, barriers + 2, chunk_index + 1);
                        gone[1] = chunk_index + 1;
                    }
                    publish(chunk_index + 1);
                    if (chunk_index + 2 < chunks) fetch(chunk_index + 2);
                }
                continue;
            }
            // Scores times values: 16 tokens by 8 columns to a warp.
            const int strip = warp / 2, n = warp % 2, row = strip * 16 + lane / 4, local = n * 8 + lane % 4 * 2;
            float inside[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            chunk::barrier_wait(barriers + 3, chunk_index & 1, gone);
            if (strip < kStrips) {
                if (!careful) {
                    float small_sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    for (int step = 0; step <= strip; ++step) {
                        uint32_t b[kOperand][2];
#pragma unroll
                        for (int p = 0; p < kOperand; ++p) chunk::load_pair_turned(b[p], vs + (p * kTokens + step * 16 + lane % 16) * 24 + n * 8);
#pragma unroll
                        for (int p = 0; p < chunk::kPieces; ++p) {
                            uint32_t a[4];
                            chunk::load_matrices(a, ps + (p * kTokens + strip * 16 + lane % 16) * Sizes::kScorePitch + step * 16 + lane / 16 * 8);
#pragma unroll
                            for (int other = 0; other < kOperand && other + p < chunk::kPieces; ++other) chunk::multiply(p + other == 0 ? inside : small_sums, a, b[other][0], b[other][1]);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) inside[e] += small_sums[e];
                } else {      // an infinity or NaN must not reach the tokens before it, as a score of zero times it would
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = row + e / 2 * 8;
                        for (int j = 0; j <= i; ++j) {
                            float score = 0.0f, value = __bfloat162float(vs[j * 24 + local + e % 2]);
#pragma unroll
                            for (int p = chunk::kPieces - 1; p >= 0; --p) score += __bfloat162float(ps[(p * kTokens + i) * Sizes::kScorePitch + j]);
#pragma unroll
                            for (int p = 1; p < kOperand; ++p)
                                if (fabsf(value) < INFINITY) value += __bfloat162float(vs[(p * kTokens + j) * 24 + local + e % 2]);
                            inside[e] = fmaf(score, value, inside[e]);
                        }
                    }
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int from = 0; from < kGroups; ++from) {
                        const float2 part_sum = *reinterpret_cast<const float2*>(partial + (from * kTokens + row + half * 8) * Sizes::kSumPitch + (n ^ lane / 8 % 2) * 8 + lane % 4 * 2);
                        sum.x += part_sum.x;
                        sum.y += part_sum.y;
                    }
                    inside[half * 2] = fmaf(scalar[row + half * 8], sum.x, inside[half * 2]);
                    inside[half * 2 + 1] = fmaf(scalar[row + half * 8], sum.y, inside[half * 2 + 1]);
                    if (exponential && n == 1 && lane % 4 == 3) denominators[row + half * 8] = fmaxf(fabsf(inside[half * 2 + 1]), scalar[2 * kTokens + row + half * 8]) + 1e-6f;
                }
            }
            if (exponential) asm volatile("bar.sync 1, %0;" ::"n"(kHalf) : "memory");      // the first half alone
            if (strip < kStrips) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int token = begin + chunk_index * kTokens + row + e / 2 * 8, column = column_of(local + e % 2);
                    if (token < end && column >= 0 && column < value_dim)
                        out[static_cast<size_t>(token) * heads * value_dim + head * value_dim + column] = exponential ? inside[e] / denominators[row + e / 2 * 8] : inside[e];
                }
            }
        }
        if (__syncthreads_or(gone[0] != 0)) {
            settle(chunks - 1, chunks - 1);
            return;
        }
        if (exponential && blockIdx.z == 0 && threadIdx.x == 0) record[static_cast<size_t>(columns) * kDim] = numbers[((chunks - 1) & 1) * Sizes::kScalars + 3 * kTokens + 1];
        if (part == 0) {
#pragma unroll
            for (int mine = 0; mine < kMine; ++mine)
#pragma unroll
                for (int side = 0; side < 2; ++side)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int column = column_of(lane / 4 + e / 2 * 8), element = (group + mine * kGroups) * 16 + side * 8 + lane % 4 * 2 + e % 2;
                        if (column >= 0 && element < kDim && (column < value_dim || blockIdx.z == 0)) record[static_cast<size_t>(column) * kDim + element] = S[mine][side][e];
                    }
        }
    }
}

// Whether runs of these sizes can be walked in chunks.
bool chunks_served(int activation) { return kChunked && (!activation || kDim <= 128); }

// The workspace's parts, each on a 16-byte border: n and m before the run first, the rest for chunks.
struct Workspace {
    size_t scores, scalars, tiles, forget_sums, maxima, before, bytes;
};
Workspace workspace_of(int tokens, int n_seqs, int heads, int exponential, int activation, int chunks_from) {
    const size_t numbers = chunk::most_chunks(tokens, n_seqs, chunks_from, activation ? Chunk<3>::kTokens : Chunk<1>::kTokens);
    Workspace w;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t here = at; at += (bytes + 15) / 16 * 16; return here; };
    take(exponential ? start_floats(n_seqs, heads) * 4 : 0);
    w.scores = take(numbers * heads * (activation ? Chunk<3>::kScoreBytes : Chunk<1>::kScoreBytes));
    w.scalars = take(numbers * heads * (activation ? Chunk<3>::kScalars : Chunk<1>::kScalars) * 4);
    w.tiles = take(numbers * heads * 2 * (activation ? Chunk<3>::kKeyBytes : Chunk<1>::kKeyBytes));
    w.forget_sums = take(exponential ? static_cast<size_t>(tokens) * heads * 8 : 0);
    w.maxima = take(exponential ? static_cast<size_t>(tokens) * heads * 4 : 0);
    w.before = take(exponential ? numbers * heads * 4 : 0);
    w.bytes = at;
    return w;
}

template <int kOperand>
int launch_chunks(const bf16* q, const bf16* k, const bf16* v, long long stride, const float* gates, const float* decays, float* state, long long slot_stride,
                  const int* cu_seqlens, const int* seq_slot, float* out, int tokens, int n_seqs, int heads, int value_dim, int exponential, float query_scale,
                  int chunks_from, unsigned char* workspace, cudaStream_t s) {
    using Sizes = Chunk<kOperand>;
    const Workspace w = workspace_of(tokens, n_seqs, heads, exponential, kOperand == 3, chunks_from);
    const int runs = chunk::most_runs(tokens, n_seqs, chunks_from);
    if (runs == 0) return 0;      // all are shorter
    bf16* scores = reinterpret_cast<bf16*>(workspace + w.scores);
    bf16* tiles = reinterpret_cast<bf16*>(workspace + w.tiles);
    float* scalars = reinterpret_cast<float*>(workspace + w.scalars);
    double* forget_sums = reinterpret_cast<double*>(workspace + w.forget_sums);
    float* maxima = reinterpret_cast<float*>(workspace + w.maxima);
    float* before = reinterpret_cast<float*>(workspace + w.before);
    const int score_bytes = 2 * Sizes::kKeyBytes + Sizes::kTokens * 16 + (Sizes::kTokens + 1) * 4;
    if (cudaFuncSetAttribute(chunk_scores_kernel<kOperand>, cudaFuncAttributeMaxDynamicSharedMemorySize, score_bytes) != cudaSuccess
        || cudaFuncSetAttribute(chunk_state_kernel<kOperand>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sizes::kBytes) != cudaSuccess)
        return cudaErrorInvalidValue;
    if (exponential)
        tau_launch(gate_scan_kernel<Sizes::kTokens>, dim3(heads, runs), dim3(kScanThreads), 0, s, gates, state, slot_stride, cu_seqlens, seq_slot, forget_sums, maxima, before, heads, value_dim,
                   n_seqs, chunks_from);
    // These two start when the kernel before them has finished, and the next when they have (as the delta rule's chunks do, and for the reason given there).
    tau_launch_as(false, chunk_scores_kernel<kOperand>, dim3(chunk::most_chunks(tokens, n_seqs, chunks_from, Sizes::kTokens), heads), dim3(128), score_bytes, s, q, k, stride, gates, decays,
               static_cast<const double*>(forget_sums), static_cast<const float*>(maxima), static_cast<const float*>(before), cu_seqlens, n_seqs, scores, scalars, tiles,
               heads, exponential, query_scale, chunks_from);
    const int tile = exponential ? kTile - 1 : kTile;
    tau_launch_as(false, chunk_state_kernel<kOperand>, dim3(heads, runs, (value_dim + tile - 1) / tile), dim3(kWalkers), Sizes::kBytes, s, static_cast<const bf16*>(tiles), v, stride,
               static_cast<const bf16*>(scores), static_cast<const float*>(scalars), reinterpret_cast<const float*>(workspace), state, slot_stride, cu_seqlens, seq_slot, out,
               heads, value_dim, exponential, n_seqs, chunks_from);
    return tau_launch_status();
}

}  // namespace

TAU_EXPORT int tau_recurrence_key_dim() { return kDim; }
// The chunks of a run that a lane of the gates' scan writes (host arithmetic, for tests).
TAU_EXPORT void tau_recurrence_gate_piece(int length, int tokens, int lane, int* first, int* behind) { gate_piece(length, tokens, lane, first, behind); }

// 1 if a bounded wait ran out since the library was loaded (synchronises the device).
TAU_EXPORT int tau_recurrence_status() { return chunk::wait_status(); }
// Whether bfloat16 runs of these sizes can be walked in chunks, and the bytes of workspace that `tau_linear_recurrence` wants with that `chunks` (0: none).
TAU_EXPORT int tau_recurrence_chunks(int activation) { return chunks_served(activation) ? 1 : 0; }
TAU_EXPORT long long tau_recurrence_workspace(int tokens, int n_seqs, int heads, int exponential, int activation, int chunks) {
    if (tokens <= 0 || n_seqs <= 0 || heads <= 0) return 0;
    if (!chunks) return exponential ? start_floats(n_seqs, heads) * 4 : 0;
    return static_cast<long long>(workspace_of(tokens, n_seqs, heads, exponential, activation, chunks).bytes);
}

// q, k, v: rows `stride` elements apart, heads side by side.  gates [tokens, 2 heads] (exponential; pre-activations, turned into log
// gates in place) or decays [heads].
// state: records `slot_stride` floats apart per slot.  out [tokens, heads * value_dim], 32-bit.
// `workspace`: 16-byte aligned, `tau_recurrence_workspace` bytes.  `chunks` > 0: bfloat16 runs of that many tokens and more go in chunks, and with `shorter`
// the others token by token (without it there are none).
TAU_EXPORT int tau_linear_recurrence(int dtype, const void* q, const void* k, const void* v, long long stride, float* gates,
                                     const float* decays, float* state, long long slot_stride, const int* cu_seqlens, const int* seq_slot,
                                     float* out, int tokens, int n_seqs, int heads, int value_dim, int exponential, float gate_cap, float query_scale,
                                     int activation, int chunks, int shorter, void* workspace, long long workspace_bytes, void* stream) {
    if (n_seqs <= 0) return 0;
    if (!q || !k || !v || !state || !cu_seqlens || !seq_slot || !out || heads <= 0 || value_dim <= 0 || (exponential ? !gates : !decays))
        return cudaErrorInvalidValue;
    const long long needed = tau_recurrence_workspace(tokens, n_seqs, heads, exponential, activation, chunks);
    if (needed > 0 && (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 15) != 0 || workspace_bytes < needed)) return cudaErrorInvalidValue;
    if (chunks && (dtype != TAU_BF16 || !chunks_served(activation) || tokens <= 0 || stride % 8 != 0 || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k)) & 15) != 0))
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float* start = static_cast<float*>(workspace);
    if (exponential) {
        if (tokens <= 0) return cudaErrorInvalidValue;
        const long long count = static_cast<long long>(tokens) * 2 * heads, most = count > start_floats(n_seqs, heads) ? count : start_floats(n_seqs, heads);
        tau_launch(log_gates_kernel, dim3(static_cast<unsigned>((most + 255) / 256 < 1184 ? (most + 255) / 256 : 1184)), dim3(256), 0, s, gates, count, heads, gate_cap,
                   static_cast<const float*>(state), slot_stride, seq_slot, n_seqs, value_dim, start);
        const int status = tau_launch_status();
        if (status != 0) return status;
    }
    if constexpr (kChunked) {
        if (chunks) {
            const bf16 *qs = static_cast<const bf16*>(q), *ks = static_cast<const bf16*>(k), *vs = static_cast<const bf16*>(v);
            unsigned char* bytes = static_cast<unsigned char*>(workspace);
            int status = 0;
            bool done = false;
            if constexpr (kDim <= 128)
                if (activation) {
                    status = launch_chunks<3>(qs, ks, vs, stride, gates, decays, state, slot_stride, cu_seqlens, seq_slot, out, tokens, n_seqs, heads, value_dim, exponential, query_scale, chunks, bytes, s);
                    done = true;
                }
            if (!done) status = launch_chunks<1>(qs, ks, vs, stride, gates, decays, state, slot_stride, cu_seqlens, seq_slot, out, tokens, n_seqs, heads, value_dim, exponential, query_scale, chunks, bytes, s);
            if (status != 0 || !shorter) return status;
        }
    }
    const int below = chunks ? chunks : 0x7fffffff;
    const int wide = exponential ? 31 : 32;
    const bool narrow = heads * n_seqs * ((value_dim + wide - 1) / wide) < 148 && kSplit <= 16;     // blocks of 16 columns reach more SMs
    const int tile = narrow ? (exponential ? 15 : 16) : wide;
    dim3 grid(heads, n_seqs, (value_dim + tile - 1) / tile), block((narrow ? 16 : 32) * kSplit);
    if (dtype != TAU_F32 && dtype != TAU_BF16) return cudaErrorInvalidValue;
    const bool dependent = chunks || tokens <= 4 * n_seqs;      // the few long blocks of a walk over runs pile up on the SMs that fall free first if they start early
#define TAU_RECURRENCE(T, COLUMNS)                                                                                                          \
    tau_launch_as(dependent, linear_recurrence_kernel<T, COLUMNS>, grid, block, 0, s, static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), \
               stride, gates, decays, static_cast<const float*>(start), state, slot_stride, cu_seqlens, seq_slot, out, heads, value_dim, exponential, gate_cap, query_scale, activation, below)
    if (dtype == TAU_F32) {
        if (narrow) TAU_RECURRENCE(float, 16); else TAU_RECURRENCE(float, 32);
    } else {
        if (narrow) TAU_RECURRENCE(bf16, 16); else TAU_RECURRENCE(bf16, 32);
    }
#undef TAU_RECURRENCE
    return tau_launch_status();
}
