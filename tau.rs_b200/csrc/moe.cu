// Routed experts, token by token: a router that scores the experts in 32-bit and picks `top` of them, the chosen
// experts' gated products, and the weighted sum of their outputs (plus a shared expert's, scaled by its own gate).
//
//   route:    z = W_router h + bias (32-bit weights and sums; the bias is optional); s = sigmoid(z) or softmax(z); the `top` largest of
//             s + correction are chosen (the lowest index among equals), their weights are s itself, divided by
//             their sum (+ 1e-20) if `renormalize`, times a constant; shared_gate = sigmoid(w_sg . h).  With `groups` > 1 the
//             experts form that many equal groups of neighbours; a group is ranked by the sum of the two largest of its
//             s + correction (by its only one in groups of one), and only experts of the `keep` best groups (the lowest index
//             among equals) can be chosen.
//   gate_up:  inner[token, place] = silu(W_gate[e] h) * (W_up[e] h) for the expert e of each (token, place), or with a limit
//             L > 0 g sigmoid(1.702 g) (u + 1), g = min(W_gate[e] h, L), u = W_up[e] h held between -L and L.
//   down:     out[token] = sum over places of weight * (W_down[e] inner[token, place]) + shared_gate * shared[token], 32-bit.
//
// Experts numbered `real_experts` and up have no weights: they return what they read (identity experts), so a pair that chose one adds
// weight * h to the token's sum.
//
// These are weight-streaming kernels: a warp per output feature, the activation row in shared memory as floats.
#include "chunk_mma.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Dot product of a weight row with a float vector in shared memory, over the warp.
template <typename T>
__device__ __forceinline__ float warp_dot(const T* __restrict__ weights, const float* __restrict__ vector, int length, int lane) {
    float sum = 0.0f;
    for (int column = lane; column < length; column += 32) sum = fmaf(to_float(weights[column]), vector[column], sum);
    return warp_sum(sum);
}

// Dot products of one 32-bit row (the router's) with `kRows` vectors in shared memory, `pitch` floats apart, over the warp; a row that starts
// on a 16-byte boundary is read four elements at a time.  The order of the sums is the same for every `kRows`.
template <int kRows>
__device__ __forceinline__ void warp_dot_rows(const float* __restrict__ weights, const float* __restrict__ vectors, int pitch, int length, int lane, float (&sums)[kRows]) {
    float other[kRows];
#pragma unroll
    for (int row = 0; row < kRows; ++row) sums[row] = other[row] = 0.0f;
    if ((reinterpret_cast<uintptr_t>(weights) & 15) == 0 && length % 4 == 0) {
        auto add = [](float sum, const float4& w, const float4& x) { return fmaf(w.x, x.x, fmaf(w.y, x.y, fmaf(w.z, x.z, fmaf(w.w, x.w, sum)))); };
        int column = lane * 4;
        // A block of one token is a chain of these loads: eight on their way at once.
#pragma unroll (kRows == 1 ? 4 : 1)
        for (; column + 128 < length; column += 256) {
            const float4 w0 = *reinterpret_cast<const float4*>(weights + column), w1 = *reinterpret_cast<const float4*>(weights + column + 128);
#pragma unroll
            for (int row = 0; row < kRows; ++row) {
                sums[row] = add(sums[row], w0, *reinterpret_cast<const float4*>(vectors + row * pitch + column));
                other[row] = add(other[row], w1, *reinterpret_cast<const float4*>(vectors + row * pitch + column + 128));
            }
        }
        if (column < length) {
            const float4 w0 = *reinterpret_cast<const float4*>(weights + column);
#pragma unroll
            for (int row = 0; row < kRows; ++row) sums[row] = add(sums[row], w0, *reinterpret_cast<const float4*>(vectors + row * pitch + column));
        }
    } else {
        for (int column = lane; column < length; column += 32) {
            const float w = weights[column];
#pragma unroll
            for (int row = 0; row < kRows; ++row) sums[row] = fmaf(w, vectors[row * pitch + column], sums[row]);
        }
    }
#pragma unroll
    for (int row = 0; row < kRows; ++row) sums[row] = warp_sum(sums[row] + other[row]);
}

// Eight bfloat16 weights against eight floats of shared memory, which are read as two 16-byte words (lanes 32 bytes apart meet
// two to a bank that way, not eight).
__device__ __forceinline__ float dot8(const uint4& raw, const float* __restrict__ vector) {
    const float4 low = *reinterpret_cast<const float4*>(vector), high = *reinterpret_cast<const float4*>(vector + 4);
    float sum = __uint_as_float(raw.x << 16) * low.x;
    sum = fmaf(__uint_as_float(raw.x & 0xffff0000u), low.y, sum);
    sum = fmaf(__uint_as_float(raw.y << 16), low.z, sum);
    sum = fmaf(__uint_as_float(raw.y & 0xffff0000u), low.w, sum);
    sum = fmaf(__uint_as_float(raw.z << 16), high.x, sum);
    sum = fmaf(__uint_as_float(raw.z & 0xffff0000u), high.y, sum);
    sum = fmaf(__uint_as_float(raw.w << 16), high.z, sum);
    sum = fmaf(__uint_as_float(raw.w & 0xffff0000u), high.w, sum);
    return sum;
}

// bfloat16 rows that start on a 16-byte boundary are read eight elements at a time.
template <>
__device__ __forceinline__ float warp_dot<bf16>(const bf16* __restrict__ weights, const float* __restrict__ vector, int length, int lane) {
    float sum = 0.0f;
    if ((reinterpret_cast<uintptr_t>(weights) & 15) == 0 && length % 8 == 0) {
        for (int column = lane * 8; column < length; column += 256) sum += dot8(*reinterpret_cast<const uint4*>(weights + column), vector + column);
    } else {
        for (int column = lane; column < length; column += 32) sum = fmaf(__bfloat162float(weights[column]), vector[column], sum);
    }
    return warp_sum(sum);
}

// Two dot products at once (a gate row and its up row, or the rows of two places), so that a lane has four 16-byte loads in
// flight where the rows allow them.
template <typename T>
__device__ __forceinline__ void warp_dot_pair(const T* __restrict__ first, const float* __restrict__ first_vector, const T* __restrict__ second,
                                              const float* __restrict__ second_vector, int length, int lane, float& first_sum, float& second_sum) {
    first_sum = warp_dot(first, first_vector, length, lane);
    second_sum = warp_dot(second, second_vector, length, lane);
}

template <>
__device__ __forceinline__ void warp_dot_pair<bf16>(const bf16* __restrict__ first, const float* __restrict__ first_vector, const bf16* __restrict__ second,
                                                    const float* __restrict__ second_vector, int length, int lane, float& first_sum, float& second_sum) {
    if (((reinterpret_cast<uintptr_t>(first) | reinterpret_cast<uintptr_t>(second)) & 15) != 0 || length % 8 != 0) {
        first_sum = warp_dot(first, first_vector, length, lane);
        second_sum = warp_dot(second, second_vector, length, lane);
        return;
    }
    float a = 0.0f, b = 0.0f, c = 0.0f, d = 0.0f;
    int column = lane * 8;
    for (; column + 768 < length; column += 1024) {      // eight loads in flight
        uint4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[i] = *reinterpret_cast<const uint4*>(first + column + 256 * i);
            y[i] = *reinterpret_cast<const uint4*>(second + column + 256 * i);
        }
        a += dot8(x[0], first_vector + column) + dot8(x[2], first_vector + column + 512);
        b += dot8(y[0], second_vector + column) + dot8(y[2], second_vector + column + 512);
        c += dot8(x[1], first_vector + column + 256) + dot8(x[3], first_vector + column + 768);
        d += dot8(y[1], second_vector + column + 256) + dot8(y[3], second_vector + column + 768);
    }
    for (; column + 256 < length; column += 512) {
        const uint4 a0 = *reinterpret_cast<const uint4*>(first + column), b0 = *reinterpret_cast<const uint4*>(second + column);
        const uint4 a1 = *reinterpret_cast<const uint4*>(first + column + 256), b1 = *reinterpret_cast<const uint4*>(second + column + 256);
        a += dot8(a0, first_vector + column);
        b += dot8(b0, second_vector + column);
        c += dot8(a1, first_vector + column + 256);
        d += dot8(b1, second_vector + column + 256);
    }
    if (column < length) {
        const uint4 a0 = *reinterpret_cast<const uint4*>(first + column), b0 = *reinterpret_cast<const uint4*>(second + column);
        a += dot8(a0, first_vector + column);
        b += dot8(b0, second_vector + column);
    }
    first_sum = warp_sum(a + c);
    second_sum = warp_sum(b + d);
}

// Activation rows as floats in shared memory: `count` elements from `source` on, 16 bytes at a time where they allow it.
__device__ __forceinline__ void unpack_eight(const uint4& raw, float* target) {
    *reinterpret_cast<float4*>(target) = make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
    *reinterpret_cast<float4*>(target + 4) = make_float4(__uint_as_float(raw.z << 16), __uint_as_float(raw.z & 0xffff0000u), __uint_as_float(raw.w << 16), __uint_as_float(raw.w & 0xffff0000u));
}

template <typename T>
__device__ __forceinline__ void stage_row(const T* __restrict__ source, float* __restrict__ target, int count) {
    if constexpr (sizeof(T) == 2) {
        if (((reinterpret_cast<uintptr_t>(source) | reinterpret_cast<uintptr_t>(target)) & 15) == 0 && count % 8 == 0) {
            for (int column = threadIdx.x * 8; column < count; column += blockDim.x * 8) unpack_eight(*reinterpret_cast<const uint4*>(source + column), target + column);
            return;
        }
    }
    for (int column = threadIdx.x; column < count; column += blockDim.x) target[column] = to_float(source[column]);
}

// One warp chooses a token's experts: `scores` [experts] holds its z and is followed by room for what is chosen by [experts] and the groups' ranks [groups].
__device__ __forceinline__ void choose_experts(float* scores, int token, int lane, const float* __restrict__ correction, int* __restrict__ chosen, float* __restrict__ weights,
                                               int experts, int top, int softmax, int renormalize, int groups, int keep, float scale) {
    float* choice = scores + experts;
    float* ranks = choice + experts;
    if (softmax) {
        float top_z = -INFINITY;
        for (int expert = lane; expert < experts; expert += 32) top_z = fmaxf(top_z, scores[expert]);
        top_z = warp_max(top_z);
        float total = 0.0f;
        for (int expert = lane; expert < experts; expert += 32) total += expf(scores[expert] - top_z);
        total = warp_sum(total);
        for (int expert = lane; expert < experts; expert += 32) scores[expert] = expf(scores[expert] - top_z) / total;
    } else {
        for (int expert = lane; expert < experts; expert += 32) scores[expert] = 1.0f / (1.0f + expf(-scores[expert]));
    }
    for (int expert = lane; expert < experts; expert += 32) choice[expert] = scores[expert] + (correction ? correction[expert] : 0.0f);
    __syncwarp();
    if (groups > 1) {
        const int size = experts / groups;
        for (int group = lane; group < groups; group += 32) {
            float first = -INFINITY, second = -INFINITY;
            for (int expert = group * size; expert < (group + 1) * size; ++expert) {
                const float value = choice[expert];
                if (value > first) { second = first; first = value; }
                else if (value > second) second = value;
            }
            ranks[group] = size > 1 ? first + second : first;
        }
        __syncwarp();
        // A group stays if fewer than `keep` groups stand before it.
        for (int expert = lane; expert < experts; expert += 32) {
            const int mine = expert / size;
            int before = 0;
            for (int group = 0; group < groups; ++group) before += ranks[group] > ranks[mine] || (ranks[group] == ranks[mine] && group < mine);
            if (before >= keep) choice[expert] = -INFINITY;
        }
        __syncwarp();
    }
    float total = 0.0f;
    for (int place = 0; place < top; ++place) {
        float best = -INFINITY;
        int best_expert = 0x7fffffff;
        for (int expert = lane; expert < experts; expert += 32) {
            const float value = choice[expert];
            if (value > best) { best = value; best_expert = expert; }   // ascending scan: the lowest index among equals stays
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            const float other = __shfl_xor_sync(0xffffffffu, best, offset);
            const int other_expert = __shfl_xor_sync(0xffffffffu, best_expert, offset);
            if (other > best || (other == best && other_expert < best_expert)) { best = other; best_expert = other_expert; }
        }
        if (best_expert >= experts) best_expert = place;     // only rows of NaN come here
        if (lane == 0) {
            chosen[static_cast<size_t>(token) * top + place] = best_expert;
            weights[static_cast<size_t>(token) * top + place] = scores[best_expert];
            choice[best_expert] = -INFINITY;
        }
        total += scores[best_expert];
        __syncwarp();
    }
    if ((renormalize || scale != 1.0f) && lane == 0)
        for (int place = 0; place < top; ++place) {
            float* weight = weights + static_cast<size_t>(token) * top + place;
            *weight = (renormalize ? *weight / (total + 1e-20f) : *weight) * scale;
        }
}

// A block scores `kRows` tokens, so that a router row is read once for all of them; a warp per token then chooses.
template <typename T, int kRows>
__global__ void __launch_bounds__(kRows == 1 ? 1024 : kThreads)
moe_route_kernel(const T* __restrict__ hidden, const float* __restrict__ router, const float* __restrict__ logit_bias, const float* __restrict__ correction,
                 const float* __restrict__ shared_gate_weight, int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ shared_gate,
                 int tokens, int width, int experts, int top, int softmax, int renormalize, int groups, int keep, float scale) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ __align__(16) float shared[];
    const int pitch = (width + 3) & ~3, per_token = 2 * experts + groups;
    const int first = blockIdx.x * kRows, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int count = min(kRows, tokens - first);
    float* numbers = shared + kRows * pitch;      // per token: scores [experts], what is chosen by [experts], the groups' ranks [groups]
    for (int row = 0; row < kRows; ++row) stage_row(hidden + static_cast<size_t>(first + min(row, count - 1)) * width, shared + row * pitch, width);
    __syncthreads();
    for (int expert = warp; expert < experts; expert += warps) {
        float z[kRows];
        warp_dot_rows<kRows>(router + static_cast<size_t>(expert) * width, shared, pitch, width, lane, z);
        if (lane == 0)
#pragma unroll
            for (int row = 0; row < kRows; ++row) numbers[row * per_token + expert] = z[row] + (logit_bias ? logit_bias[expert] : 0.0f);
    }
    if (shared_gate_weight && warp == warps - 1) {
        float z[kRows];
        warp_dot_rows<kRows>(shared_gate_weight, shared, pitch, width, lane, z);
        if (lane == 0)
#pragma unroll
            for (int row = 0; row < kRows; ++row)
                if (row < count) shared_gate[first + row] = 1.0f / (1.0f + expf(-z[row]));
    }
    __syncthreads();
    if (warp >= count) return;
    choose_experts(numbers + warp * per_token, first + warp, lane, correction, chosen, weights, experts, top, softmax, renormalize, groups, keep, scale);
}

// Prompts: a block scores 16 tokens on the tensor cores, 64 experts at a time.  Bound above by the router's rows, which every block reads (with four tokens to
// a block, 2,048 tokens of 64 experts of 2,048 columns were 268 MB through L2 and 56 us; here 67 MB and 22 us) and cuts into three bfloat16 pieces; a bfloat16
// activation is one piece (three products, exact but for the sums), a 32-bit one three (six products).  A warp takes 32 columns in turn; their
// sums leave the tensor core after each (the large pieces' product by product) and meet in shared memory, two by two.
// Its time hardly depends on the number of tokens and is that of 64 experts where there are fewer; which kernel a call takes: `by_tile`.
constexpr int kTileTokens = 16, kTileExperts = 64;

__device__ __forceinline__ void cut_pair(float x, float y, uint32_t* pieces, int apart) {      // cut off, not rounded: the three pieces add up exactly
#pragma unroll
    for (int p = 0; p < chunk::kPieces; ++p) {
        pieces[p * apart] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
        x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
        y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
moe_route_tile_kernel(const T* __restrict__ hidden, const float* __restrict__ router, const float* __restrict__ logit_bias, const float* __restrict__ correction,
                      const float* __restrict__ shared_gate_weight, int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ shared_gate,
                      int tokens, int width, int experts, int top, int softmax, int renormalize, int groups, int keep, float scale) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ __align__(16) float shared[];
    constexpr int kSums = kTileExperts * (kTileTokens + 1), kXPieces = sizeof(T) == 2 ? 1 : chunk::kPieces;
    float* numbers = shared + kWarps * kSums;
    const int per_token = 2 * experts + groups;
    const int first = blockIdx.x * kTileTokens, count = min(kTileTokens, tokens - first), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const T* rows[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) rows[j] = hidden + static_cast<size_t>(first + min(j * 8 + g, count - 1)) * width;
    const int chunks = width / 32;
    for (int base = 0; base < experts; base += kTileExperts) {
        float sums[4][2][4] = {};
        float4 ahead[4][4];      // the next chunk's router rows g and g + 8 of each 16, eight columns each
        auto load = [&](int chunk) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float* row = router + static_cast<size_t>(min(base + m * 16 + half * 8 + g, experts - 1)) * width + chunk * 32 + t * 8;
                    ahead[m][2 * half] = __ldg(reinterpret_cast<const float4*>(row));
                    ahead[m][2 * half + 1] = __ldg(reinterpret_cast<const float4*>(row + 4));
                }
        };
        if (warp < chunks) load(warp);
        for (int at = warp; at < chunks; at += kWarps) {
            uint32_t x[2][kXPieces * 4];      // eight columns of this lane's tokens in each piece
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if constexpr (sizeof(T) == 2) {
                    *reinterpret_cast<uint4*>(x[j]) = *reinterpret_cast<const uint4*>(rows[j] + at * 32 + t * 8);
                } else {
                    const float4 low = *reinterpret_cast<const float4*>(rows[j] + at * 32 + t * 8), high = *reinterpret_cast<const float4*>(rows[j] + at * 32 + t * 8 + 4);
                    cut_pair(low.x, low.y, x[j], 4); cut_pair(low.z, low.w, x[j] + 1, 4);
                    cut_pair(high.x, high.y, x[j] + 2, 4); cut_pair(high.z, high.w, x[j] + 3, 4);
                }
            }
            float4 now[4][4];
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int i = 0; i < 4; ++i) now[m][i] = ahead[m][i];
            if (at + kWarps < chunks) load(at + kWarps);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                uint32_t low[chunk::kPieces * 4], high[chunk::kPieces * 4];      // rows g and g + 8
                cut_pair(now[m][0].x, now[m][0].y, low, 4); cut_pair(now[m][0].z, now[m][0].w, low + 1, 4);
                cut_pair(now[m][1].x, now[m][1].y, low + 2, 4); cut_pair(now[m][1].z, now[m][1].w, low + 3, 4);
                cut_pair(now[m][2].x, now[m][2].y, high, 4); cut_pair(now[m][2].z, now[m][2].w, high + 1, 4);
                cut_pair(now[m][3].x, now[m][3].y, high + 2, 4); cut_pair(now[m][3].z, now[m][3].w, high + 3, 4);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float small[4] = {}, first[4] = {}, second[4] = {};      // the large pieces' products one by one: the tensor core cuts its sums off
#pragma unroll
                    for (int order = kXPieces == 1 ? chunk::kPieces - 1 : chunk::kPieces; order > 0; --order)      // of two cut numbers also the products that lie 2^-24 below
#pragma unroll
                        for (int q = 0; q < kXPieces; ++q) {
                            const int p = order - q;
                            if (p < 0 || p >= chunk::kPieces) continue;
                            chunk::multiply(small, {low[p * 4], high[p * 4], low[p * 4 + 1], high[p * 4 + 1]}, x[j][q * 4], x[j][q * 4 + 1]);
                            chunk::multiply(small, {low[p * 4 + 2], high[p * 4 + 2], low[p * 4 + 3], high[p * 4 + 3]}, x[j][q * 4 + 2], x[j][q * 4 + 3]);
                        }
                    chunk::multiply(first, {low[0], high[0], low[1], high[1]}, x[j][0], x[j][1]);
                    chunk::multiply(second, {low[2], high[2], low[3], high[3]}, x[j][2], x[j][3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) sums[m][j][i] += (first[i] + second[i]) + small[i];
                }
            }
        }
        float* own = shared + warp * kSums;      // [expert][token]
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) own[(m * 16 + i / 2 * 8 + g) * (kTileTokens + 1) + j * 8 + 2 * t + i % 2] = sums[m][j][i];
        __syncthreads();
        for (int item = threadIdx.x; item < kTileExperts * kTileTokens; item += kThreads) {
            const int expert = base + item / kTileTokens, token = item % kTileTokens;
            if (expert >= experts) break;
            float part[kWarps];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) part[w] = shared[w * kSums + item / kTileTokens * (kTileTokens + 1) + token];
#pragma unroll
            for (int apart = kWarps / 2; apart > 0; apart /= 2)
#pragma unroll
                for (int w = 0; w < apart; ++w) part[w] += part[w + apart];
            float z = part[0];
            if (!isfinite(z)) {      // pieces of an infinite or very large number are NaN where the plain sum need not be
                z = 0.0f;
                const T* x = hidden + static_cast<size_t>(first + min(token, count - 1)) * width;
                for (int column = 0; column < width; ++column) z = fmaf(router[static_cast<size_t>(expert) * width + column], to_float(x[column]), z);
            }
            numbers[token * per_token + expert] = z + (logit_bias ? logit_bias[expert] : 0.0f);
        }
        __syncthreads();
    }
    for (int row = warp; row < count; row += kWarps) {
        if (shared_gate_weight) {
            const T* x = hidden + static_cast<size_t>(first + row) * width;
            float part[4] = {};
            for (int column = lane * 4; column < width; column += 128) {
                const float4 w = *reinterpret_cast<const float4*>(shared_gate_weight + column);
                part[0] = fmaf(w.x, to_float(x[column]), part[0]);
                part[1] = fmaf(w.y, to_float(x[column + 1]), part[1]);
                part[2] = fmaf(w.z, to_float(x[column + 2]), part[2]);
                part[3] = fmaf(w.w, to_float(x[column + 3]), part[3]);
            }
            const float z = warp_sum((part[0] + part[1]) + (part[2] + part[3]));
            if (lane == 0) shared_gate[first + row] = 1.0f / (1.0f + expf(-z));
        }
        choose_experts(numbers + row * per_token, first + row, lane, correction, chosen, weights, experts, top, softmax, renormalize, groups, keep, scale);
    }
}

// grid (token-place pairs, feature tiles).  gate_up: [experts, 2 * inner, width], gate rows first.
template <typename T>
__global__ void __launch_bounds__(kThreads)
moe_gate_up_kernel(const T* __restrict__ hidden, const T* __restrict__ gate_up, const int* __restrict__ chosen, const float* __restrict__ input_weights,
                   T* __restrict__ inner_out, int width, int inner, int top, int features_per_block, int interleave, int real_experts, float limit) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ __align__(16) float row[];
    const int pair = blockIdx.x, token = pair / top, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (chosen[pair] >= real_experts) return;      // an identity expert has no inner features
    stage_row(hidden + static_cast<size_t>(token) * width, row, width);
    __syncthreads();
    const T* weights = gate_up + static_cast<size_t>(chosen[pair]) * 2 * inner * width;
    // A weight on the expert's input: both products are linear in the row, so the weight multiplies their 32-bit sums.
    const float input_weight = input_weights ? input_weights[pair] : 1.0f;
    const int begin = blockIdx.y * features_per_block, end = min(inner, begin + features_per_block);
    for (int feature = begin + warp; feature < end; feature += kWarps) {
        // Plain: gate rows, then up rows.  Interleaved: groups of `interleave` gate rows, each followed by its up rows.
        const int gate_row = interleave ? feature / interleave * 2 * interleave + feature % interleave : feature;
        const int up_row = interleave ? gate_row + interleave : inner + feature;
        float gate, up;
        warp_dot_pair(weights + static_cast<size_t>(gate_row) * width, row, weights + static_cast<size_t>(up_row) * width, row, width, lane, gate, up);
        gate *= input_weight;
        up *= input_weight;
        if (lane == 0)
            inner_out[static_cast<size_t>(pair) * inner + feature] = from_float<T>(limit > 0.0f ? clamped_gate_exact(gate, up, limit) : gate / (1.0f + expf(-gate)) * up);
    }
}

// grid (tokens, feature tiles).  down: [experts, width, inner].
template <typename T>
__global__ void __launch_bounds__(kThreads)
moe_down_kernel(const T* __restrict__ inner_in, const T* __restrict__ down, const int* __restrict__ chosen, const float* __restrict__ weights,
                const T* __restrict__ shared_out, const float* __restrict__ shared_gate, float* __restrict__ out, int width, int inner, int top,
                int features_per_block, const T* __restrict__ hidden, int real_experts) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ __align__(16) float rows[];     // [top][inner]
    const int token = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* source = inner_in + static_cast<size_t>(token) * top * inner;
    if (!hidden) {                                   // without identity experts every place was written
        stage_row(source, rows, top * inner);
    } else {
        for (int item = threadIdx.x; item < top * inner; item += blockDim.x)      // an identity expert's place was never written: nothing of it is read
            rows[item] = chosen[static_cast<size_t>(token) * top + item / inner] < real_experts ? to_float(source[item]) : 0.0f;
    }
    __syncthreads();
    const int begin = blockIdx.y * features_per_block, end = min(width, begin + features_per_block);
    for (int feature = begin + warp; feature < end; feature += kWarps) {
        float sum = 0.0f;
        int place = 0;
        // What one place adds: its expert's row against the place's inner features, or the token's own feature for an identity expert.
        auto alone = [&](int at) {
            const int expert = chosen[static_cast<size_t>(token) * top + at];
            if (expert >= real_experts) return hidden ? to_float(hidden[static_cast<size_t>(token) * width + feature]) : 0.0f;
            return warp_dot(down + (static_cast<size_t>(expert) * width + feature) * inner, rows + at * inner, inner, lane);
        };
        for (; place + 1 < top; place += 2) {     // two places at a time, summed in place order
            const int e0 = chosen[static_cast<size_t>(token) * top + place], e1 = chosen[static_cast<size_t>(token) * top + place + 1];
            float a, b;
            if (e0 < real_experts && e1 < real_experts) {
                const T* first = down + (static_cast<size_t>(e0) * width + feature) * inner;
                const T* second = down + (static_cast<size_t>(e1) * width + feature) * inner;
                warp_dot_pair(first, rows + place * inner, second, rows + (place + 1) * inner, inner, lane, a, b);
            } else {
                a = alone(place);
                b = alone(place + 1);
            }
            sum = fmaf(weights ? weights[static_cast<size_t>(token) * top + place] : 1.0f, a, sum);
            sum = fmaf(weights ? weights[static_cast<size_t>(token) * top + place + 1] : 1.0f, b, sum);
        }
        if (place < top) sum = fmaf(weights ? weights[static_cast<size_t>(token) * top + place] : 1.0f, alone(place), sum);
        if (lane == 0) {
            if (shared_out) sum += (shared_gate ? shared_gate[token] : 1.0f) * to_float(shared_out[static_cast<size_t>(token) * width + feature]);
            out[static_cast<size_t>(token) * width + feature] = sum;
        }
    }
}

// ---- bfloat16 experts of few tokens: every chosen expert's weights streamed once ------------------------------------------
// The kernels above read an expert's rows again for each pair that chose it, through L2, and a warp's chain of loads ends with every row; here the
// pairs of an expert are the columns of mma.sync products whose 16 rows are weight rows (up to 32 pairs at a time), so each
// chosen expert is read once.  Bound by that stream.  The blocks stay, one to an SM: each sorts the pairs by expert for itself (a few hundred
// numbers), and each of its 16 warps takes items of work of its own, 16 rows of one expert against its pairs: no warp waits for another.  The
// weights go through lane-private slots of shared memory by cp.async, spans of 128 columns asked for ahead and across the ends of items (the
// fragment order is gemm_skinny.cu's).  A warp begins its rows at a span of its own and goes around: where all warps began at column 0, their addresses lay whole
// rows apart and met in a few memory channels (4.0 TB/s; 5.3 now; items shared by four warps or by the whole block, which then meet over their sums, 4.0 and 2.6).
// So the order of a row's sums depends on what the other tokens of the step chose, as the compensated sums' last bits then do (1e-8); the same step gives the same bits.
//   Gated: rows come in groups of 8 gate rows and their 8 up rows (`interleave` 8); out [pairs, N / 2] = silu(gate) * up or its clamped form.
//   else:  out [pairs, N] in 32-bit, unweighted; moe_combine_kernel sums a token's places.
// Both products and the sum, experts of 1,408 x 2,048, 6 of 64 a token, in us, before (kernels above) -> now: 8 tokens 147 -> 117, 16 265 -> 156, 32 476 -> 196,
// 64 825 -> 213, 200 2,416 -> 307; 704 x 1,024: 8 tokens 51.6 -> 45.4, 32 148 -> 66.
constexpr int kStreamWarps = 16, kStreamThreads = kStreamWarps * 32, kStreamDepth = 2, kStreamPairs = 32;
constexpr int kStreamSpan = 128, kStreamPieces = kStreamSpan / 8, kStreamSlot = 16 * kStreamPieces;      // columns that a warp asks for at once; 16-byte pieces of a row, and of the 16
constexpr int kStreamMostPairs = 4096, kStreamMostExperts = 512;

struct StreamList {      // behind the rings; each chosen expert's pairs in groups of up to kStreamPairs
    int groups;
    int expert[kStreamMostExperts + kStreamMostPairs / kStreamPairs];
    int first[kStreamMostExperts + kStreamMostPairs / kStreamPairs + 1];      // of a group's pairs in `order`
    int cursor[kStreamMostExperts];
    int order[kStreamMostPairs];
};
constexpr int kStreamShared = kStreamWarps * kStreamDepth * kStreamSlot * 16 + static_cast<int>(sizeof(StreamList));
static_assert(kStreamShared <= 227 * 1024, "rings and list fit an SM");

__device__ __forceinline__ void stream_copy(void* target, const void* source, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(target))), "l"(source), "r"(real ? 16 : 0) : "memory");
}

template <bool Gated>
__global__ void __launch_bounds__(kStreamThreads, 1)
moe_stream_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, const int* __restrict__ chosen, const float* __restrict__ input_weights, void* __restrict__ out,
                  int pairs, int real_experts, int N, int K, int top, float limit) {
    extern __shared__ __align__(16) uint8_t stream_shared[];
    uint4* rings = reinterpret_cast<uint4*>(stream_shared);
    StreamList& list = *reinterpret_cast<StreamList*>(stream_shared + kStreamWarps * kStreamDepth * kStreamSlot * 16);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    // The router's choice: the gated kernel waits for it before it lets the next kernel start, so for that one (the down product) it lies there from the start.
    if (Gated) grid_dependency_wait();
    grid_dependents_launch();
    // A warp counts, and later lists, an expert's pairs in their order: every block must cut an expert's pairs into the same groups.
    for (int expert = warp; expert < real_experts; expert += kStreamWarps) {
        int count = 0;
        for (int base = 0; base < pairs; base += 32) count += __popc(__ballot_sync(0xffffffffu, base + lane < pairs && chosen[base + lane] == expert));
        if (lane == 0) list.cursor[expert] = count;
    }
    __syncthreads();
    if (warp == 0) {
        int pairs_before = 0, groups_before = 0;
        for (int base = 0; base < real_experts; base += 32) {
            const int expert = base + lane, count = expert < real_experts ? list.cursor[expert] : 0, groups = (count + kStreamPairs - 1) / kStreamPairs;
            int pair_sum = count, group_sum = groups;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const int other_pairs = __shfl_up_sync(0xffffffffu, pair_sum, offset), other_groups = __shfl_up_sync(0xffffffffu, group_sum, offset);
                if (lane >= offset) pair_sum += other_pairs, group_sum += other_groups;
            }
            const int first = pairs_before + pair_sum - count;
            for (int i = 0; i < groups; ++i) {
                list.expert[groups_before + group_sum - groups + i] = expert;
                list.first[groups_before + group_sum - groups + i] = first + i * kStreamPairs;
            }
            if (expert < real_experts) list.cursor[expert] = first;
            pairs_before += __shfl_sync(0xffffffffu, pair_sum, 31);
            groups_before += __shfl_sync(0xffffffffu, group_sum, 31);
        }
        if (lane == 0) {
            list.groups = groups_before;
            list.first[groups_before] = pairs_before;
        }
    }
    __syncthreads();
    for (int expert = warp; expert < real_experts; expert += kStreamWarps) {
        int place = list.cursor[expert];
        for (int base = 0; base < pairs; base += 32) {
            const bool mine = base + lane < pairs && chosen[base + lane] == expert;
            const unsigned all = __ballot_sync(0xffffffffu, mine);
            if (mine) list.order[place + __popc(all & ((1u << lane) - 1u))] = base + lane;
            place += __popc(all);
        }
    }
    __syncthreads();

    // Neighbouring warps take neighbouring rows, neighbouring blocks' warps those behind them.
    const int tiles = N / 16, items = list.groups * tiles, spans = (K + kStreamSpan - 1) / kStreamSpan, stride = gridDim.x * kStreamWarps;
    uint4* ring = rings + static_cast<size_t>(warp) * kStreamDepth * kStreamSlot;      // [depth][row][piece]
    const int turn = (blockIdx.x * kStreamWarps + warp) % spans;
    int ahead_item = blockIdx.x * kStreamWarps + warp, ahead_span = 0, issued = 0;
    const bf16* ahead_row = nullptr;
    // A copy instruction is whole runs of a row, kStreamSpan elements each; odd rows' halves of 128 bytes change places so that eight lanes read 128 different bytes.
    auto issue = [&]() {
        if (ahead_item < items) {
            if (ahead_span == 0) ahead_row = w + (static_cast<size_t>(list.expert[ahead_item / tiles]) * N + ahead_item % tiles * 16) * K;
            const int piece = lane % kStreamPieces, k = (ahead_span + turn < spans ? ahead_span + turn : ahead_span + turn - spans) * kStreamSpan + piece * 8;      // K % 8 == 0: a piece is whole or absent (zeros)
            uint4* slot = ring + issued % kStreamDepth * kStreamSlot;
#pragma unroll
            for (int i = 0; i < kStreamSlot / 32; ++i) {
                const int row = i * (32 / kStreamPieces) + lane / kStreamPieces;
                stream_copy(slot + row * kStreamPieces + (piece ^ ((row & 1) << 2)), ahead_row + static_cast<size_t>(row) * K + (k < K ? k : 0), k < K);
            }
            if (++ahead_span == spans) ahead_span = 0, ahead_item += stride;
        }
        ++issued;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kStreamDepth - 1; ++i) issue();
    if (!Gated) grid_dependency_wait();      // what the products read and write
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    int used = 0;
    for (int item = blockIdx.x * kStreamWarps + warp; item < items; item += stride) {
        const int group = item / tiles, tile = item % tiles, first = list.first[group];
        const int count = min(kStreamPairs, list.first[group + 1] - first), blocks = (count + 7) / 8;
        const bf16* rows[kStreamPairs / 8];
#pragma unroll
        for (int j = 0; j < kStreamPairs / 8; ++j) {
            const int pair = list.order[first + min(j * 8 + g, count - 1)];      // columns behind the last repeat it; their sums are not stored
            rows[j] = x + static_cast<size_t>(Gated ? pair / top : pair) * K;
        }
        float rest[kStreamPairs / 8][4] = {}, sums[kStreamPairs / 8][4] = {};      // {D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1]}, D[weight row][pair of block j]
        for (int at = 0; at < spans; ++at) {
            const int span = at + turn < spans ? at + turn : at + turn - spans;
            asm volatile("cp.async.wait_group %0;" ::"n"(kStreamDepth - 2) : "memory");      // this span has landed,
            __syncwarp();                                                                    // for every lane, and every lane is done with the slot that is written next
            issue();
            const uint4* slot = ring + used++ % kStreamDepth * kStreamSlot + g * kStreamPieces;
            float acc[kStreamPairs / 8][4] = {};
#pragma unroll 1
            for (int part = 0; part < kStreamSpan / 64; ++part) {
                const int k_first = span * kStreamSpan + part * 64 + t * 8, k_second = k_first + 32;
                if (span * kStreamSpan + part * 64 >= K) break;
                uint4 x1[kStreamPairs / 8], x2[kStreamPairs / 8];
#pragma unroll
                for (int j = 0; j < kStreamPairs / 8; ++j)
                    if (j < blocks) {
                        x1[j] = k_first < K ? __ldg(reinterpret_cast<const uint4*>(rows[j] + k_first)) : zero;
                        x2[j] = k_second < K ? __ldg(reinterpret_cast<const uint4*>(rows[j] + k_second)) : zero;
                    }
                const int first_piece = part * 8 + (t ^ ((g & 1) << 2)), second_piece = first_piece ^ 4;
                const uint4 lo1 = slot[first_piece], hi1 = slot[first_piece + 8 * kStreamPieces], lo2 = slot[second_piece], hi2 = slot[second_piece + 8 * kStreamPieces];
#pragma unroll
                for (int j = 0; j < kStreamPairs / 8; ++j)
                    if (j < blocks) {
                        // One instruction to a chain (the tensor core cuts its sums off), joined two by two.
                        float chain[4][4] = {};
                        chunk::multiply(chain[0], {lo1.x, hi1.x, lo1.y, hi1.y}, x1[j].x, x1[j].y);
                        chunk::multiply(chain[1], {lo1.z, hi1.z, lo1.w, hi1.w}, x1[j].z, x1[j].w);
                        chunk::multiply(chain[2], {lo2.x, hi2.x, lo2.y, hi2.y}, x2[j].x, x2[j].y);
                        chunk::multiply(chain[3], {lo2.z, hi2.z, lo2.w, hi2.w}, x2[j].z, x2[j].w);
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[j][i] += (chain[0][i] + chain[1][i]) + (chain[2][i] + chain[3][i]);
                    }
            }
#pragma unroll
            for (int j = 0; j < kStreamPairs / 8; ++j)
#pragma unroll
                for (int i = 0; i < 4 && j < blocks; ++i) {      // the spans' sums with what the additions before left over: as near to 64 bits as the kernels above
                    const float more = acc[j][i] + rest[j][i], sum = sums[j][i] + more;
                    rest[j][i] = isfinite(sum) ? more - (sum - sums[j][i]) : 0.0f;      // an infinite sum leaves nothing over (inf - inf) and stays infinite, as there
                    sums[j][i] = sum;
                }
        }
#pragma unroll
        for (int j = 0; j < kStreamPairs / 8; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int column = j * 8 + 2 * t + i;
                if (column >= count) continue;
                const int pair = list.order[first + column];
                if constexpr (Gated) {      // a gate row and its up row lie in one thread
                    const float input_weight = input_weights ? input_weights[pair] : 1.0f, gate = sums[j][i] * input_weight, up = sums[j][2 + i] * input_weight;
                    static_cast<bf16*>(out)[static_cast<size_t>(pair) * (N / 2) + tile * 8 + g] =
                        __float2bfloat16_rn(limit > 0.0f ? clamped_gate_exact(gate, up, limit) : gate / (1.0f + expf(-gate)) * up);
                } else {
                    float* target = static_cast<float*>(out) + static_cast<size_t>(pair) * N + tile * 16 + g;
                    target[0] = sums[j][i];
                    target[8] = sums[j][2 + i];
                }
            }
    }
}

// The (token, place) pairs grouped by expert, by one block: offsets[e] .. offsets[e + 1] are the places of expert e's pairs in
// `order`; position[pair] is where a pair went.  The order inside a group depends on timing; nothing computed from it does.
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int* __restrict__ chosen, int pairs, int experts, int* __restrict__ offsets, int* __restrict__ order, int* __restrict__ position) {
    grid_dependents_launch();
    grid_dependency_wait();
    extern __shared__ int counters[];       // [experts] counts, then [experts] cursors
    int* cursor = counters + experts;
    // A thread's first pairs are loaded together and stay in registers: one round trip to memory, not one for each pair of each of the two passes (12,288 pairs of 64
    // experts 11.0 us so, 9.2 now).  Turns that no thread has a pair for are left out (1,000 pairs 2.2 us one by one, 3.2 with all turns).
    constexpr int kKept = 16;
    int kept[kKept];
#pragma unroll
    for (int i = 0; i < kKept; ++i) {
        const int pair = threadIdx.x + i * blockDim.x;
        if (i * blockDim.x >= pairs) break;
        kept[i] = pair < pairs ? chosen[pair] : -1;
    }
    for (int expert = threadIdx.x; expert < experts; expert += blockDim.x) counters[expert] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kKept; ++i) {
        if (i * blockDim.x >= pairs) break;
        if (kept[i] >= 0) atomicAdd(&counters[kept[i]], 1);
    }
    for (int pair = threadIdx.x + kKept * blockDim.x; pair < pairs; pair += blockDim.x) atomicAdd(&counters[chosen[pair]], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
        int before = 0;
        for (int base = 0; base < experts; base += 32) {
            const int expert = base + threadIdx.x, count = expert < experts ? counters[expert] : 0;
            int sum = count;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, sum, offset);
                if (threadIdx.x >= offset) sum += other;
            }
            if (expert < experts) offsets[expert] = cursor[expert] = before + sum - count;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (threadIdx.x == 0) offsets[experts] = before;
    }
    __syncthreads();
    auto put = [&](int pair, int expert) {
        const int place = atomicAdd(&cursor[expert], 1);
        order[place] = pair;
        position[pair] = place;
    };
#pragma unroll
    for (int i = 0; i < kKept; ++i) {
        if (i * blockDim.x >= pairs) break;
        if (kept[i] >= 0) put(threadIdx.x + i * blockDim.x, kept[i]);
    }
    for (int pair = threadIdx.x + kKept * blockDim.x; pair < pairs; pair += blockDim.x) put(pair, chosen[pair]);
}

// gathered[i] = hidden[order[i] / top] (times input_weights[order[i]], if given): the rows of each expert's tokens side by side.
template <typename T>
__global__ void moe_gather_kernel(const T* __restrict__ hidden, const int* __restrict__ order, const float* __restrict__ input_weights, T* __restrict__ gathered,
                                  int width, int top) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int pair = order[blockIdx.x];
    const T* source = hidden + static_cast<size_t>(pair / top) * width;
    T* target = gathered + static_cast<size_t>(blockIdx.x) * width;
    constexpr int kPiece = 16 / sizeof(T);
    if (!input_weights && width % kPiece == 0 && ((reinterpret_cast<uintptr_t>(hidden) | reinterpret_cast<uintptr_t>(gathered)) & 15) == 0) {
        for (int column = threadIdx.x * kPiece; column < width; column += blockDim.x * kPiece)
            *reinterpret_cast<uint4*>(target + column) = *reinterpret_cast<const uint4*>(source + column);
    } else if (input_weights) {
        const float weight = input_weights[pair];
        for (int column = threadIdx.x; column < width; column += blockDim.x) target[column] = from_float<T>(weight * to_float(source[column]));
    } else {
        for (int column = threadIdx.x; column < width; column += blockDim.x) target[column] = source[column];
    }
}

// out[token] = sum over places of weight * rows[position[token, place]] + shared_gate * shared[token], in place order; without positions the rows lie pair by pair.
// Bound by the rows' bytes: 2,048 tokens of 6 places of 2,048 columns (125 MB) 26.7 us with one place's row after another, 24.7 with six on their way.  Up to five places the
// compiler's own order of one row after another is the faster one (us, six at once against it: 3,000 x 1 13.8 against 7.5, 20,000 x 2 112 against 82, 25,000 x 4 168 against 158), and
// eight at once for 7 and 8 (375 x 8 6.0, 6.7 with six).  `kPositions`: whether there are, known when the rows are read one after another.
template <typename T, int kAtOnce, bool kPositions>
__global__ void moe_combine_kernel(const float* __restrict__ rows, const int* __restrict__ position, const float* __restrict__ weights,
                                   const T* __restrict__ shared_out, const float* __restrict__ shared_gate, float* __restrict__ out, int width, int top,
                                   const int* __restrict__ chosen, const T* __restrict__ hidden, int real_experts) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int token = blockIdx.x;
    if (!chosen && width % 4 == 0 && ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out)) & 15) == 0
        && (reinterpret_cast<uintptr_t>(shared_out) & (4 * sizeof(T) - 1)) == 0) {
        const float shared_weight = shared_out && shared_gate ? shared_gate[token] : 1.0f;
        for (int column = threadIdx.x * 4; column < width; column += blockDim.x * 4) {      // the same sums, four columns at a time
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            auto row_of = [&](size_t pair) { return *reinterpret_cast<const float4*>(rows + ((kAtOnce == 1 ? kPositions : position != nullptr) ? static_cast<size_t>(position[pair]) : pair) * width + column); };
            if constexpr (kAtOnce == 1) {
                for (int place = 0; place < top; ++place) {
                    const size_t pair = static_cast<size_t>(token) * top + place;
                    const float weight = weights ? weights[pair] : 1.0f;
                    const float4 row = row_of(pair);
                    sum.x = fmaf(weight, row.x, sum.x); sum.y = fmaf(weight, row.y, sum.y);
                    sum.z = fmaf(weight, row.z, sum.z); sum.w = fmaf(weight, row.w, sum.w);
                }
            } else {
                for (int first = 0; first < top; first += kAtOnce) {      // the rows of several places travel together; they are added in place order
                    float weight[kAtOnce];
                    float4 row[kAtOnce];
#pragma unroll
                    for (int i = 0; i < kAtOnce; ++i) {
                        const size_t pair = static_cast<size_t>(token) * top + min(first + i, top - 1);
                        weight[i] = weights ? weights[pair] : 1.0f;
                        if (first + i < top) row[i] = row_of(pair);
                    }
#pragma unroll
                    for (int i = 0; i < kAtOnce; ++i) {
                        if (first + i >= top) break;
                        sum.x = fmaf(weight[i], row[i].x, sum.x); sum.y = fmaf(weight[i], row[i].y, sum.y);
                        sum.z = fmaf(weight[i], row[i].z, sum.z); sum.w = fmaf(weight[i], row[i].w, sum.w);
                    }
                }
            }
            if (shared_out) {
                const T* source = shared_out + static_cast<size_t>(token) * width + column;
                float x[4];
                if constexpr (sizeof(T) == 2) {
                    const uint2 raw = *reinterpret_cast<const uint2*>(source);
                    x[0] = __uint_as_float(raw.x << 16); x[1] = __uint_as_float(raw.x & 0xffff0000u);
                    x[2] = __uint_as_float(raw.y << 16); x[3] = __uint_as_float(raw.y & 0xffff0000u);
                } else {
                    const float4 raw = *reinterpret_cast<const float4*>(source);
                    x[0] = raw.x; x[1] = raw.y; x[2] = raw.z; x[3] = raw.w;
                }
                sum.x += shared_weight * x[0]; sum.y += shared_weight * x[1];
                sum.z += shared_weight * x[2]; sum.w += shared_weight * x[3];
            }
            *reinterpret_cast<float4*>(out + static_cast<size_t>(token) * width + column) = sum;
        }
        return;
    }
    for (int column = threadIdx.x; column < width; column += blockDim.x) {
        float sum = 0.0f;
        for (int place = 0; place < top; ++place) {
            const size_t pair = static_cast<size_t>(token) * top + place;
            const bool identity = chosen && chosen[pair] >= real_experts;      // such a pair's row was never computed
            const float row = identity ? to_float(hidden[static_cast<size_t>(token) * width + column]) : rows[(position ? static_cast<size_t>(position[pair]) : pair) * width + column];
            sum = fmaf(weights ? weights[pair] : 1.0f, row, sum);
        }
        if (shared_out) sum += (shared_gate ? shared_gate[token] : 1.0f) * to_float(shared_out[static_cast<size_t>(token) * width + column]);
        out[static_cast<size_t>(token) * width + column] = sum;
    }
}

template <typename T>
void launch_combine(const float* rows, const int* position, const float* weights, const void* shared_out, const float* shared_gate, float* out, int tokens, int width, int top,
                    const int* chosen, const void* hidden, int real_experts, cudaStream_t s) {
    auto* const kernel = top <= 5 ? (position ? moe_combine_kernel<T, 1, true> : moe_combine_kernel<T, 1, false>)
                         : top == 7 || top == 8 ? moe_combine_kernel<T, 8, false> : moe_combine_kernel<T, 6, false>;
    tau_launch(kernel, dim3(tokens), dim3(kThreads), 0, s, rows, position, weights, static_cast<const T*>(shared_out), shared_gate, out,
               width, top, chosen, static_cast<const T*>(hidden), real_experts);
}

// Whether the tiles score a router faster than a block for each token (with up to 4 * 148 tokens) or for four (us, the others against the tiles).  bfloat16 tokens of 64 experts and
// more from the first wave of the others' 256-thread blocks on: the kernels alone are as fast or a little slower there (64 of 2,048 columns: 256 tokens 22.7 against 29, 500 29.4 against
// 29.5, 2,048 60 against 33; 256 of 2,048: 300 94 against 82), but the tiles' few blocks leave SMs to the kernel behind (a layer of 64 experts of 2,048: 250 tokens 278
// against 297, 350 304 against 299, 600 337 against 319; of 1,024: 250 134 against 141, 500 149 against 143).  32-bit tokens take twice the products (256 of 2,048: 300 92
// against 109, 600 136 against 112).  32 experts of 2,048: 600 21 against 23, 1,000 30 against 23; 64 of 512: 600 20.5 against 23, 1,000 25.9 against 23.2.  Few experts never fill the
// tiles (8 of 4,096: 300 9.6 against 28, 4,096 44 against 55; 24 of 2,048: 1,000 25 against 24), nor do narrow ones (64 of 256: 1,000 20.6 against 21).
bool by_tile(int tokens, int experts, int width, bool bits16) {
    const long long work = static_cast<long long>(experts) * width;
    if (experts < 32 || work < 1 << 15) return false;
    if (experts < 64 || work < (bits16 ? 1 << 16 : 1 << 17)) return tokens >= 1000;
    return tokens >= (bits16 ? 2 * 148 + 1 : 4 * 148);
}

template <typename T>
int launch_all(int what, const void* a, const void* b, const void* c, const void* d, const void* e, const void* f, void* o1, void* o2, void* o3,
               int tokens, int width, int inner, int experts, int top, int flag_a, int flag_b, cudaStream_t s, const void* g = nullptr, float constant = 1.0f,
               int groups = 1, int keep = 1) {
    if (what == 0) {
        // `inner`: whether the tiles score the router (1, 0 or -1: `by_tile`).  Few tokens: one to a block with many warps, since its rows of the router are a chain of loads; many: four to a block.
        const size_t one = (static_cast<size_t>((width + 3) & ~3) + 2 * experts + groups) * sizeof(float);
        const size_t tile = (static_cast<size_t>(kWarps) * kTileExperts * (kTileTokens + 1) + static_cast<size_t>(kTileTokens) * (2 * experts + groups)) * sizeof(float);
        if (inner != 0 && (inner > 0 || by_tile(tokens, experts, width, sizeof(T) == 2)) && width % 32 == 0 && tile <= 200 * 1024
            && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(d)) & 15) == 0) {
            if (tile > 48 * 1024 && cudaFuncSetAttribute(moe_route_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tile)) != cudaSuccess)
                return cudaErrorInvalidValue;
            tau_launch(moe_route_tile_kernel<T>, dim3((tokens + kTileTokens - 1) / kTileTokens), dim3(kThreads), tile, s, static_cast<const T*>(a), static_cast<const float*>(b),
                       static_cast<const float*>(e), static_cast<const float*>(c), static_cast<const float*>(d), static_cast<int*>(o1), static_cast<float*>(o2),
                       static_cast<float*>(o3), tokens, width, experts, top, flag_a, flag_b, groups, keep, constant);
            return tau_launch_status();
        }
        const bool four = tokens >= 4 * 148 && 4 * one <= 200 * 1024;
        const size_t bytes = four ? 4 * one : one;
        auto* kernel = four ? moe_route_kernel<T, 4> : moe_route_kernel<T, 1>;
        if (bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess) return cudaErrorInvalidValue;
        tau_launch(kernel, dim3(four ? (tokens + 3) / 4 : tokens), dim3(tokens <= 2 * 148 ? 1024 : kThreads), bytes, s, static_cast<const T*>(a), static_cast<const float*>(b), static_cast<const float*>(e),
                   static_cast<const float*>(c), static_cast<const float*>(d), static_cast<int*>(o1), static_cast<float*>(o2), static_cast<float*>(o3), tokens, width, experts, top, flag_a, flag_b,
                   groups, keep, constant);
    } else if (what == 1) {
        // Few pairs: smaller tiles, so that every SM has blocks (one token of 6 experts of 1,408 features: 90 us in tiles of 64, 76 us in tiles of 16).
        const int per_block = static_cast<long long>(tokens) * top * ((inner + 63) / 64) >= 2 * 148 ? 64 : 16;
        const size_t bytes = static_cast<size_t>(width) * sizeof(float);
        if (bytes > 48 * 1024 && cudaFuncSetAttribute(moe_gate_up_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess)
            return cudaErrorInvalidValue;
        tau_launch(moe_gate_up_kernel<T>, dim3(tokens * top, (inner + per_block - 1) / per_block), dim3(kThreads), bytes, s, static_cast<const T*>(a),
                   static_cast<const T*>(b), static_cast<const int*>(c), static_cast<const float*>(d), static_cast<T*>(o1), width, inner, top, per_block, flag_a, experts,
                   constant);
    } else {
        const int per_block = tokens * ((width + 63) / 64) >= 1024 ? 64 : tokens * ((width + 31) / 32) >= 1024 ? 32 : 16;   // few tokens: smaller tiles, more blocks
        const size_t bytes = static_cast<size_t>(top) * inner * sizeof(float);
        if (bytes > 48 * 1024 && cudaFuncSetAttribute(moe_down_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess)
            return cudaErrorInvalidValue;
        tau_launch(moe_down_kernel<T>, dim3(tokens, (width + per_block - 1) / per_block), dim3(kThreads), bytes, s, static_cast<const T*>(a), static_cast<const T*>(b),
                   static_cast<const int*>(c), static_cast<const float*>(d), static_cast<const T*>(e), static_cast<const float*>(f), static_cast<float*>(o1),
                   width, inner, top, per_block, static_cast<const T*>(g), experts);
    }
    return tau_launch_status();
}

}  // namespace

// `tile`: 1 scores the router in tiles of 16 tokens (where widths and alignment allow), 0 token by token, -1 as is faster.
TAU_EXPORT int tau_moe_route(int dtype, const void* hidden, const float* router, const float* logit_bias, const float* correction, const float* shared_gate_weight, int* chosen,
                             float* weights, float* shared_gate, int tokens, int width, int experts, int top, int softmax, int renormalize, int groups, int keep,
                             float scale, int tile, void* stream) {
    if (tokens <= 0) return 0;
    if (!hidden || !router || !chosen || !weights || width <= 0 || experts <= 0 || top <= 0 || top > experts || (shared_gate_weight && !shared_gate)
        || groups < 1 || experts % groups != 0 || keep < 1 || keep > groups || top > keep * (experts / groups))
        return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TAU_F32) return launch_all<float>(0, hidden, router, correction, shared_gate_weight, logit_bias, nullptr, chosen, weights, shared_gate, tokens, width, tile, experts, top, softmax, renormalize, s, nullptr, scale, groups, keep);
    if (dtype == TAU_BF16) return launch_all<bf16>(0, hidden, router, correction, shared_gate_weight, logit_bias, nullptr, chosen, weights, shared_gate, tokens, width, tile, experts, top, softmax, renormalize, s, nullptr, scale, groups, keep);
    return cudaErrorInvalidValue;
}

// `real_experts`: experts with weights (gate_up holds that many); a pair that chose a higher number is left alone.
TAU_EXPORT int tau_moe_gate_up(int dtype, const void* hidden, const void* gate_up, const int* chosen, const float* input_weights, void* inner_out, int tokens,
                               int width, int inner, int top, int interleave, int real_experts, float limit, void* stream) {
    if (tokens <= 0) return 0;
    if (!hidden || !gate_up || !chosen || !inner_out || width <= 0 || inner <= 0 || top <= 0 || static_cast<long long>(tokens) * top > 0x7fffffff) return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TAU_F32) return launch_all<float>(1, hidden, gate_up, chosen, input_weights, nullptr, nullptr, inner_out, nullptr, nullptr, tokens, width, inner, real_experts, top, interleave, 0, s, nullptr, limit);
    if (dtype == TAU_BF16) return launch_all<bf16>(1, hidden, gate_up, chosen, input_weights, nullptr, nullptr, inner_out, nullptr, nullptr, tokens, width, inner, real_experts, top, interleave, 0, s, nullptr, limit);
    return cudaErrorInvalidValue;
}

TAU_EXPORT int tau_moe_down(int dtype, const void* inner_in, const void* down, const int* chosen, const float* weights, const void* shared_out,
                            const float* shared_gate, float* out, int tokens, int width, int inner, int top, const void* hidden, int real_experts,
                            void* stream) {
    if (tokens <= 0) return 0;
    if (!inner_in || !down || !chosen || !out || width <= 0 || inner <= 0 || top <= 0) return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TAU_F32) return launch_all<float>(2, inner_in, down, chosen, weights, shared_out, shared_gate, out, nullptr, nullptr, tokens, width, inner, real_experts, top, 0, 0, s, hidden);
    if (dtype == TAU_BF16) return launch_all<bf16>(2, inner_in, down, chosen, weights, shared_out, shared_gate, out, nullptr, nullptr, tokens, width, inner, real_experts, top, 0, 0, s, hidden);
    return cudaErrorInvalidValue;
}

// Both products of bfloat16 experts of few tokens by moe_stream_kernel, one behind the other: `hidden` [tokens, width], `gate_up` [experts, 2 inner, width] with
// groups of 8 gate rows and their 8 up rows, `down` [experts, width, inner], `inner_out` [pairs, inner] bfloat16, `rows` [pairs, width] 32-bit, unweighted.
// Width and inner multiples of 16 and at least 256, all on 16 bytes, at most 512 experts with weights and 4,096 pairs.
TAU_EXPORT int tau_moe_stream(const void* hidden, const void* gate_up, const void* down, const int* chosen, const float* input_weights, void* inner_out, void* rows,
                              int pairs, int real_experts, int width, int inner, int top, float limit, void* stream) {
    if (pairs <= 0) return 0;
    if (!hidden || !gate_up || !down || !chosen || !inner_out || !rows || real_experts <= 0 || real_experts > kStreamMostExperts || pairs > kStreamMostPairs || width < 256
        || width % 16 || inner < 256 || inner % 16 || top <= 0
        || ((reinterpret_cast<uintptr_t>(hidden) | reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(down) | reinterpret_cast<uintptr_t>(inner_out)) & 15))
        return cudaErrorInvalidValue;
    static int sms = 0;
    if (!sms) {
        int device = 0, count = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status == cudaSuccess) status = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
        if (status == cudaSuccess) status = cudaFuncSetAttribute(moe_stream_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamShared);
        if (status == cudaSuccess) status = cudaFuncSetAttribute(moe_stream_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamShared);
        if (status != cudaSuccess) return static_cast<int>(status);
        sms = count;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    tau_launch(moe_stream_kernel<true>, dim3(sms), dim3(kStreamThreads), kStreamShared, s, static_cast<const bf16*>(hidden), static_cast<const bf16*>(gate_up), chosen,
               input_weights, inner_out, pairs, real_experts, 2 * inner, width, top, limit);
    const int status = tau_launch_status();
    if (status) return status;
    // Launched right behind the other, which the early reads of `chosen` rest on.
    tau_launch(moe_stream_kernel<false>, dim3(sms), dim3(kStreamThreads), kStreamShared, s, static_cast<const bf16*>(inner_out), static_cast<const bf16*>(down), chosen,
               nullptr, rows, pairs, real_experts, width, inner, top, 0.0f);
    return tau_launch_status();
}

TAU_EXPORT int tau_moe_sort(const int* chosen, int pairs, int experts, int* offsets, int* order, int* position, void* stream) {
    if (pairs <= 0) return 0;
    if (!chosen || !offsets || !order || !position || experts <= 0 || experts > 4096) return cudaErrorInvalidValue;
    tau_launch(moe_sort_kernel, dim3(1), dim3(1024), static_cast<size_t>(2 * experts) * sizeof(int), static_cast<cudaStream_t>(stream), chosen, pairs, experts,
               offsets, order, position);
    return tau_launch_status();
}

TAU_EXPORT int tau_moe_gather(int dtype, const void* hidden, const int* order, const float* input_weights, void* gathered, int pairs, int width, int top,
                              void* stream) {
    if (pairs <= 0) return 0;
    if (!hidden || !order || !gathered || width <= 0 || top <= 0) return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TAU_F32) tau_launch(moe_gather_kernel<float>, dim3(pairs), dim3(kThreads), 0, s, static_cast<const float*>(hidden), order, input_weights, static_cast<float*>(gathered), width, top);
    else if (dtype == TAU_BF16) tau_launch(moe_gather_kernel<bf16>, dim3(pairs), dim3(kThreads), 0, s, static_cast<const bf16*>(hidden), order, input_weights, static_cast<bf16*>(gathered), width, top);
    else return cudaErrorInvalidValue;
    return tau_launch_status();
}

TAU_EXPORT int tau_moe_combine(int dtype, const float* rows, const int* position, const float* weights, const void* shared_out, const float* shared_gate,
                               float* out, int tokens, int width, int top, const int* chosen, const void* hidden, int real_experts, void* stream) {
    if (tokens <= 0) return 0;
    if (!rows || !out || width <= 0 || top <= 0 || (chosen && !hidden)) return cudaErrorInvalidValue;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TAU_F32) launch_combine<float>(rows, position, weights, shared_out, shared_gate, out, tokens, width, top, chosen, hidden, real_experts, s);
    else if (dtype == TAU_BF16) launch_combine<bf16>(rows, position, weights, shared_out, shared_gate, out, tokens, width, top, chosen, hidden, real_experts, s);
    else return cudaErrorInvalidValue;
    return tau_launch_status();
}
