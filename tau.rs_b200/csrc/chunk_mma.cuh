// 32-bit products on the bfloat16 tensor cores, for kernels that walk a sequence chunk by chunk.
//
// A 32-bit number is the sum of three bfloat16 pieces (8 bits of mantissa each: x = h + m + l to 2^-25 of x).  A product of two such numbers is
// the sum of the six piece products whose order is 2^-16 or more; with one operand exact in bfloat16 it is three.  The products of pieces are
// exact in 32-bit.  The tensor core adds to a 32-bit accumulator but cuts the sum off instead of rounding it, an error of one sign that adds up over
// a long chain (measured: 4e-6 of a state after 262 products onto it); so chains are kept to a few products, the small pieces' products have
// accumulators of their own or come first, and what is longer is joined by ordinary additions.
#pragma once
#include "common.cuh"

namespace chunk {

__device__ __forceinline__ uint32_t shared_address(const void* pointer) { return static_cast<uint32_t>(__cvta_generic_to_shared(pointer)); }

// 16 bytes from global to shared memory; zeros where `live` is false (nothing is read then).
__device__ __forceinline__ void copy16(void* target, const void* source, bool live) {
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(shared_address(target)), "l"(source), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kNewer> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kNewer) : "memory"); }

__device__ __forceinline__ void load_matrices(uint32_t (&out)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3]) : "r"(shared_address(row)) : "memory");
}
__device__ __forceinline__ void load_matrices_turned(uint32_t (&out)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3]) : "r"(shared_address(row)) : "memory");
}
__device__ __forceinline__ void load_pair_turned(uint32_t (&out)[2], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(out[0]), "=r"(out[1]) : "r"(shared_address(row)) : "memory");
}
// c += a b: a is 16 x 16 (row), b is 16 x 8 (col), c is 16 x 8.
__device__ __forceinline__ void multiply(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Bulk copies (16-byte aligned, sizes of whole 16 bytes) complete on an mbarrier, which counts their bytes.  They are for whole tiles: a copy costs about
// 80 cycles however small (rows of 256 to 512 bytes one by one took 5 to 8 us a chunk), while cp.async of the same tiles by 256 threads held the
// load/store pipe for 2,200 cycles of a chunk and with it every shared-memory access behind it (4.4 us a chunk).
__device__ __forceinline__ void barrier_init(uint64_t* barrier) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(barrier))); }
__device__ __forceinline__ void barriers_ready() { asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void shared_writes_ready() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }      // before a bulk store reads them
__device__ __forceinline__ void barrier_expect(uint64_t* barrier, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(barrier)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* target, const void* source, int bytes, uint64_t* barrier) {
#ifndef TAU_LOST_COPIES      // the tests of waits that run out: a copy that is never asked for
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared_address(target)), "l"(source), "r"(bytes),
                 "r"(shared_address(barrier)) : "memory");
#endif
}
// A tile from shared to global memory; the thread that stored it waits before it ends.
__device__ __forceinline__ void bulk_store(void* target, const void* source, int bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;" ::"l"(target), "r"(shared_address(source)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_stored() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ int wait_ran_out = 0;   // raised when a wait took longer than the limit (see `barrier_wait`)
#ifndef TAU_WAIT_LIMIT_NS
#define TAU_WAIT_LIMIT_NS 2000000000ull      // the tests of waits that run out compile with a shorter one
#endif
// Waits for the phase with the given parity, within the limit; the whole warp calls it.  When it runs out, `gone` (a number of the block in shared
// memory, zero before) and the library's flag are raised and the warp goes on with whatever is there.  No wait takes long from then on; who asks for
// copies looks at `gone` first and asks for no more; at a barrier that it has anyway, at the latest before it would write a result that others build on,
// the block learns of it, waits for the copies in flight once more (`gone` null) and ends.
// Lanes may see the phase end at different turns of the loop; they meet again before the warp goes on to instructions that want all of them (ldmatrix,
// mma, a block's barrier).
__device__ __forceinline__ bool barrier_try(uint64_t* barrier, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(shared_address(barrier)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __noinline__ void barrier_wait_on(uint64_t* barrier, uint32_t parity, volatile int* gone) {      // out of line: most waits end at the first try
    uint64_t started = 0;
    while (!barrier_try(barrier, parity)) {
        uint64_t now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (started == 0) started = now;
        if (gone && *gone) break;
        if (now - started > TAU_WAIT_LIMIT_NS) {
            if (gone) *gone = 1;
            atomicExch(&wait_ran_out, 1);
            break;
        }
    }
}
__device__ __forceinline__ void barrier_wait(uint64_t* barrier, uint32_t parity, volatile int* gone) {
    if (!barrier_try(barrier, parity)) barrier_wait_on(barrier, parity, gone);
    __syncwarp();
}
// 1 if a wait of this library ran out since it was loaded (synchronises the device).
inline int wait_status() {
    int raised = 1;
    return cudaMemcpyFromSymbol(&raised, wait_ran_out, sizeof(raised)) == cudaSuccess ? raised : 1;
}

// Runs of `from` tokens and more go in chunks of `size` tokens, numbered one run after the other.  There are at most tokens / from such runs and
// tokens / size + that many chunks, which is what the host launches: a step of many single tokens beside one long run has no blocks for them (15,616 blocks of
// delta_state that returned at once took 45 us).
struct Run {
    int sequence, first;      // of the step, and the number of its first chunk; sequence -1: there is no such run
};
inline int most_runs(int tokens, int n_seqs, int from) { return tokens / from < n_seqs ? tokens / from : n_seqs; }
inline int most_chunks(int tokens, int n_seqs, int from, int size) { return tokens / size + most_runs(tokens, n_seqs, from); }
// The run that `wanted` belongs to, counting runs (`by_chunk` false) or chunks.  Every lane of the warp calls it and gets the answer.
template <bool by_chunk>
__device__ __forceinline__ Run find_run(const int* __restrict__ cu_seqlens, int n_seqs, int from, int size, int wanted) {
    const int lane = threadIdx.x & 31;
    int runs_before = 0, chunks_before = 0;
    for (int base = 0; base < n_seqs; base += 32) {
        const int sequence = base + lane;
        const int length = sequence < n_seqs ? cu_seqlens[sequence + 1] - cu_seqlens[sequence] : 0;
        const int own = length >= from && length > 0 ? (length + size - 1) / size : 0;
        const unsigned runs = __ballot_sync(0xffffffffu, own > 0);
        int chunks = own;      // up to this run, itself included
#pragma unroll
        for (int offset = 1; offset < 32; offset <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, chunks, offset);
            if (lane >= offset) chunks += other;
        }
        const int run = runs_before + __popc(runs & ((1u << lane) - 1u)), first = chunks_before + chunks - own;
        const unsigned here = __ballot_sync(0xffffffffu, own > 0 && (by_chunk ? wanted >= first && wanted < first + own : wanted == run));
        if (here) {
            const int at = __ffs(here) - 1;
            return {base + at, __shfl_sync(0xffffffffu, first, at)};
        }
        runs_before += __popc(runs);
        chunks_before += __shfl_sync(0xffffffffu, chunks, 31);
    }
    return {-1, 0};
}

constexpr int kPieces = 3;

// The pieces of two neighbouring numbers, packed for a fragment (the first in the low half).
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&pieces)[kPieces]) {
#pragma unroll
    for (int p = 0; p < kPieces; ++p) {
        const __nv_bfloat162 rounded = __floats2bfloat162_rn(x, y);
        pieces[p] = *reinterpret_cast<const uint32_t*>(&rounded);
        x -= __low2float(rounded);
        y -= __high2float(rounded);
    }
}
__device__ __forceinline__ void split_one(float x, bf16 (&pieces)[kPieces]) {
#pragma unroll
    for (int p = 0; p < kPieces; ++p) {
        pieces[p] = __float2bfloat16_rn(x);
        x -= __bfloat162float(pieces[p]);
    }
}

}  // namespace chunk
