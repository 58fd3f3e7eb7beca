// What the tcgen05 kernels share: bounded waits on mbarriers, TMA copies, matrix and instruction descriptors, products and
// reads of tensor memory.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace {

#ifndef TAU_WAIT_LIMIT_NS
#define TAU_WAIT_LIMIT_NS 2000000000ull      // the tests of waits that run out compile with a shorter one
#endif
constexpr unsigned long long kWaitLimitNs = TAU_WAIT_LIMIT_NS;

// Whether a block of so much dynamic shared memory has an SM (228 KB, a kilobyte of them the system's for each block) to itself.  A block that takes all 512 columns of
// tensor memory must: a second one beside it would wait for them, unbounded, and its cluster's other blocks for it, while two clusters that hold an SM each
// wait for each other.
constexpr bool alone_on_an_sm(int shared_bytes) { return 2 * (shared_bytes + 1024) > 228 * 1024; }

__device__ int wait_error = 0;   // raised when a wait of this library ran out; read by its status function

__device__ __forceinline__ uint32_t smem_address(const void* pointer) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(pointer));
}

__device__ __forceinline__ unsigned long long global_timer() {
    unsigned long long now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    return now;
}

__device__ __forceinline__ void barrier_init(uint64_t* barrier, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_address(barrier)), "r"(count));
}

__device__ __forceinline__ void barrier_expect_bytes(uint64_t* barrier, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_address(barrier)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void barrier_arrive(uint64_t* barrier) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_address(barrier)) : "memory");
}

__device__ __forceinline__ bool barrier_try_wait(uint64_t* barrier, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_address(barrier)), "r"(parity)
        : "memory");
    return done != 0;
}

// Waits for the phase with the given parity to complete.  Returns false if the block is giving up.
__device__ __forceinline__ bool barrier_wait(uint64_t* barrier, uint32_t parity, volatile int* abort_flag) {
    if (barrier_try_wait(barrier, parity)) return true;
    const unsigned long long started = global_timer();
    for (uint32_t spin = 1;; ++spin) {
        if (barrier_try_wait(barrier, parity)) return true;
        if ((spin & 63u) == 0u) {
            if (*abort_flag) return false;
            if (global_timer() - started > kWaitLimitNs) {
                *abort_flag = 1;
                atomicExch(&wait_error, 1);
                return false;
            }
        }
    }
}

// Waits no longer than the limit for a copy, also where the block is giving up: until it has landed the shared memory is the copy's.
__device__ __forceinline__ void barrier_outlast(uint64_t* barrier, uint32_t parity) {
    if (barrier_try_wait(barrier, parity)) return;
    const unsigned long long started = global_timer();
    while (!barrier_try_wait(barrier, parity) && global_timer() - started <= kWaitLimitNs) {}
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    return rank;
}

// The tests of waits that run out name a rank: the operands of the blocks of that rank in their clusters never arrive.
__device__ __forceinline__ bool operands_lost() {
#ifdef TAU_LOST_RANK
    return cluster_rank() == TAU_LOST_RANK;
#else
    return false;
#endif
}

__device__ __forceinline__ void tma_load_2d(void* destination, const CUtensorMap* map, int inner, int outer, uint64_t* barrier) {
    if (operands_lost()) return;
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_address(destination)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(inner), "r"(outer), "r"(smem_address(barrier))
                 : "memory");
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes with the 128-byte swizzle:
// groups of 8 rows are 1024 bytes apart; version 1; the leading offset is not used by swizzled K-major tiles.
__device__ __forceinline__ uint64_t tile_descriptor(uint32_t address) {
    return static_cast<uint64_t>((address >> 4) & 0x3fffu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor: float accumulate, bfloat16 A and B, both K-major, M = m, N = n.
__device__ __forceinline__ uint32_t instruction_descriptor(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// True in one lane of a whole warp.  A role that issues products runs as a whole warp and lets this lane issue: what the warp computes is then the same for every lane to the
// compiler, which keeps descriptors in uniform registers.  Computed by a single thread they cost more than the products: one tcgen05.mma of 128 x 128 x 16 in 77 to 107 clocks, here 64.
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}

__device__ __forceinline__ void mma_issue(uint32_t accumulator, uint64_t a, uint64_t b, uint32_t descriptor, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(accumulator), "l"(a), "l"(b), "r"(descriptor), "r"(accumulate)
        : "memory");
}

// Makes the barrier complete when every tcgen05.mma issued so far by this thread has finished.
__device__ __forceinline__ void mma_commit(uint64_t* barrier) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_address(barrier)) : "memory");
}

__device__ __forceinline__ void tensor_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tensor_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tensor_load_16(uint32_t address, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(address));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 consecutive columns of this thread's lane; the caller waits (`tensor_load_wait`) before it uses them.
__device__ __forceinline__ void tensor_load_32(uint32_t address, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
        "%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(address));
}

__device__ __forceinline__ void tensor_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The address, in the cluster's shared window, of `pointer`'s twin in the block of rank `rank`.
__device__ __forceinline__ uint32_t cluster_address(const void* pointer, uint32_t rank) {
    uint32_t address;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(address) : "r"(smem_address(pointer)), "r"(rank));
    return address;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_address_of(uint32_t shared_address, int rank) {
    uint32_t address;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(address) : "r"(shared_address), "r"(rank));
    return address;
}

__device__ __forceinline__ float cluster_load(uint32_t address) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(address) : "memory");
    return v;
}

// By all threads of a block before its cluster's blocks meet: one that gave up raises the others' flags too, so that none joins what it did not finish.  (The blocks asking for each
// other's flags between their two meetings took 0.3 us and more.)
__device__ __forceinline__ void cluster_share_abort(const int* abort_flag, int blocks) {
    if (*static_cast<const volatile int*>(abort_flag) != 0 && static_cast<int>(threadIdx.x) < blocks)
        asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(cluster_address(abort_flag, threadIdx.x)), "r"(1) : "memory");
}

// Four floats from the shared memory of a block of the cluster (an address from `cluster_address`).
__device__ __forceinline__ float4 cluster_load_4(uint32_t address) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address) : "memory");
    return v;
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static EncodeTiled function = nullptr;
    if (!function) {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            function = reinterpret_cast<EncodeTiled>(entry);
    }
    return function;
}

}  // namespace
