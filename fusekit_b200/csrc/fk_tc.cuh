// Barriers and issue helpers of the warp-specialised tcgen05 kernels (fk_gemm_tc.cuh, fk_flash_tc.cuh, fk_qgemm.cuh).
//
// Every wait for copies, for MMAs and for what another warp hands over is bounded: TC_WAIT_LIMIT polls by default (FklEnv::wait_limit), after which
// the kernel sets an error bit, waits for its own copies and MMAs in flight (TC_DRAIN polls at most, whatever the limit above), frees its
// tensor memory and returns.  A warp whose lanes go on together decides together: tc_wait_warp and tc_all give all 32 lanes one answer, so that no lane
// leaves a loop whose other lanes enter an aligned instruction or a full-mask shuffle.
// What cannot be counted: the allocation of tensor memory (it waits for a block on the same SM that holds some to leave, and no such block waits for the one
// that allocates), barriers of threads of a block or a cluster (every warp reaches each of them, also after it gave up; where some would not,
// the warps vote first: qg_all), and griddepcontrol.wait.
#pragma once
#include "fk_common.cuh"
#include <cuda.h>

#define TC_WAIT_LIMIT (1u << 21)
#define TC_DRAIN (1u << 21)

__device__ __forceinline__ uint32_t tc_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void tc_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tc_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tc_expect(uint32_t bar, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool tc_poll(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// one thread waits
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) if (tc_poll(bar, parity)) return true;
    return false;
}
// a whole warp waits
__device__ __forceinline__ bool tc_wait_warp(uint32_t bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) if (__all_sync(0xffffffffu, tc_poll(bar, parity))) return true;
    return false;
}
// looks once without waiting; the warp takes the answer with a vote where it needs it (a vote right here would wait for the look)
__device__ __forceinline__ bool tc_look(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool tc_all(bool v) { return __all_sync(0xffffffffu, v); }
// true in one lane of a warp whose lanes are together, the same one every time
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// The MMAs that this warp's elected lane has issued are done (called by the whole warp, on a barrier of one arrival that nothing else uses).
__device__ __forceinline__ bool tc_drain_mmas(uint32_t bar) {
    if (tc_elect()) tc_commit(bar);
    __syncwarp();
    return tc_wait_warp(bar, 0u, TC_DRAIN);
}
__device__ __forceinline__ void tc_load(uint32_t dst, const CUtensorMap *map, int k, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(k), "r"(row), "r"(bar) : "memory");
}
// K-major operand with 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// an address of this block's shared memory in block `rank` of the cluster; a barrier of all threads of the cluster's blocks
__device__ __forceinline__ uint32_t tc_remote(uint32_t addr, uint32_t rank) { uint32_t r; asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r; }
__device__ __forceinline__ void tc_cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
