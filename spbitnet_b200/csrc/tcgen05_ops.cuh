// Barriers, copies and descriptors of the tcgen05 kernels (gemm_tcsp_ws.cu, half_gemm_tc.cu).
#pragma once
#include <cuda.h>

#include "spb_common.cuh"

namespace spb {

constexpr long long kWsWaitCycles = 40000000;

__device__ __forceinline__ void ws_count_timeout(int* counter) {
    if (counter) atomicAdd_system(counter, 1);
}

__device__ __forceinline__ uint32_t ws_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// K-major, 128-byte swizzle: 8-row groups of 1024 B (SBO), 16-byte leading offset.
__device__ __forceinline__ uint64_t ws_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
// Bounded by time, not by polls (a poll may suspend for a while): kWsWaitCycles is about 20 ms at 2 GHz.
__device__ __forceinline__ bool ws_wait(uint32_t mbar, uint32_t parity, long long limit) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    const long long t0 = clock64();
    for (;;) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > limit) return false;
    }
}
// For what comes only after the grid's predecessors: their time does not count towards the bound.
__device__ __forceinline__ bool ws_wait_dep(uint32_t mbar, uint32_t parity, long long limit) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    grid_dep_wait();
    return ws_wait(mbar, parity, limit);
}
__device__ __forceinline__ void ws_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void ws_init(uint32_t mbar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count));
}
__device__ __forceinline__ void ws_expect(uint32_t mbar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ws_tma(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}
__device__ __forceinline__ void ws_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
// Position in a ring of barriers: stage and phase, advanced without a division.
struct WsCursor {
    int s = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void advance(int depth, int by = 1) {
        s += by;
        if (s >= depth) {
            s -= depth;
            ph ^= 1u;
        }
    }
};
__device__ __forceinline__ bool ws_elect() {
    uint32_t e;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(e));
    return e != 0;
}
// 16-byte piece c of row r of a 128-byte-swizzled tile
__device__ __forceinline__ uint32_t ws_swz(int r, int c) {
    return static_cast<uint32_t>((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}
// Tensor map of a row-major matrix: rows of `inner` elements `stride_bytes` apart, zero fill outside.  False when the driver
// does not offer or refuses it.
bool ws_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int inner, int outer, size_t stride_bytes,
            int box_inner, int box_outer, CUtensorMapSwizzle swizzle);

}  // namespace spb
