// LM head of a batch on the tensor cores: y[b, r] = sum_c W[r, c] * x[b, c], half operands, fp32 sums (half_gemv_gpu of the
// reference, src/kernels/inference_kernels.cu:488-531, for up to 64 vectors).
//
// A block owns 256 rows of W (two accumulators of 128 x N in tensor memory) and the whole width: W and x come in 64-column
// tiles by tensor-map copies, five stages of 32 + 8 KB in flight, one thread issues tcgen05.mma.kind::f16, four warps read
// the sums back.  Bound: HBM, W is read once (x out of L2: 256 rows per block keep that traffic at a quarter of W's).  The
// row tiles of the last round still stream at nearly the full rate, an SM alone pulls more than its share.
//   128256 x 8192, 64 vectors (2.1 GB): 810 -> 326 us = 6.4 TB/s, against warp-level MMAs fed by ordinary loads.
#include "fused_ops.cuh"
#include "tcgen05_ops.cuh"

namespace spb {

namespace {

constexpr int kHgRows = 256, kHgStages = 5, kHgWBytes = kHgRows * 128, kHgThreads = 192;

struct HgArgs {
    float* y;
    int rows, cols, batch, n;  // n: batch rounded up to 16
    int* timeouts;
};
struct HgMaps {
    CUtensorMap w, x;
};

__global__ void __launch_bounds__(kHgThreads, 1) half_gemm_tc_kernel(const HgArgs a, const __grid_constant__ HgMaps maps) {
    extern __shared__ uint8_t hg_raw[];
    // [barriers 256 B] ... 1024-aligned: [stage: W rows 0-127 | W rows 128-255 | x] x kHgStages
    const uint32_t raw_s = ws_smem(hg_raw), full = raw_s, freeb = raw_s + 64, done = raw_s + 128;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(hg_raw + 136);
    const uint32_t ring = (raw_s + 256 + 1023) & ~1023u;
    const int x_bytes = a.n * 128, stage = kHgWBytes + x_bytes;
    const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * kHgRows, nk = (a.cols + 63) / 64;
    const uint32_t tmem_cols = 2 * a.n <= 32 ? 32u : 2 * a.n <= 64 ? 64u : 128u;
    grid_dep_launch();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kHgStages; ++s) {
            ws_init(full + 8 * s, 1);
            ws_init(freeb + 8 * s, 1);
        }
        ws_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the weights of the first stages depend on no predecessor
        for (int s = 0; s < min(kHgStages, nk); ++s) {
            ws_expect(full + 8 * s, stage);
            ws_tma(ring + s * stage, &maps.w, 64 * s, row0, full + 8 * s);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ws_smem(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            grid_dep_wait();
            int issued = 0;
            for (; issued < min(kHgStages, nk); ++issued)
                ws_tma(ring + issued * stage + kHgWBytes, &maps.x, 64 * issued, 0, full + 8 * issued);
            WsCursor c;
            for (; issued < nk; ++issued, c.advance(kHgStages)) {
                if (!(ok = ws_wait(freeb + 8 * c.s, c.ph, kWsWaitCycles))) break;
                ws_expect(full + 8 * c.s, stage);
                ws_tma(ring + c.s * stage, &maps.w, 64 * issued, row0, full + 8 * c.s);
                ws_tma(ring + c.s * stage + kHgWBytes, &maps.x, 64 * issued, 0, full + 8 * c.s);
            }
            for (int k = max(0, issued - kHgStages); k < issued; ++k)  // nothing in flight when the block leaves
                if (!ws_wait(full + 8 * (k % kHgStages), static_cast<uint32_t>(k / kHgStages) & 1u, kWsWaitCycles)) ok = false;
            if (!ok) ws_count_timeout(a.timeouts);
        }
    } else if (warp == 1) {
        if (ws_elect()) {
            // f16 operands, f32 accumulators, both K-major
            const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(a.n >> 3) << 17) | ((128u >> 4) << 24);
            WsCursor c;
            uint32_t acc = 0;
            for (int k = 0; k < nk; ++k, c.advance(kHgStages)) {
                if (!(ok = ws_wait_dep(full + 8 * c.s, c.ph, kWsWaitCycles))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = ring + c.s * stage;
                const uint64_t w0 = ws_smem_desc(st), w1 = ws_smem_desc(st + kHgWBytes / 2), x = ws_smem_desc(st + kHgWBytes);
#pragma unroll
                for (int q = 0; q < 4; ++q) {  // 16 columns: 32 bytes of either operand
#pragma unroll
                    for (int g = 0; g < 2; ++g)
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            :
                            : "r"(tmem + g * a.n), "l"((g ? w1 : w0) + 2 * q), "l"(x + 2 * q), "r"(idesc), "r"(acc | q)
                            : "memory");
                }
                acc = 1;
                ws_commit(freeb + 8 * c.s);
            }
            ws_commit(done);
            if (!ok) ws_count_timeout(a.timeouts);
        }
    } else {
        grid_dep_wait();
        ok = ws_wait(done, 0, 4 * kWsWaitCycles);
        ok = __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;
        if (!ok && lane == 0) ws_count_timeout(a.timeouts);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int quarter = warp & 3;  // tensor-memory lanes 32 (warp % 4) .. + 31
        if (ok)
            for (int g = 0; g < 2; ++g)
                for (int c0 = 0; c0 < a.n; c0 += 16) {
                    uint32_t r[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                        : "r"(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(g * a.n + c0))
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const int row = row0 + g * 128 + quarter * 32 + lane;
                    if (row < a.rows)
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < a.batch) a.y[static_cast<size_t>(c0 + i) * a.rows + row] = __uint_as_float(r[i]);
                }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

}  // namespace

// W: rows x cols half, x: batch x cols half (16-byte rows), y: batch x rows float; up to 64 vectors.
int half_gemm_tc(const __half* W, const __half* x, float* y, int rows, int cols, int batch, void* stream) {
    const char* name = "half_gemm_tc";
    if (cols % 8 || batch > 64 || ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(x)) & 15u))
        return fail(SPB_E_UNSUPPORTED, "%s: layout", name);
    HgArgs a{y, rows, cols, batch, (batch + 15) / 16 * 16, timeout_counter()};
    alignas(64) HgMaps maps;
    if (!ws_map(&maps.w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, W, cols, rows, static_cast<size_t>(cols) * 2, 64, kHgRows, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !ws_map(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, cols, batch, static_cast<size_t>(cols) * 2, 64, a.n, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(SPB_E_UNSUPPORTED, "%s: no tensor map", name);
    const size_t smem = 256 + 1024 + static_cast<size_t>(kHgStages) * (kHgWBytes + a.n * 128);
    if (int rc = ensure_dynamic_smem(name, half_gemm_tc_kernel, smem)) return rc;
    return launch(name, half_gemm_tc_kernel, dim3((rows + kHgRows - 1) / kHgRows), dim3(kHgThreads), smem, stream, a, maps);
}

}  // namespace spb
