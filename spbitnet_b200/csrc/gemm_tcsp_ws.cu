// Batched sparse-ternary product on tcgen05.mma.sp, warp-specialised (sm_100a).
//
//   Y[j, r] = sum_c W[r, c] * X[j, c]      W: rows x cols compressed 2:4 ternary, X: n x cols int8
//
// Operands: the sign bytes (+1 / -1) of a tile as the compressed A operand in shared memory (K-major, 128-byte
// swizzle), the index pairs as metadata in tensor memory (one byte per 8 columns, lane = weight row), the activation
// tiles by tensor-map bulk copies, int32 accumulators in tensor memory.  A block owns 128 weight rows (mh = 1) or 256
// (mh = 2, two accumulators on one activation tile), up to 256 (240) batch rows and a range of K; its roles meet only at
// mbarriers:
//   warps 0-15  re-encode: the packed words of a step (256 columns) from shared memory to sign bytes and index pairs.
//               mh = 1: two groups of eight warps take alternate steps; mh = 2: group g takes rows 128 g .. of every step;
//   warp 16     issues the MMAs (one lane), half a step at a time;
//   warp 17     brings the activation tiles: one tensor-map copy per half step (128 columns);
//   warp 18     brings the packed weights: tensor-map copies of 512 columns of every row, as they lie in memory, several
//               chunks ahead.  They depend on no predecessor and start before the dependency wait.
// With few row tiles the K extent is cut over a cluster of S blocks, each of which adds and stores a slice of the columns
// from all blocks' partial sums (distributed shared memory).  Sums are integers: same bits.
//
// What bounds it.  An MMA of 64 columns takes 47 + N / 2 clocks.  With wide batches the tensor pipe and the activation
// traffic out of L2 (256-row blocks halve it); with few batch rows the re-encoding, 650 clocks per step; below a dozen
// steps per block the start of a block (2 us) and, with a split, the exchange at 13 B per clock and SM.
//   28672 x 8192, n = 1024: 276 -> 147 us a call;  in a graph n = 64: 105 -> 25 us;  2560 x 6912, n = 200: 20.1 -> 9.7, against a form in
//   which weights came by 16-byte loads of a row per lane (32 cache lines per instruction), signs through a table in shared
//   memory, and the MMA thread divided four times per half step to find its ring slots (1050 of 1100 clocks).
// A sign word of 32 weights becomes 32 bytes by a bit transpose and eight byte permutes whose selectors are the sign bits
// themselves: 21 instructions, no table.
//
// LAYOUT = kTiled: cols % 16 == 0, row strides multiples of 4 words, 16-byte aligned meta / values / X (tensor maps).
// LAYOUT = kSigns8: the same, but sign rows on 8-byte boundaries only, in whole 8-byte pieces: a width that is an odd multiple
//   of 128 has tight sign rows of 8 (mod 16) bytes, which no tensor map takes.  Warp 18 brings the signs by 8-byte asynchronous
//   copies, four lanes per row and chunk, on the barrier that the bitmaps' copy completes.  28672 x 5504, n = 200: 27 us, in the
//   form for any layout 217;  6912 x 3200, n = 64: 9.1 and 17.5;  5000 x 1408, n = 200: 7.5 and 17.1.
// LAYOUT = kEdge: kTiled for widths that are no multiple of 128.
// LAYOUT = kAny: any other: the re-encoding warps load their words themselves, eight warps copy the activation tiles.
//
// kEdge and kAny decode every bitmap as the reference's table has it, also those without two bits set: these layouts have
// always been decoded by the table (6912 x 3204, n = 16, half: 12.2 -> 12.7 us).  The others take packed rows as the packing
// rules make them.
//
// Every wait is bounded; a role whose wait runs out records it and leaves its loop, the others then run out of their own
// bounds, the copy warps wait (bounded) for their copies in flight, tensor memory is freed and the block returns.
#include <atomic>
#include <cmath>
#include <mutex>

#include "gemm_tcsp_ws.cuh"
#include "tcgen05_ops.cuh"

namespace spb {

constexpr int kWsTileM = 128;
constexpr int kWsStepK = 256;                  // logical columns per step: two units per row
constexpr int kWsABytes = kWsTileM * 128;      // compressed A tile of a step: 128 rows x 128 bytes
constexpr int kWsWBytes = kWsTileM * (64 + 32);  // packed words of 512 columns of 128 rows: meta, values
constexpr int kWsExpandWarps = 16;
constexpr int kWsMmaWarp = 16, kWsXWarp = 17, kWsWWarp = 18;
constexpr int kWsThreadsTiled = 32 * 19;
constexpr int kWsCopyWarps = 8;                // kAny: warps 17 .. 24 copy the activation tiles
constexpr int kWsThreadsAny = 32 * (kWsXWarp + kWsCopyWarps);
constexpr int kWsBarBytes = 512, kWsScaleBytes = 1024;
constexpr int kWsSmemCap = 226 * 1024;

enum WsLayout { kTiled = 0, kAny = 1, kSigns8 = 2, kEdge = 3 };

struct WsMat {
    const uint32_t* meta;
    const uint32_t* values;
    void* out;  // int32 sums or half
    float gamma;
    int rows, meta_stride, values_stride, tile0;  // tile0: first row tile of this matrix in the grid
};
struct WsArgs {
    WsMat m[kWsMaxMats];
    const int8_t* X;
    const float* absmax;
    int nmat, cols, n;
    int nt;                 // batch rows per block: multiple of 16, at most 256
    int mh;                 // 128-row halves per block
    int sa, sb, sw;         // ring depths: A (steps), activations (half steps), packed words (512 columns)
    int tmem_cols;          // power of two >= mh * (nt + 8 * sa)
    int split;              // blocks per cluster that share the K extent
    int* timeouts;          // counter of waits that ran out (pinned host memory, system-scope atomics), may be null
    long long wait_cycles;  // bound of every wait in the kernel
};
struct WsMaps {
    CUtensorMap x, meta[kWsMaxMats], values[kWsMaxMats];
};

// 0 automatic, 1 / 2 force one / two weight-row halves per block (spb_set_gemm_row_halves; testing and measurement)
static int g_ws_mh = 0;

// kind::i8 instruction descriptor with the sparse flag: S32 accumulate, signed 8-bit A and B, K-major.
__device__ __forceinline__ uint32_t ws_idesc(int m, int n) {
    return (1u << 2) | (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(m >> 4) << 24);
}
// One MMA: 128 rows x N, 64 logical columns.  a_lo, b_lo: low words of the operands' descriptors.
__device__ __forceinline__ void ws_mma(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate, uint32_t meta) {
    constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (1u << 30);
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 a, {%1, %6};\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "tcgen05.mma.sp.cta_group::1.kind::i8 [%0], a, b, [%5], %3, p;\n\t}"
        :
        : "r"(d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(meta), "r"(hi)
        : "memory");
}
// Bitmaps of zero (past the end of a row or of the matrix: the activations there are zero, the rows are not stored)
// become {0, 1}: the tensor core is only given valid pairs.
__device__ __forceinline__ uint32_t ws_fill_empty(uint32_t m) {
    const uint32_t h = m | (m >> 1);
    const uint32_t z = ~(h | (h >> 2)) & 0x11111111u;
    return m | z | (z << 1);
}
// Eight bitmaps (two of four bits set each) -> eight index pairs {low index | high index << 2}.
__device__ __forceinline__ uint32_t ws_index_pairs(uint32_t m) {
    const uint32_t mr = m >> 1, ml = m << 1;
    const uint32_t t1 = (0x11111111u & (~m & mr)) | (~0x11111111u & (mr | ~m));
    const uint32_t t2 = (0x22222222u & (~ml & ~m)) | (~0x22222222u & (m | ml));
    return (t1 & 0x55555555u) | (t2 & 0xAAAAAAAAu);
}
// Bit 4 g set: bitmap g has not two bits set.
__device__ __forceinline__ uint32_t ws_odd_bitmaps(uint32_t m) {
    m -= (m >> 1) & 0x55555555u;
    const uint32_t x = ((m & 0x33333333u) + ((m >> 2) & 0x33333333u)) ^ 0x22222222u;  // counts of bits, 0 where two
    return (x | (x >> 1) | (x >> 2)) & 0x11111111u;
}
// 32 sign bits -> 32 bytes of +1 / -1 in order.  Transposing the 4 x 4 bits of each 16-bit half puts the signs 4 r .. 4 r
// + 3 at bit r of the half's four nibbles; a byte permute with the nibbles as selectors and a source whose byte i is -1
// where bit r of i is set then yields those four bytes.  A selector's top bit means "replicate the sign", so the nibbles
// are masked to three bits and bit 3 is read at bit 2.
__device__ __forceinline__ void ws_sign_bytes(uint32_t v, uint32_t (&w)[8]) {
    uint32_t t = (v ^ (v >> 3)) & 0x0A0A0A0Au;
    v ^= t ^ (t << 3);
    t = (v ^ (v >> 6)) & 0x00CC00CCu;
    v ^= t ^ (t << 6);
    const uint32_t lo = v & 0x77777777u, hi = (v >> 1) & 0x44444444u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t l = h ? lo >> 16 : lo, u = h ? hi >> 16 : hi;
        w[4 * h + 0] = __byte_perm(0xFF01FF01u, 0xFF01FF01u, l);
        w[4 * h + 1] = __byte_perm(0xFFFF0101u, 0xFFFF0101u, l);
        w[4 * h + 2] = __byte_perm(0x01010101u, 0xFFFFFFFFu, l);
        w[4 * h + 3] = __byte_perm(0x01010101u, 0xFFFFFFFFu, u);
    }
}

// ROWS4: every output starts its groups of four rows on a boundary of four elements (rows % 4 == 0, an aligned base)
template <bool HALF_OUT, int LAYOUT, bool ROWS4>
__global__ void __launch_bounds__(LAYOUT != kAny ? kWsThreadsTiled : kWsThreadsAny, 1)
    gemm_tcsp_ws_kernel(const WsArgs a, const __grid_constant__ WsMaps maps) {
    constexpr bool kMapped = LAYOUT != kAny, kAsyncSigns = LAYOUT == kSigns8, kAnyBitmap = LAYOUT == kAny || LAYOUT == kEdge;
    extern __shared__ uint8_t ws_raw[];
    // [barriers][row scales] ... 1024-aligned: [A ring][activation ring][packed-word ring]; the epilogue's sums take the
    // place of the rings when the products are done
    uint64_t* bars = reinterpret_cast<uint64_t*>(ws_raw);
    const uint32_t raw_s = ws_smem(ws_raw);
    const uint32_t a_full = raw_s, a_free = raw_s + 64, b_full = raw_s + 128, b_free = raw_s + 192, w_full = raw_s + 256,
                   w_free = raw_s + 320, done_b = raw_s + 384;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 50);
    float* scales = reinterpret_cast<float*>(ws_raw + kWsBarBytes);
    const uint32_t ring_s = (raw_s + kWsBarBytes + kWsScaleBytes + 1023) & ~1023u;
    const int a_bytes = a.mh * kWsABytes, b_bytes = a.nt * 128, w_bytes = a.mh * kWsWBytes;
    const uint32_t bring_s = ring_s + a.sa * a_bytes, wring_s = bring_s + a.sb * b_bytes;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    int mi = 0;
    if (a.nmat > 1 && static_cast<int>(blockIdx.x) >= a.m[1].tile0) mi = 1;
    if (a.nmat > 2 && static_cast<int>(blockIdx.x) >= a.m[2].tile0) mi = 2;
    const WsMat m = mi == 0 ? a.m[0] : mi == 1 ? a.m[1] : a.m[2];
    const int row0 = (static_cast<int>(blockIdx.x) - m.tile0) * kWsTileM * a.mh;
    const int n0 = blockIdx.y * a.nt;
    const int all_steps = (a.cols + kWsStepK - 1) / kWsStepK;
    const int s0 = static_cast<int>(blockIdx.z) * all_steps / a.split;
    const int nsteps = (static_cast<int>(blockIdx.z) + 1) * all_steps / a.split - s0;

    grid_dep_launch();
    const int nchunks = (nsteps + 1) >> 1;
    // packed words of 512 columns, 16 words of meta and 8 of values per row: called by lane 0, with kAsyncSigns by the warp
    auto load_chunk = [&](int c, int s) {
        const uint32_t bar = w_full + 8 * s, dst = wring_s + s * w_bytes, vdst = dst + a.mh * kWsTileM * 64;
        const int k2 = s0 + 2 * c;
        if (!kAsyncSigns || lane == 0) {
            ws_expect(bar, kAsyncSigns ? a.mh * kWsTileM * 64 : w_bytes);
            ws_tma(dst, &maps.meta[mi], 8 * k2, row0, bar);
        }
        if (!kAsyncSigns) {
            ws_tma(vdst, &maps.values[mi], 4 * k2, row0, bar);
            return;
        }
        const int piece = lane & 3, word = 4 * k2 + 2 * piece;  // a lane's two words of every eighth row
        const bool in_row = word < (a.cols >> 6);
        for (int r = lane >> 2; r < a.mh * kWsTileM; r += 8) {  // the tensor map's order: 16-byte halves swapped by bit 2 of the row
            const bool valid = in_row && row0 + r < m.rows;
            const uint32_t* src = m.values + (valid ? static_cast<size_t>(row0 + r) * m.values_stride + word : 0);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                             vdst + r * 32 + (((piece >> 1) ^ ((r >> 2) & 1)) << 4) + 8 * (piece & 1)),
                         "l"(src), "r"(valid ? 8 : 0)
                         : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    };
    if (kMapped && warp == kWsWWarp) {  // the first chunks leave before the block has set itself up (1100 clocks)
        if (lane == 0) {
            for (int s = 0; s < a.sw; ++s) {
                ws_init(w_full + 8 * s, kAsyncSigns ? 33 : 1);
                ws_init(w_free + 8 * s, kWsExpandWarps);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        if (kAsyncSigns || lane == 0)
            for (int s = 0; s < min(a.sw, nchunks); ++s) load_chunk(s, s);
    }
    if (tid == 32 * kWsXWarp) {
        if (kMapped) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.x)) : "memory");
        for (int s = 0; s < a.sa; ++s) {
            ws_init(a_full + 8 * s, 8 * a.mh);
            ws_init(a_free + 8 * s, 1);
        }
        for (int s = 0; s < a.sb; ++s) {
            ws_init(b_full + 8 * s, kMapped ? 1 : kWsCopyWarps);
            ws_init(b_free + 8 * s, 1);
        }
        ws_init(done_b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ws_smem(tmem_slot)),
                     "r"(static_cast<uint32_t>(a.tmem_cols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    const uint32_t tmem_e = tmem_d + static_cast<uint32_t>(a.nt * a.mh);  // metadata slots behind the accumulators
    bool ok = true;

    if (kMapped && warp == kWsWWarp) {
        // ---- packed weights: 512 columns of every row per chunk ---------------------------------------------------
        if (kAsyncSigns || lane == 0) {
            WsCursor w;
            int issued = min(a.sw, nchunks);
            w.ph = 1;
            for (; issued < nchunks; ++issued, w.advance(a.sw)) {
                if (!(ok = ws_wait_dep(w_free + 8 * w.s, w.ph ^ 1u, a.wait_cycles))) break;
                load_chunk(issued, w.s);
            }
            for (int c = max(0, issued - a.sw); c < issued; ++c)  // nothing in flight when the block leaves
                if (!ws_wait(w_full + 8 * (c % a.sw), static_cast<uint32_t>(c / a.sw) & 1u, a.wait_cycles)) ok = false;
            if (kAsyncSigns) asm volatile("cp.async.wait_all;" ::: "memory");
            if (!ok) ws_count_timeout(a.timeouts);
        }
    } else if (kMapped && warp == kWsXWarp) {
        // ---- activation tiles ----------------------------------------------------------------------------------------
        if (lane == 0) {
            grid_dep_wait();  // X may be a predecessor's output
            WsCursor x;
            int issued = 0;
            for (; issued < 2 * nsteps; ++issued, x.advance(a.sb)) {
                if (!(ok = ws_wait(b_free + 8 * x.s, x.ph ^ 1u, a.wait_cycles))) break;
                ws_expect(b_full + 8 * x.s, b_bytes);
                ws_tma(bring_s + x.s * b_bytes, &maps.x, s0 * kWsStepK + issued * 128, n0, b_full + 8 * x.s);
            }
            for (int h = max(0, issued - a.sb); h < issued; ++h)
                if (!ws_wait(b_full + 8 * (h % a.sb), static_cast<uint32_t>(h / a.sb) & 1u, a.wait_cycles)) ok = false;
            if (!ok) ws_count_timeout(a.timeouts);
        }
    } else if (!kMapped && warp >= kWsXWarp) {
        // ---- activation tiles, any alignment: a warp per batch row and half step, four columns per lane ------------
        grid_dep_wait();
        const int cw = warp - kWsXWarp;
        const bool words = (reinterpret_cast<uintptr_t>(a.X) & 3u) == 0;
        WsCursor xb;
        for (int h = 0; h < 2 * nsteps; ++h, xb.advance(a.sb)) {
            const int s = xb.s;
            ok = ws_wait(b_free + 8 * s, xb.ph ^ 1u, a.wait_cycles);
            ok = __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;
            if (!ok) break;
            const int col = s0 * kWsStepK + h * 128 + lane * 4;
            for (int r0 = cw; r0 < a.nt; r0 += 8 * kWsCopyWarps) {
                uint32_t x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int j = n0 + r0 + i * kWsCopyWarps;
                    x[i] = 0;
                    if (r0 + i * kWsCopyWarps < a.nt && j < a.n && col < a.cols) {
                        const int8_t* p = a.X + static_cast<size_t>(j) * a.cols + col;
                        if (words) {
                            x[i] = __ldg(reinterpret_cast<const uint32_t*>(p));
                        } else {
                            for (int b = 0; b < 4; ++b) x[i] |= static_cast<uint32_t>(static_cast<uint8_t>(p[b])) << (8 * b);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = r0 + i * kWsCopyWarps;
                    if (r < a.nt)
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(bring_s + s * b_bytes + ws_swz(r, lane >> 2) + 4 * (lane & 3)),
                                     "r"(x[i])
                                     : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) ws_arrive(b_full + 8 * s);
        }
        if (!ok && lane == 0) ws_count_timeout(a.timeouts);
    } else if (warp == kWsMmaWarp) {
        // ---- MMAs: two per half step and 128 rows.  One elected lane; addresses and phases advance by additions only: the
        //      tensor pipe takes 47 + N / 2 clocks per MMA, so the bookkeeping between two of them counts.
        if (ws_elect()) {
            const uint32_t idesc = ws_idesc(kWsTileM, a.nt);
            const uint32_t a_step = a_bytes >> 4, b_step = b_bytes >> 4;
            const uint32_t a_lo0 = static_cast<uint32_t>(ws_smem_desc(ring_s)), b_lo0 = static_cast<uint32_t>(ws_smem_desc(bring_s));
            uint32_t a_lo = a_lo0, b_lo = b_lo0, te = tmem_e, acc = 0;
            uint32_t abar = a_full, bbar = b_full;  // the matching "free" barriers lie 64 bytes on
            uint32_t aph = 0, bph = 0;
            auto half = [&](uint32_t h) {
                if (!ws_wait_dep(bbar, bph, a.wait_cycles)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                ws_mma(tmem_d, a_lo + 4 * h, b_lo, idesc, acc, te + 4 * h);
                ws_mma(tmem_d, a_lo + 4 * h + 2, b_lo + 4, idesc, 1, te + 4 * h + 2);
                if (a.mh == 2) {  // the second half of the weight rows into its own accumulator
                    ws_mma(tmem_d + a.nt, a_lo + (kWsABytes >> 4) + 4 * h, b_lo, idesc, acc, te + 8 + 4 * h);
                    ws_mma(tmem_d + a.nt, a_lo + (kWsABytes >> 4) + 4 * h + 2, b_lo + 4, idesc, 1, te + 8 + 4 * h + 2);
                }
                acc = 1;
                ws_commit(bbar + 64);
                b_lo += b_step;
                bbar += 8;
                if (bbar == b_full + 8 * a.sb) {
                    b_lo = b_lo0;
                    bbar = b_full;
                    bph ^= 1u;
                }
                return true;
            };
            for (int kc = 0; kc < nsteps; ++kc) {
                ok = ws_wait(abar, aph, a.wait_cycles) && half(0) && half(1);
                if (!ok) break;
                ws_commit(abar + 64);
                a_lo += a_step;
                te += 8 * a.mh;
                abar += 8;
                if (abar == a_full + 8 * a.sa) {
                    a_lo = a_lo0;
                    te = tmem_e;
                    abar = a_full;
                    aph ^= 1u;
                }
            }
            ws_commit(done_b);
            if (!ok) ws_count_timeout(a.timeouts);
        }
    } else if (warp < kWsExpandWarps) {
        // ---- re-encoding: thread t and thread t + 128 of a group share a weight row, one takes the even unit (128
        //      columns) of a step, the other the odd one.  A warp's rows are the tensor-memory lanes it may access.
        const int grp = warp >> 3;
        const int etid = (warp & 7) * 32 + lane;
        const int trow = etid & (kWsTileM - 1), thalf = etid >> 7;
        const int mhalf = a.mh == 2 ? grp : 0;
        const int first = a.mh == 2 ? 0 : grp, stride = a.mh == 2 ? 1 : 2;
        const int wr = mhalf * kWsTileM + trow;  // row within the block's packed words
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const int mwords = (a.cols + 31) >> 5, vwords = (a.cols + 63) >> 6;
        auto load_words = [&](int i, uint4& mm, uint2& vv) {  // kAny: step i's words, zero past the row's end
            uint32_t w[6] = {0, 0, 0, 0, 0, 0};
            if (row0 + wr < m.rows && i < nsteps) {
                const int u = 2 * (s0 + i) + thalf;
                const uint32_t* pm = m.meta + static_cast<size_t>(row0 + wr) * m.meta_stride;
                const uint32_t* pv = m.values + static_cast<size_t>(row0 + wr) * m.values_stride;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (4 * u + q < mwords) w[q] = __ldg(pm + 4 * u + q);
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (2 * u + q < vwords) w[4 + q] = __ldg(pv + 2 * u + q);
            }
            mm = make_uint4(w[0], w[1], w[2], w[3]);
            vv = make_uint2(w[4], w[5]);
        };
        const bool row_tail = row0 + a.mh * kWsTileM > m.rows;
        WsCursor ca, cw;
        ca.s = first;  // fewer steps than stages ahead: first < sa
        uint4 mm, mn;
        uint2 vv, vn;
        if (!kMapped) load_words(first, mn, vn);
        for (int i = first; i < nsteps; i += stride, ca.advance(a.sa, stride)) {
            if (kMapped) {
                const int s = cw.s, x = i & 1;
                ok = ws_wait(w_full + 8 * s, cw.ph, a.wait_cycles);
                ok = __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;
                if (!ok) break;
                const uint32_t pm = wring_s + s * w_bytes + wr * 64 + (((2 * x + thalf) ^ ((wr >> 1) & 3)) << 4);
                const uint32_t pv = wring_s + s * w_bytes + a.mh * kWsTileM * 64 + wr * 32 + ((x ^ ((wr >> 2) & 1)) << 4) + 8 * thalf;
                asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(mm.x), "=r"(mm.y), "=r"(mm.z), "=r"(mm.w) : "r"(pm) : "memory");
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(vv.x), "=r"(vv.y) : "r"(pv) : "memory");
            } else {
                mm = mn;
                vv = vn;
                load_words(i + stride, mn, vn);
            }
            uint32_t odd0 = 0, odd1 = 0, odd2 = 0, odd3 = 0;  // groups of the row whose bitmap has not two bits set
            if (kAnyBitmap) {
                const int left = row0 + wr < m.rows ? (a.cols >> 2) - 32 * (2 * (s0 + i) + thalf) : 0;  // the row's groups from here on
                auto odd = [&](uint32_t word, int q) {
                    const int g = left - 8 * q;
                    return g <= 0 ? 0u : ws_odd_bitmaps(word) & (g >= 8 ? 0xFFFFFFFFu : (1u << (4 * g)) - 1u);
                };
                odd0 = odd(mm.x, 0);
                odd1 = odd(mm.y, 1);
                odd2 = odd(mm.z, 2);
                odd3 = odd(mm.w, 3);
            }
            if (row_tail || (s0 + i + 1) * kWsStepK > a.cols) {
                mm.x = ws_fill_empty(mm.x);
                mm.y = ws_fill_empty(mm.y);
                mm.z = ws_fill_empty(mm.z);
                mm.w = ws_fill_empty(mm.w);
            }
            uint32_t w0[8], w1[8];
            uint32_t e0 = ws_index_pairs(mm.x), e1 = ws_index_pairs(mm.y), e2 = ws_index_pairs(mm.z), e3 = ws_index_pairs(mm.w);
            // The table puts both signs of such a group on its first column: index pair {0, 1} with the bytes {s0 + s1, 0}, the bytes
            // mended below.  (At an edge, groups past it were filled with {0, 1} above; an empty group inside gets the same.)
            if (kAnyBitmap) {
                e0 = (e0 & ~(odd0 * 15u)) | (odd0 << 2);
                e1 = (e1 & ~(odd1 * 15u)) | (odd1 << 2);
                e2 = (e2 & ~(odd2 * 15u)) | (odd2 << 2);
                e3 = (e3 & ~(odd3 * 15u)) | (odd3 << 2);
            }
            ws_sign_bytes(vv.x, w0);
            ws_sign_bytes(vv.y, w1);
            const int sA = ca.s;
            ok = ws_wait_dep(a_free + 8 * sA, ca.ph ^ 1u, a.wait_cycles);
            ok = __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;  // tcgen05.st below is warp-wide
            if (!ok) break;
            const uint32_t eaddr = tmem_e + lane_base + static_cast<uint32_t>((sA * a.mh + mhalf) * 8 + thalf * 4);
            asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(eaddr), "r"(e0), "r"(e1), "r"(e2),
                         "r"(e3)
                         : "memory");
            const uint32_t sm = ring_s + sA * a_bytes + mhalf * kWsABytes;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t* w = (c & 2) ? w1 + 4 * (c & 1) : w0 + 4 * (c & 1);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sm + ws_swz(trow, thalf * 4 + c)), "r"(w[0]),
                             "r"(w[1]), "r"(w[2]), "r"(w[3])
                             : "memory");
            }
            if (kAnyBitmap && (odd0 | odd1 | odd2 | odd3)) {
#pragma unroll 1
                for (int g = 0; g < 32; ++g) {
                    const uint32_t word = g < 8 ? odd0 : g < 16 ? odd1 : g < 24 ? odd2 : odd3;
                    if (!((word >> (4 * (g & 7))) & 1u)) continue;
                    const uint32_t signs = ((g < 16 ? vv.x : vv.y) >> (2 * (g & 15))) & 3u;
                    const uint32_t pair = signs == 0 ? 2u : signs == 3 ? 0xFEu : 0u;  // s0 + s1 | 0 << 8
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(sm + ws_swz(trow, thalf * 4 + (g >> 3)) + 2 * (g & 7)),
                                 "h"(static_cast<unsigned short>(pair))
                                 : "memory");
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the tensor core
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) ws_arrive(a_full + 8 * sA);
            // The chunk is given back only here, after its words have gone through registers into the stores above: with the
            // arrival right behind the loads the copy engine overwrote words that a load still had to read.
            if (kMapped && (a.mh == 1 || (i & 1))) {
                if (lane == 0) ws_arrive(w_free + 8 * cw.s);
                cw.advance(a.sw);
            }
        }
        if (!ok && lane == 0) ws_count_timeout(a.timeouts);
    }
    __syncwarp();
    // ---- epilogue: accumulators -> shared memory, [column][128 rows] words in place of the rings -> output.  Every
    //      thread of the block then takes four rows of a column: the output is written 256 (512) bytes at a time.  Where four
    //      rows do not lie on one boundary that would be four stores of 2 (4) bytes at a stride of 8 (16), so a block that has
    //      no peers stores from the registers, 32 consecutive rows at a time (1001 x 640, n = 64, int32: 5.2 -> 4.5 us; with
    //      rows on such boundaries the way through shared memory is the faster one, 28672 x 640, n = 200, half: 10.5
    //      against 12.5 us).  In a cluster block z adds and stores the columns [z cs, + cs) of all blocks' sums.
    grid_dep_wait();  // the output may still be read by a predecessor, the scales are its result
    if (HALF_OUT && tid < a.nt) scales[tid] = dequant_scale(m.gamma, a.absmax[min(n0 + tid, a.n - 1)]);
    if (warp < kWsExpandWarps) {
        ok = ws_wait(done_b, 0, a.wait_cycles) && ok;
        ok = __all_sync(0xFFFFFFFFu, ok ? 1 : 0) != 0;
        if (!ok && lane == 0) ws_count_timeout(a.timeouts);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();  // every copy has landed and every MMA is done (or a wait ran out: the output is unspecified)
    const int S = a.split, cs = (a.nt + S - 1) / S, me = static_cast<int>(blockIdx.z);
    auto sums16 = [&](int g, int c0, uint32_t (&r)[16]) {  // tensor-memory lanes 32 (w % 4) .. + 31, 16 columns
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem_d + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(g * a.nt + c0))
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    };
    if (!ROWS4 && S == 1 && warp < kWsExpandWarps && ok)
        for (int g = 0; g < a.mh; ++g) {  // a lane's row, 32 consecutive rows per store
            const int row = row0 + g * kWsTileM + (warp & 3) * 32 + lane;
            for (int c0 = 16 * (warp >> 2); c0 < a.nt; c0 += 64) {
                uint32_t r[16];
                sums16(g, c0, r);
                if (row >= m.rows) continue;
                const int left = a.n - n0 - c0;  // batch rows of these columns
                const size_t o = static_cast<size_t>(n0 + c0) * m.rows + row;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (i < left) {
                        if (HALF_OUT)
                            static_cast<__half*>(m.out)[o + static_cast<size_t>(i) * m.rows] =
                                __float2half_rn(__fmul_rn(static_cast<float>(static_cast<int>(r[i])), scales[c0 + i]));
                        else
                            static_cast<int32_t*>(m.out)[o + static_cast<size_t>(i) * m.rows] = static_cast<int>(r[i]);
                    }
            }
        }
    for (int g = 0; g < (ROWS4 || S > 1 ? a.mh : 0); ++g) {
        if (warp < kWsExpandWarps && ok)
            for (int c0 = 16 * (warp >> 2); c0 < a.nt; c0 += 64) {
                uint32_t r[16];
                sums16(g, c0, r);
                const uint32_t at = ring_s + static_cast<uint32_t>((c0 * kWsTileM + (warp & 3) * 32 + lane) * 4);
#pragma unroll
                for (int i = 0; i < 16; ++i) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + i * kWsTileM * 4), "r"(r[i]) : "memory");
            }
        if (S > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
        const int c_lo = me * cs, c_hi = min(a.nt, c_lo + cs);
        for (int e = c_lo * 32 + tid; e < c_hi * 32; e += static_cast<int>(blockDim.x)) {
            const int c = e >> 5, row = row0 + g * kWsTileM + 4 * (e & 31), j = n0 + c;
            const uint32_t at = ring_s + static_cast<uint32_t>(e) * 16;
            int4 sum;
            if (S == 1) {
                asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(sum.x), "=r"(sum.y), "=r"(sum.z), "=r"(sum.w) : "r"(at) : "memory");
            } else {
                sum = make_int4(0, 0, 0, 0);
#pragma unroll
                for (int p = 0; p < 8; ++p)
                    if (p < S) {
                        uint32_t remote;
                        int4 v;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(p));
                        asm volatile("ld.shared::cluster.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(remote));
                        sum.x += v.x;
                        sum.y += v.y;
                        sum.z += v.z;
                        sum.w += v.w;
                    }
            }
            if (j >= a.n || row >= m.rows) continue;
            const size_t o = static_cast<size_t>(j) * m.rows + row;
            if (HALF_OUT) {
                const float sc = scales[c];
                __half h[4];
                h[0] = __float2half_rn(__fmul_rn(static_cast<float>(sum.x), sc));
                h[1] = __float2half_rn(__fmul_rn(static_cast<float>(sum.y), sc));
                h[2] = __float2half_rn(__fmul_rn(static_cast<float>(sum.z), sc));
                h[3] = __float2half_rn(__fmul_rn(static_cast<float>(sum.w), sc));
                __half* dst = static_cast<__half*>(m.out) + o;
                if (ROWS4) {
                    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (row + i < m.rows) dst[i] = h[i];
                }
            } else {
                int32_t* dst = static_cast<int32_t*>(m.out) + o;
                if (ROWS4) {
                    *reinterpret_cast<int4*>(dst) = sum;
                } else {
                    const int32_t v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (row + i < m.rows) dst[i] = v[i];
                }
            }
        }
        if (S > 1) {  // nobody leaves, or overwrites its sums, while a peer reads them
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else if (g + 1 < a.mh) {
            __syncthreads();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d),
                     "r"(static_cast<uint32_t>(a.tmem_cols))
                     : "memory");
}

// One block that allocates tensor memory, waits with ws_wait on a barrier nobody arrives at, reports the run-out
// like the product kernel does, frees the tensor memory and returns.  No copy is in flight at any time.
__global__ void __launch_bounds__(128, 1) ws_wait_selftest_kernel(int* timeouts, long long limit) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ws_smem(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ws_smem(&tmem_slot)), "r"(32u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    if (threadIdx.x == 0 && !ws_wait(ws_smem(&bar), 0u, limit)) ws_count_timeout(timeouts);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32u) : "memory");
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeFn tensor_map_encoder() {
    static const EncodeFn encode = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<EncodeFn>(p);
    }();
    return encode;
}

static const int* ws_max_clusters();

// Everything the launchers look up or allocate lazily on the host (driver entry point, the pinned timeout counter,
// the SM and cluster counts), done now: an engine calls this at creation so that none of it first happens inside a stream
// capture, where allocations and look-ups are not allowed.
void prepare_host_state() {
    tensor_map_encoder();
    timeout_counter();
    sm_count();
    ws_max_clusters();
}

bool ws_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int inner, int outer,
                   size_t stride_bytes, int box_inner, int box_outer, CUtensorMapSwizzle swizzle) {
    const EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t gdim[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
    const cuuint64_t gstride[1] = {static_cast<cuuint64_t>(stride_bytes)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_outer)};
    const cuuint32_t estr[2] = {1u, 1u};
    return encode(map, type, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct WsShape {
    int mh, nt, split, sa, sb, sw;
    size_t smem;
};

// Ring depths for a tile: as many stages as fit, the activations first (their latency is the longest after the weights').
static void ws_rings(WsShape& c, bool tiled) {
    const int ab = c.mh * kWsABytes, bb = c.nt * 128, wb = tiled ? c.mh * kWsWBytes : 0;
    c.sa = 2;
    c.sb = 2;
    c.sw = tiled ? 2 : 0;
    const int cap = kWsSmemCap - kWsBarBytes - kWsScaleBytes - 1024;
    auto used = [&] { return c.sa * ab + c.sb * bb + c.sw * wb; };
    for (bool grew = true; grew;) {
        grew = false;
        if (c.sb < 4 && used() + bb <= cap) { ++c.sb; grew = true; }
        if (tiled && c.sw < 4 && used() + wb <= cap) { ++c.sw; grew = true; }
        if (c.sa < 4 && c.mh * (c.nt + 8 * (c.sa + 1)) <= 512 && used() + ab <= cap) { ++c.sa; grew = true; }
    }
    // the epilogue's sums take the place of the rings
    c.smem = kWsBarBytes + kWsScaleBytes + 1024 + static_cast<size_t>(max(used(), c.nt * kWsTileM * 4));
}

constexpr int kWsMaxSplit = 8;
// Clusters of S = 1 .. kWsMaxSplit blocks, one block per SM, that the current device holds at a time: table[S].  A cluster sits
// in one GPC, so it is less than SMs / S by an amount that only the driver knows; asked once per device.
static const int* ws_max_clusters() {
    static int table[64][kWsMaxSplit + 1];
    static std::atomic<bool> ready[64];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (ready[dev].load(std::memory_order_acquire)) return table[dev];
    std::lock_guard<std::mutex> lock(mu);
    const auto kernel = gemm_tcsp_ws_kernel<true, kTiled, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kWsThreadsTiled);
    cfg.dynamicSmemBytes = kWsSmemCap;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool can_ask = ensure_dynamic_smem("cluster occupancy", kernel, cfg.dynamicSmemBytes) == SPB_OK;
    table[dev][1] = sm_count();
    for (int S = 2; S <= kWsMaxSplit; ++S) {
        cfg.gridDim = dim3(1, 1, S);
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = S;
        int n = 0;
        if (!can_ask || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = max(1, sm_count() * 3 / 4 / S);
        }
        table[dev][S] = n;
    }
    ready[dev].store(true, std::memory_order_release);
    return table[dev];
}

// How a product is cut: 128- or 256-row blocks, batch rows per block, blocks per cluster along K: the least of
//   waves * (start + steps * clocks per step + drain [+ exchange])
// in clocks, as measured (nt = batch rows per block, clocks per step of 256 columns):
//   128 rows: 690 up to nt = 128 (re-encoding), 925 at 176, 1047 at 256 (activations out of L2, 62 B per clock and SM);
//   256 rows: 1250 at nt = 64 (re-encoding), 1530 at 208: half the activation traffic per weight row, so it wins where
//   the batch is wide, and where it saves a wave;
//   start: 4500 to the first product (weights from HBM, re-encoding, activations);
//   drain: 9 per batch row to stage the sums, 16 to write them out;
//   exchange: two cluster barriers and (S - 1) / S of the sums at 13 B per clock, in place of writing them all out.
static WsShape ws_choose(const TcspMat* mats, int nmat, int cols, int n, bool tiled) {
    const int* clusters = ws_max_clusters();
    const int steps = (cols + kWsStepK - 1) / kWsStepK;
    WsShape best{};
    double best_cost = 1e30;
    for (int mh = 1; mh <= (tiled ? 2 : 1); ++mh) {
        if (g_ws_mh && tiled && mh != g_ws_mh) continue;
        long long tiles = 0;
        for (int i = 0; i < nmat; ++i) tiles += (mats[i].rows + mh * kWsTileM - 1) / (mh * kWsTileM);
        const int max_nt = mh == 2 ? 240 : 256;
        const int first = (n + max_nt - 1) / max_nt;
        // a few cuts of the batch; of short blocks, where start and drain are most of the time, as many as run at once (384 x 640,
        // n = 900, int32: 5.5 us in blocks of 144 rows, 4.9 in blocks of 64; at six steps or more narrower blocks lose)
        const int more = steps <= 4 ? clusters[1] : 0;
        for (int nn = first;; ++nn) {
            const int nt = ((n + nn - 1) / nn + 15) / 16 * 16;
            if (nn > first && (nt < 64 || (nn > first + 3 && tiles * nn > more))) break;
            if (nt > max_nt) continue;
            const long long blocks = tiles * ((n + nt - 1) / nt);
            const double step = mh == 2 ? fmax(1250.0, 370.0 + 5.6 * nt) : fmax(690.0, 330.0 + 2.8 * nt);
            for (int S = 1; S <= (mh == 1 ? kWsMaxSplit : 1) && S <= steps; ++S) {
                const double waves = ceil(static_cast<double>(blocks) / clusters[S]);
                const double out = S > 1 ? 2800.0 + 36.0 * nt * (S - 1) / S : 16.0 * nt * mh;
                const double cost = waves * (4500.0 + (steps + S - 1) / S * step + 9.0 * nt * mh + out);
                if (cost < best_cost) {
                    best_cost = cost;
                    best.mh = mh;
                    best.nt = nt;
                    best.split = S;
                }
            }
        }
    }
    ws_rings(best, tiled);
    return best;
}

int gemm_tcsp_ws_launch(const TcspMat* mats, int nmat, const int8_t* X, const float* absmax, int cols, int n, void* stream) {
    const char* name = "spb_sparse_ternary_gemm(tcgen05.sp)";
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    bool tiled = cols % 16 == 0 && al(X), signs16 = true, signs8 = cols % 128 == 0;
    for (int i = 0; i < nmat; ++i) {
        tiled = tiled && al(mats[i].meta) && mats[i].meta_stride % 4 == 0;
        signs16 = signs16 && al(mats[i].values) && mats[i].values_stride % 4 == 0;
        signs8 = signs8 && (reinterpret_cast<uintptr_t>(mats[i].values) & 7u) == 0 && mats[i].values_stride % 2 == 0;
    }
    tiled = tiled && (signs16 || signs8);
    WsArgs a{};
    alignas(64) WsMaps maps{};
    WsShape c = ws_choose(mats, nmat, cols, n, tiled);
    auto encode_all = [&] {
        bool good = ws_map(&maps.x, CU_TENSOR_MAP_DATA_TYPE_UINT8, X, cols, n, cols, 128, c.nt, CU_TENSOR_MAP_SWIZZLE_128B);
        for (int i = 0; i < nmat && good; ++i)
            good = ws_map(&maps.meta[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, mats[i].meta, (cols + 31) / 32, mats[i].rows,
                          static_cast<size_t>(mats[i].meta_stride) * 4, 16, c.mh * kWsTileM, CU_TENSOR_MAP_SWIZZLE_64B) &&
                   (!signs16 || ws_map(&maps.values[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, mats[i].values, (cols + 63) / 64, mats[i].rows,
                          static_cast<size_t>(mats[i].values_stride) * 4, 8, c.mh * kWsTileM, CU_TENSOR_MAP_SWIZZLE_32B));
        return good;
    };
    if (tiled && !encode_all()) {
        tiled = false;
        c = ws_choose(mats, nmat, cols, n, tiled);
    }
    a.X = X;
    a.absmax = absmax;
    a.nmat = nmat;
    a.cols = cols;
    a.n = n;
    a.nt = c.nt;
    a.mh = c.mh;
    a.sa = c.sa;
    a.sb = c.sb;
    a.sw = c.sw;
    a.split = c.split;
    int tiles = 0;
    for (int i = 0; i < nmat; ++i) {
        a.m[i] = WsMat{mats[i].meta, mats[i].values, mats[i].out, mats[i].gamma, mats[i].rows, mats[i].meta_stride,
                       mats[i].values_stride, tiles};
        tiles += (mats[i].rows + c.mh * kWsTileM - 1) / (c.mh * kWsTileM);
    }
    a.tmem_cols = 32;
    while (a.tmem_cols < c.mh * (c.nt + 8 * c.sa)) a.tmem_cols <<= 1;
    a.timeouts = timeout_counter();
    a.wait_cycles = kWsWaitCycles;
    using Kernel = void (*)(WsArgs, WsMaps);
    static const Kernel kernels[4][2][2] = {  // layout, half output, four rows on a boundary
        {{gemm_tcsp_ws_kernel<false, kTiled, false>, gemm_tcsp_ws_kernel<false, kTiled, true>},
         {gemm_tcsp_ws_kernel<true, kTiled, false>, gemm_tcsp_ws_kernel<true, kTiled, true>}},
        {{gemm_tcsp_ws_kernel<false, kAny, false>, gemm_tcsp_ws_kernel<false, kAny, true>},
         {gemm_tcsp_ws_kernel<true, kAny, false>, gemm_tcsp_ws_kernel<true, kAny, true>}},
        {{gemm_tcsp_ws_kernel<false, kSigns8, false>, gemm_tcsp_ws_kernel<false, kSigns8, true>},
         {gemm_tcsp_ws_kernel<true, kSigns8, false>, gemm_tcsp_ws_kernel<true, kSigns8, true>}},
        {{gemm_tcsp_ws_kernel<false, kEdge, false>, gemm_tcsp_ws_kernel<false, kEdge, true>},
         {gemm_tcsp_ws_kernel<true, kEdge, false>, gemm_tcsp_ws_kernel<true, kEdge, true>}}};
    bool rows4 = true;
    for (int i = 0; i < nmat; ++i)
        rows4 = rows4 && mats[i].rows % 4 == 0 && (reinterpret_cast<uintptr_t>(mats[i].out) & (absmax ? 7u : 15u)) == 0;
    const Kernel kernel = kernels[!tiled ? kAny : cols % 128 ? kEdge : signs16 ? kTiled : kSigns8][absmax != nullptr][rows4];
    if (int rc = ensure_dynamic_smem(name, kernel, c.smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, (n + c.nt - 1) / c.nt, c.split);
    cfg.blockDim = dim3(tiled ? kWsThreadsTiled : kWsThreadsAny);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (c.split > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = c.split;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, a, maps);
    if (err != cudaSuccess) {
        cudaGetLastError();
        return fail(SPB_E_CUDA, "%s: launch failed: %s", name, cudaGetErrorString(err));
    }
    return SPB_OK;
}

}  // namespace spb

extern "C" int spb_debug_bounded_wait_selftest(long long limit_cycles, void* stream) {
    using namespace spb;
    int* counter = timeout_counter();
    if (!counter) return fail(SPB_E_CUDA, "spb_debug_bounded_wait_selftest: no timeout counter");
    const long long limit = limit_cycles < 1000 ? 1000 : limit_cycles > kWsWaitCycles ? kWsWaitCycles : limit_cycles;
    const int before = timeouts_now();
    ws_wait_selftest_kernel<<<1, 128, 0, static_cast<cudaStream_t>(stream)>>>(counter, limit);
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (err != cudaSuccess) return fail(SPB_E_CUDA, "spb_debug_bounded_wait_selftest: %s", cudaGetErrorString(err));
    if (timeouts_now() != before)
        return fail(SPB_E_TIMEOUT, "spb_debug_bounded_wait_selftest: the wait ran out after %lld cycles, as it must", limit);
    return SPB_OK;
}

extern "C" int spb_set_gemm_row_halves(int halves) {
    const int old = spb::g_ws_mh;
    spb::g_ws_mh = halves == 1 || halves == 2 ? halves : 0;
    return old;
}
