// Small-batch sparse-ternary product on the warp-level sparse MMA (mma.sp m16n8k64, int8), sm_100a, for up to three matrices of
// one width on the same activation rows (q, k and v of a few prompt tokens, gate and up).
//
//   Y[j, r] = sum_c W[r, c] * X[j, c]      W: rows x cols compressed 2:4 ternary, X: n x cols int8, n small
//
// The same scheme as the GEMV on this instruction (gemv_mmasp.cu): the raw weight slab of a block comes
// in by 16-byte asynchronous copies, bitmap words are turned into index pairs and sign nibbles into
// +1 / -1 bytes in registers, and the N = 8 columns of the instruction, which the GEMV fills with copies
// of one vector, carry eight different activation rows here.  A warp re-encodes a step (64 columns of 16
// rows) once and issues one MMA per tile of eight activation rows.  The reference has no kernel of its own for this (its batched path hands a dense copy
// to cuSPARSELt, src/cusparselt_backend.cu:186-207).
//
// Work split: a block of eight warps owns RB row blocks of 16 weight rows x KS warps, each warp a range of
// steps (RB * KS = 8); blockIdx.y selects the tiles of activation rows (NT tiles of 8 per block, as many
// as fit in shared memory next to the slab).  Activations are staged after the dependency wait, permuted
// so that a lane's four B registers of a step are 16 contiguous bytes; row pitch = cols + 64 bytes, which
// keeps the 16-byte reads of a quarter warp (two activation rows x four lanes) on distinct banks.
#include "gemm_tcsp_ws.cuh"

namespace spb {

constexpr int kGqThreads = 256;
constexpr int kGqWarps = kGqThreads / 32;
constexpr int kGqSignLutBytes = 16 * 32 * 4;  // 2 KB on a 2 KB boundary
constexpr int kGqMaxTiles = 4;

struct GqMat {
    const uint32_t* meta;
    const uint32_t* values;
    void* out;  // [n, rows] int32 sums or half
    float gamma;
    int rows, meta_stride, values_stride;
    int blk0;  // first block of this matrix in the grid
};
struct GqArgs {
    GqMat m[kWsMaxMats];
    int nmat;
    const int8_t* X;      // [n, cols]
    const float* absmax;  // row scales of the half outputs
    int cols, n;
    int steps;    // cols / 64
    int ks;       // warps per row block (power of two <= 8)
    int ks_log2;
    int rb;       // row blocks per thread block = 8 / ks
    int spw;      // steps per warp
    int mpitch;   // shared-memory row pitch of the bitmap words, in words (= 4 mod 32)
    int vpitch;   // same for the sign words
    int xpitch;   // shared-memory pitch of an activation row, bytes (cols + 64)
};

__device__ __forceinline__ uint32_t gq_index_pairs(uint32_t m) {
    // eight bitmaps (two of four bits set each) -> eight index pairs {low index | high index << 2}
    const uint32_t mr = m >> 1, ml = m << 1;
    const uint32_t t1 = (0x11111111u & (~m & mr)) | (~0x11111111u & (mr | ~m));
    const uint32_t t2 = (0x22222222u & (~ml & ~m)) | (~0x22222222u & (m | ml));
    return (t1 & 0x55555555u) | (t2 & 0xAAAAAAAAu);
}

__device__ __forceinline__ uint32_t gq_lds(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// NT = tiles of eight activation rows per block.
// HALF_OUT: the epilogue writes the scaled half output instead of the int32 sums
template <int NT, bool HALF_OUT>
__global__ void __launch_bounds__(kGqThreads, 2) gemm_mmasp_kernel(const GqArgs a) {
    extern __shared__ uint8_t gq_raw[];
    // 2 KB-aligned: [sign table 2 KB][bitmap rows: 16 rb x mpitch words][sign rows: 16 rb x vpitch words]
    //               [activations, permuted: 8 NT rows x xpitch bytes; reused for the partial sums at the end]
    const uint32_t raw_s = static_cast<uint32_t>(__cvta_generic_to_shared(gq_raw));
    const uint32_t base_s = (raw_s + 2047u) & ~2047u;
    uint8_t* base = gq_raw + (base_s - raw_s);
    const int nrows_blk = 16 * a.rb;
    const uint32_t ms_s = base_s + kGqSignLutBytes;
    const uint32_t vs_s = ms_s + static_cast<uint32_t>(nrows_blk * a.mpitch) * 4u;
    const uint32_t xs_s = vs_s + static_cast<uint32_t>(nrows_blk * a.vpitch) * 4u;
    volatile int* red = reinterpret_cast<volatile int*>(base + (xs_s - base_s));  // [warp][16 rows][8 NT] after the loop

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);  // through a shuffle: known to be uniform over the warp
    int mi = 0;
    if (a.nmat > 1 && static_cast<int>(blockIdx.x) >= a.m[1].blk0) mi = 1;
    if (a.nmat > 2 && static_cast<int>(blockIdx.x) >= a.m[2].blk0) mi = 2;
    const GqMat m = mi == 0 ? a.m[0] : mi == 1 ? a.m[1] : a.m[2];
    const int row0 = (static_cast<int>(blockIdx.x) - m.blk0) * nrows_blk;
    const int valid = min(nrows_blk, m.rows - row0);
    const int j0 = blockIdx.y * 8 * NT;                       // first activation row of this block
    const uint32_t mbytes = static_cast<uint32_t>(a.cols >> 3), vbytes = static_cast<uint32_t>(a.cols >> 4);

    // the raw slab: 16-byte asynchronous copies, a warp per row, consecutive lanes on consecutive chunks
    {
        const int mch = static_cast<int>(mbytes >> 4), cpr = mch + static_cast<int>(vbytes >> 4);
        for (int k = lane; k < cpr; k += 32) {
            const bool is_m = k < mch;
            const uint8_t* src = is_m ? reinterpret_cast<const uint8_t*>(m.meta) + k * 16
                                      : reinterpret_cast<const uint8_t*>(m.values) + (k - mch) * 16;
            const size_t src_pitch = static_cast<size_t>(is_m ? m.meta_stride : m.values_stride) * 4u;
            const uint32_t dst = is_m ? ms_s + static_cast<uint32_t>(k) * 16u : vs_s + static_cast<uint32_t>(k - mch) * 16u;
            const uint32_t dst_pitch = static_cast<uint32_t>(is_m ? a.mpitch : a.vpitch) * 4u;
            src += static_cast<size_t>(row0 + warp) * src_pitch;
            for (int r = warp; r < valid; r += kGqWarps) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + static_cast<uint32_t>(r) * dst_pitch), "l"(src)
                             : "memory");
                src += kGqWarps * src_pitch;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // sign table: entry (nibble n, lane l) at n * 128 + l * 4, byte b = -1 if bit b of n is set, else +1
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint32_t i = tid + j * kGqThreads;
        const uint32_t t = ((i >> 5) * 0x00204081u) & 0x01010101u;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(base_s + i * 4u), "r"((t * 0xFEu) | 0x01010101u) : "memory");
    }

    const int g = lane >> 2, tig = lane & 3;
    const int rbi = warp >> a.ks_log2, kq = warp & (a.ks - 1);
    const int s_begin = kq * a.spw, s_end = min(a.steps, s_begin + a.spw);
    const uint32_t lane_or = base_s | (static_cast<uint32_t>(lane) << 2);
    const uint32_t rot_lo = (static_cast<uint32_t>(tig) * 4u + 25u) & 31u, rot_hi = (static_cast<uint32_t>(tig) * 4u + 9u) & 31u;
    uint32_t me_p = ms_s + static_cast<uint32_t>((rbi * 16 + g + 8 * (tig & 1)) * a.mpitch + (tig >> 1) + 2 * s_begin) * 4u;
    uint32_t v0_p = vs_s + static_cast<uint32_t>((rbi * 16 + g) * a.vpitch + s_begin) * 4u;
    const uint32_t v_half = static_cast<uint32_t>(8 * a.vpitch) * 4u;
    // B registers of a step for tile t: 16 bytes at activation row 8 t + g, step s, lane slot tig
    uint32_t xq_p = xs_s + static_cast<uint32_t>(g) * static_cast<uint32_t>(a.xpitch) + static_cast<uint32_t>(tig) * 16u +
                    static_cast<uint32_t>(s_begin) * 64u;
    const uint32_t x_tile = 8u * static_cast<uint32_t>(a.xpitch);

    // ---- after the dependency: activations, permuted: xs[row][step][tig][j][0..3] = X[row][64 step + 16 j + 4 tig ..+3];
    //      rows past n are zero ---------------------------------------------------------------------------------------
    grid_dep_wait();
    grid_dep_launch();
    {
        const int cpr = a.cols >> 4;  // 16-byte chunks per activation row
        for (int q = tid; q < 8 * NT * cpr; q += kGqThreads) {
            const int jr = q / cpr, c = q - jr * cpr;
            uint4 xv = make_uint4(0, 0, 0, 0);
            if (j0 + jr < a.n) xv = __ldg(reinterpret_cast<const uint4*>(a.X + static_cast<size_t>(j0 + jr) * a.cols) + c);
            const uint32_t s = static_cast<uint32_t>(c) >> 2, j = static_cast<uint32_t>(c) & 3u;
            const uint32_t d = xs_s + static_cast<uint32_t>(jr) * static_cast<uint32_t>(a.xpitch) + s * 64u + j * 4u;
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(d), "r"(xv.x) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(d + 16u), "r"(xv.y) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(d + 32u), "r"(xv.z) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(d + 48u), "r"(xv.w) : "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the slab, the table and the activations are visible

    int acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0;
    // One step = 64 columns of 16 weight rows: re-encode once, one MMA per tile of activation rows.  Metadata
    // register of lane (g, tig): the index pairs of bitmap word 2 s + (tig >> 1) of row g + 8 (tig & 1).
    auto step = [&](uint32_t w0, uint32_t w1, uint32_t me_off, uint32_t x_off) {
        const uint32_t e = gq_index_pairs(gq_lds(me_p + me_off));
        const uint32_t a0 = gq_lds((__funnelshift_r(w0, w0, rot_lo) & 0x780u) | lane_or);
        const uint32_t a1 = gq_lds((__funnelshift_r(w1, w1, rot_lo) & 0x780u) | lane_or);
        const uint32_t a2 = gq_lds((__funnelshift_r(w0, w0, rot_hi) & 0x780u) | lane_or);
        const uint32_t a3 = gq_lds((__funnelshift_r(w1, w1, rot_hi) & 0x780u) | lane_or);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            uint32_t b0, b1, b2, b3;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                         : "r"(xq_p + x_off + static_cast<uint32_t>(t) * x_tile));
            asm volatile(
                "mma.sp::ordered_metadata.sync.aligned.m16n8k64.row.col.s32.s8.s8.s32 "
                "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9, %10, %11}, {%0, %1, %2, %3}, %12, 0x0;"
                : "+r"(acc[t][0]), "+r"(acc[t][1]), "+r"(acc[t][2]), "+r"(acc[t][3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(b2), "r"(b3), "r"(e));
        }
    };
    auto advance = [&](uint32_t steps) {
        me_p += 8u * steps;
        v0_p += 4u * steps;
        xq_p += 64u * steps;
    };
    int st = s_begin;
    for (; st < s_end && (st & 3) != 0; ++st) {
        step(gq_lds(v0_p), gq_lds(v0_p + v_half), 0u, 0u);
        advance(1u);
    }
    for (; st + 4 <= s_end; st += 4) {  // four steps share one 16-byte read of each row's sign words
        uint4 w0, w1;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w0.x), "=r"(w0.y), "=r"(w0.z), "=r"(w0.w) : "r"(v0_p));
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w1.x), "=r"(w1.y), "=r"(w1.z), "=r"(w1.w) : "r"(v0_p + v_half));
        step(w0.x, w1.x, 0u, 0u);
        step(w0.y, w1.y, 8u, 64u);
        step(w0.z, w1.z, 16u, 128u);
        step(w0.w, w1.w, 24u, 192u);
        advance(4u);
    }
    for (; st < s_end; ++st) {
        step(gq_lds(v0_p), gq_lds(v0_p + v_half), 0u, 0u);
        advance(1u);
    }

    // Partial sums of the KS warps meet in shared memory (the activation area is free once everybody is done
    // with it): red[warp][row 0..15][column 0..8 NT).  Lane (g, tig) holds rows g, g + 8 x columns 2 tig, 2 tig + 1.
    __syncthreads();
    constexpr int NC = 8 * NT;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        volatile int* r0 = red + (warp * 16 + g) * NC + 8 * t + 2 * tig;
        r0[0] = acc[t][0];
        r0[1] = acc[t][1];
        r0[8 * NC] = acc[t][2];
        r0[8 * NC + 1] = acc[t][3];
    }
    __syncthreads();
    for (int o = tid; o < NC * nrows_blk; o += kGqThreads) {
        const int jc = o / nrows_blk, r = o - jc * nrows_blk;  // consecutive threads on consecutive weight rows
        if (r < valid && j0 + jc < a.n) {
            const int rblk = r >> 4, rr = r & 15;
            int sum = 0;
            for (int k = 0; k < a.ks; ++k) sum += red[(((rblk << a.ks_log2) + k) * 16 + rr) * NC + jc];
            const size_t o = static_cast<size_t>(j0 + jc) * m.rows + row0 + r;
            if (HALF_OUT)
                static_cast<__half*>(m.out)[o] = __float2half_rn(__fmul_rn(static_cast<float>(sum), dequant_scale(m.gamma, a.absmax[j0 + jc])));
            else
                static_cast<int32_t*>(m.out)[o] = sum;
        }
    }
}

// Whether the form applies: whole 16-byte sign rows (cols % 256 == 0), 16-byte aligned rows everywhere.
bool gemm_mmasp_supported(const TcspMat* mats, int nmat, const int8_t* X, int cols, int n) {
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    bool ok = n > 0 && n <= 4096 && cols > 0 && cols % 256 == 0 && cols <= 16384 && al16(X);
    for (int i = 0; i < nmat; ++i)
        ok = ok && mats[i].rows > 0 && mats[i].meta_stride % 4 == 0 && mats[i].values_stride % 4 == 0 && al16(mats[i].meta) &&
             al16(mats[i].values);
    return ok;
}

// Work split and shared memory of a launch: pointers and rows aside, all of GqArgs.
struct GqShape {
    int blocks_x, blocks_y, nt;
    size_t smem;
};
static GqShape gq_shape(GqArgs& a, const TcspMat* mats, int nmat, int cols, int n) {
    a.cols = cols;
    a.n = n;
    a.nmat = nmat;
    a.steps = cols / 64;
    int row_blocks = 0;
    for (int i = 0; i < nmat; ++i) row_blocks += (mats[i].rows + 15) / 16;
    a.ks = 8;
    while (a.ks > 1 && a.steps / a.ks < 16) a.ks >>= 1;
    while (a.ks < 8 && row_blocks * a.ks < 2 * sm_count() && a.steps / (2 * a.ks) >= 8) a.ks <<= 1;
    while (a.ks > a.steps) a.ks >>= 1;
    a.rb = kGqWarps / a.ks;
    a.ks_log2 = a.ks == 8 ? 3 : a.ks == 4 ? 2 : a.ks == 2 ? 1 : 0;
    a.spw = (a.steps + a.ks - 1) / a.ks;
    auto pitch = [](int words) { return words + ((4 - words % 32) + 32) % 32; };  // smallest >= words that is 4 mod 32
    a.mpitch = pitch(cols / 32);
    a.vpitch = pitch(cols / 64);
    a.xpitch = cols + 64;
    // tiles of eight activation rows per block: all of them if the activations (and, later, the partial sums)
    // fit in about 100 KB next to the slab, else fewer and more blocks along y
    const int tiles = (n + 7) / 8;
    const size_t slab = static_cast<size_t>(16 * a.rb) * (a.mpitch + a.vpitch) * 4;
    GqShape s{};
    s.nt = tiles < kGqMaxTiles ? tiles : kGqMaxTiles;
    auto xbytes = [&](int t) {
        const size_t act = static_cast<size_t>(8 * t) * a.xpitch, part = static_cast<size_t>(kGqWarps) * 16 * 8 * t * 4;
        return act > part ? act : part;
    };
    while (s.nt > 1 && (s.nt == 3 || 2048 + kGqSignLutBytes + slab + xbytes(s.nt) > 110 * 1024)) --s.nt;
    s.smem = 2048 + kGqSignLutBytes + slab + xbytes(s.nt);
    for (int i = 0; i < nmat; ++i) {
        a.m[i] = GqMat{mats[i].meta, mats[i].values, mats[i].out, mats[i].gamma, mats[i].rows, mats[i].meta_stride, mats[i].values_stride, s.blocks_x};
        s.blocks_x += (mats[i].rows + 16 * a.rb - 1) / (16 * a.rb);
    }
    s.blocks_y = (tiles + s.nt - 1) / s.nt;
    return s;
}

// Whether this form is the faster one where it applies.  It starts sooner than the tcgen05 form (some 3 against 4 us for a
// small product) and pays a pass of re-encoding per eight or sixteen batch rows (us, this form / tcgen05, half output where
// not said):
//   up to 8 batch rows while its blocks run at once, two per SM, or the matrix is small: 6912 x 6912, n = 2: 7.3 / 10.0;
//     8192 x 6912, n = 8: 8.2 / 10.2;  2560 x 14336, n = 8 (a wave and a bit, one block per SM): 13.3 / 9.2;  28672 x 5632,
//     n = 2: 20.3 / 16.0;  a half output's scales cost it more on short rows: 2560 x 512, n = 8: 3.7 / 3.6, 2560 x 256,
//     n = 8, int32: 2.9 / 3.2;
//   9 to 32 while no SM has a second block, a row block is shared by two warps or more and a block takes at most sixteen batch
//     rows: 1001 x 6912, n = 16: 5.1 / 6.3;  256 x 5632, n = 32: 4.7 / 5.5;  14336 x 2048, n = 16: 10.0 / 6.7;  640 x 2560,
//     n = 32: 8.8 / 5.4;  shorter rows for few of them or int32: 2048 x 2560, n = 9: 4.9 / 5.6;  6912 x 2560, n = 16: 7.2 / 6.7;
//     2048 x 1024, n = 9, int32: 3.8 / 4.5, half 4.3 / 4.3.
bool gemm_mmasp_preferred(const TcspMat* mats, int nmat, int cols, int n, bool half_out) {
    if (n > 32) return false;
    GqArgs a{};
    const GqShape s = gq_shape(a, mats, nmat, cols, n);
    const long long blocks = static_cast<long long>(s.blocks_x) * s.blocks_y;
    long long rows = 0;
    for (int i = 0; i < nmat; ++i) rows += mats[i].rows;
    if (n > 8)
        return cols >= (!half_out ? 1024 : rows <= 2048 ? 2048 : 4096) && a.ks >= 2 && s.nt <= 2 && blocks <= sm_count();
    if (half_out && cols < 1024 && n > 4 && rows <= 8192) return false;
    const int per_sm = s.smem > 112 * 1024 ? 1 : 2;
    return blocks <= static_cast<long long>(per_sm) * sm_count() || (cols < 8192 && rows * cols <= 60ll * 1000 * 1000);
}

// absmax: row scales, the outputs are half; without, int32 sums
int gemm_mmasp_launch(const TcspMat* mats, int nmat, const int8_t* X, const float* absmax, int cols, int n, void* stream) {
    const char* name = "spb_sparse_ternary_gemm(mma.sp)";
    GqArgs a{};
    const GqShape s = gq_shape(a, mats, nmat, cols, n);
    a.X = X;
    a.absmax = absmax;
    if (s.smem > 200 * 1024) return fail(SPB_E_UNSUPPORTED, "%s: %d columns do not fit", name, cols);
    void (*kernel)(GqArgs) = s.nt == 1 ? gemm_mmasp_kernel<1, false> : s.nt == 2 ? gemm_mmasp_kernel<2, false> : gemm_mmasp_kernel<4, false>;
    if (absmax) kernel = s.nt == 1 ? gemm_mmasp_kernel<1, true> : s.nt == 2 ? gemm_mmasp_kernel<2, true> : gemm_mmasp_kernel<4, true>;
    if (int rc = ensure_dynamic_smem(name, kernel, s.smem)) return rc;
    return launch(name, kernel, dim3(s.blocks_x, s.blocks_y), dim3(kGqThreads), s.smem, stream, a);
}

}  // namespace spb
