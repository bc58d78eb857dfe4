// Magnitude 2:4 pruning + ternary sign extraction + packing of a float32 weight matrix on the GPU,
// byte-identical to the reference's converter (python/convert_model.py:88-138 generate_24_mask and
// quantize_ternary_absmean, :270-283 the zero-at-mask fix, :141-207 pack_sparse_ternary).
//
// What the converter's five steps come to, per group of four consecutive weights of a row:
//   * kept positions = the two largest |w|; on equal magnitudes the HIGHER index is kept (a stable ascending
//     argsort leaves equal elements in index order and the top two are taken from its end);
//   * a kept weight packs as -1 exactly when w < 0: RoundClip(w / gamma) of a negative weight is -1 or 0, a
//     kept 0 is forced to the sign of w, and w >= 0 (including -0.0) packs as +1 — so the packed bits do not
//     depend on gamma at all;
//   * gamma = mean |w| goes to the manifest only.  It is accumulated here in double precision (optional);
//     numpy's float32 pairwise sum can differ from it in the last bits, so a caller that needs the manifest
//     byte-identical computes gamma with numpy.
//
// A unit is 16 groups of a row (two bitmap words, one sign word) and a half-warp's coalesced load: lane l holds group l of
// the unit.  A warp takes 16 units, eight loads in flight per lane; the eight bitmaps of a lane sit in one register, and
// three exchanges transpose the 8 x 8 of every eight lanes, which leaves each lane one whole word.  The top two of four come
// from the signs of six integer differences (|w| as bits, no overflow) and four majorities, collected bit by bit with funnel
// shifts: some 14 instructions a group.  A warp that meets a NaN, where comparisons of floats and of their bits part, decides
// those groups by float comparisons.
//
// Bound: the floats through HBM once.  One thread per unit (256 consecutive bytes per lane, 24 comparisons and additions a
// group, an atomic per warp on the one sum) took 84.6 us for 8192 x 8192, this form 58.6 us (4.8 TB/s).  The grid is a few blocks per SM
// that walk the units, so the sum takes one atomic per block.
#include "spb_common.cuh"

namespace spb {

constexpr int kPackThreads = 256;
constexpr int kPackBlocksPerSm = 4;

// bitmap | sign pair << 4 of a group by comparisons of floats: the definition above, for any values
__device__ __noinline__ uint32_t pack_group_compare(float v0, float v1, float v2, float v3) {
    const float v[4] = {v0, v1, v2, v3};
    uint32_t bitmap = 0, signs = 0;
    int seen = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int before = 0;  // rank in the stable ascending order
#pragma unroll
        for (int j = 0; j < 4; ++j) before += (fabsf(v[j]) < fabsf(v[i])) || (fabsf(v[j]) == fabsf(v[i]) && j < i);
        if (before >= 2) {
            bitmap |= 1u << i;
            if (v[i] < 0.0f) signs |= 1u << seen;
            ++seen;
        }
    }
    return bitmap | signs << 4;
}

__device__ __forceinline__ uint32_t maj(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (c & (a | b)); }

// Eight lanes hold an 8 x 8 matrix of B-bit fields, lane i row i; afterwards lane i holds column i.
template <int B>
__device__ __forceinline__ uint32_t transpose8(uint32_t r, int lane) {
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
        // fields whose index has bit d set (of a lane without it) change places with those without (of a lane with it)
        uint32_t low = 0;
#pragma unroll
        for (int f = 0; f < 8; ++f)
            if (!(f & d)) low |= ((1u << B) - 1u) << (B * f);
        const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, r, d);
        r = (lane & d) ? ((r & (low << (B * d))) | ((other >> (B * d)) & low)) : ((r & low) | ((other & low) << (B * d)));
    }
    return r;
}

// row and place in the row of unit u (a 64-bit division costs as much as the packing of several groups)
__device__ __forceinline__ void row_of(long long u, int upr, int& row, int& tc) {
    row = u <= 0xFFFFFFFFll ? static_cast<int>(static_cast<uint32_t>(u) / static_cast<uint32_t>(upr)) : static_cast<int>(u / upr);
    tc = static_cast<int>(u - static_cast<long long>(row) * upr);
}

template <bool VEC>
__global__ void __launch_bounds__(kPackThreads, kPackBlocksPerSm) prune_pack_kernel(
    const float* __restrict__ w, int rows, int cols, size_t w_row_stride, uint32_t* __restrict__ meta,
    uint32_t* __restrict__ values, int meta_stride, int values_stride, double* __restrict__ abs_sum) {
    __shared__ double sums[kPackThreads / 32];
    grid_dep_wait();  // (dependents are let in by the end of the grid: the GEMV kernels read weights before their own wait)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = cols >> 2, upr = (groups + 15) >> 4;  // units per row
    const long long units = static_cast<long long>(rows) * upr;
    const long long step = static_cast<long long>(gridDim.x) * (kPackThreads / 32) * 16;
    double local = 0.0;
    for (long long u0 = (static_cast<long long>(blockIdx.x) * (kPackThreads / 32) + warp) * 16; u0 < units; u0 += step) {
        const long long uh = u0 + (lane >> 4);  // this half-warp's unit of load 0; load k: 2 k units on
        int row, tc;
        row_of(uh, upr, row, tc);
        float4 f[8];
        uint32_t valid = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int g = tc * 16 + (lane & 15);
            f[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < rows && g < groups) {
                valid |= 1u << k;
                const float* src = w + static_cast<size_t>(row) * w_row_stride + static_cast<size_t>(g) * 4;
                if (VEC) {
                    f[k] = __ldcs(reinterpret_cast<const float4*>(src));
                } else {
                    f[k] = make_float4(__ldcs(src), __ldcs(src + 1), __ldcs(src + 2), __ldcs(src + 3));
                }
            }
            tc += 2;
            while (tc >= upr) {
                tc -= upr;
                ++row;
            }
        }
        uint32_t bm = 0, sg = 0, top = 0;
#pragma unroll
        for (int k = 7; k >= 0; --k) {
            const float v[4] = {f[k].x, f[k].y, f[k].z, f[k].w};
            int a[4];
            uint32_t s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i] = __float_as_int(fabsf(v[i]));
                s[i] = __float_as_uint(v[i] + 0.0f);  // -0 + 0 = +0: the top bit says v < 0
                top = max(top, static_cast<uint32_t>(a[i]));
                local += static_cast<double>(fabsf(v[i]));
            }
            // top bit of p_ij: |v_i| > |v_j|, i < j, so i comes after j; else (equality too) j after i
            const uint32_t p01 = a[1] - a[0], p02 = a[2] - a[0], p03 = a[3] - a[0], p12 = a[2] - a[1], p13 = a[3] - a[1], p23 = a[3] - a[2];
            const uint32_t k0 = maj(p01, p02, p03), k1 = maj(~p01, p12, p13), k2 = maj(~p02, ~p12, p23), k3 = maj(~p03, ~p13, ~p23);
            const uint32_t lo = (k0 & s[0]) | (~k0 & ((k1 & s[1]) | (~k1 & s[2])));
            const uint32_t hi = (k3 & s[3]) | (~k3 & ((k2 & s[2]) | (~k2 & s[1])));
            bm = __funnelshift_l(k3, bm, 1);
            bm = __funnelshift_l(k2, bm, 1);
            bm = __funnelshift_l(k1, bm, 1);
            bm = __funnelshift_l(k0, bm, 1);
            sg = __funnelshift_l(hi, sg, 1);
            sg = __funnelshift_l(lo, sg, 1);
        }
        if (__any_sync(0xFFFFFFFFu, top > 0x7F800000u)) {
            bm = sg = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t t = pack_group_compare(f[k].x, f[k].y, f[k].z, f[k].w);
                bm |= (t & 15u) << (4 * k);
                sg |= (t >> 4) << (2 * k);
            }
        }
        if (valid != 0xFFu) {  // groups past a row's end pack as zero bits
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (!(valid & (1u << k))) {
                    bm &= ~(15u << (4 * k));
                    sg &= ~(3u << (2 * k));
                }
        }
        bm = transpose8<4>(bm, lane);
        sg = transpose8<2>(sg, lane);
        sg |= __shfl_xor_sync(0xFFFFFFFFu, sg, 8) << 16;  // lanes 0-7 and 16-23: the upper eight groups of their unit
        // lane 8 s + i holds the word of load i, groups 8 (s & 1) .. + 7 of unit 2 i + s / 2
        const long long uo = u0 + 2 * (lane & 7) + (lane >> 4);
        if (uo < units) {
            int orow, otc;
            row_of(uo, upr, orow, otc);
            const int half = (lane >> 3) & 1;
            if (otc * 16 + 8 * half < groups) meta[static_cast<size_t>(orow) * meta_stride + 2 * otc + half] = bm;
            if (!half) values[static_cast<size_t>(orow) * values_stride + otc] = sg;
        }
    }
    if (abs_sum) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) local += __shfl_xor_sync(0xFFFFFFFFu, local, off);
        if (lane == 0) sums[warp] = local;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < kPackThreads / 32; ++i) local += sums[i];
            if (local != 0.0) atomicAdd(abs_sum, local);
        }
    }
}

}  // namespace spb

using namespace spb;

extern "C" int spb_prune_pack_gpu(const float* weights, int rows, int cols, size_t weights_row_stride, uint32_t* meta,
                                  uint32_t* values, int meta_row_stride, int values_row_stride, double* abs_sum,
                                  void* stream) {
    const char* name = "spb_prune_pack_gpu";
    if (rows < 0 || cols < 0) return fail(SPB_E_INVALID, "%s: negative size", name);
    if (rows == 0 || cols == 0) return SPB_OK;
    if (cols % 4 != 0) return fail(SPB_E_INVALID, "%s: cols=%d is not a multiple of 4", name, cols);
    if (!weights || !meta || !values) return fail(SPB_E_INVALID, "%s: null pointer", name);
    if (weights_row_stride < static_cast<size_t>(cols)) return fail(SPB_E_INVALID, "%s: row stride shorter than a row", name);
    if (meta_row_stride < (cols / 4 + 7) / 8 || values_row_stride < (cols / 4 + 15) / 16)
        return fail(SPB_E_INVALID, "%s: row stride shorter than a row", name);
    const long long units = static_cast<long long>(rows) * ((cols / 4 + 15) / 16);
    const long long per_block = 16 * (kPackThreads / 32);
    const long long want = (units + per_block - 1) / per_block;
    const long long cap = static_cast<long long>(sm_count()) * kPackBlocksPerSm;
    const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
    const bool vec = (reinterpret_cast<uintptr_t>(weights) & 15u) == 0 && weights_row_stride % 4 == 0;
    return launch(name, vec ? prune_pack_kernel<true> : prune_pack_kernel<false>, dim3(grid), dim3(kPackThreads), 0, stream,
                  weights, rows, cols, weights_row_stride, meta, values, meta_row_stride, values_row_stride, abs_sum);
}
