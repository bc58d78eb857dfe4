// Causal attention of a prompt chunk: T tokens at positions *d_pos .. *d_pos + T - 1 over the KV cache, as T calls of
// attention_scores_gpu + softmax_gpu + attention_output_gpu (src/kernels/inference_kernels.cu:241-371) give it.
//
// A block takes the G query heads of one KV head and R tiles of 16 tokens, a warp one (head, tile): the 16 tokens are
// the rows of mma.sync m16n8k16.  K and V go through shared memory in tiles of 64 positions, two in flight, read once
// for all warps of the block.  Scores, running maximum, sum and output are fp32.  A weight enters the second product as the sum
// of two halves, value and remainder, of 2^15 times itself: the factor cancels against the sum of the weights, the largest
// weight is still a half, and weights down to 2^-29 of the row's largest keep 22 bits (without it a weight below 2^-14 lost
// bits and one below 2^-25 all of them, while the sum it is divided by still had it).
// Tiles of positions start at multiples of 64 whatever the chunk, and a tile past a row's own position leaves the row
// untouched, so a row's bits do not depend on how a prompt is cut into calls (while V is finite: a block that comes upon other
// values forms its rows again, pa_rows_one_by_one, whose sums are in another order).
//
// Sums on the tensor core are cut off at each addition, not rounded.  Neither product therefore keeps one accumulator for long:
// scores are formed in two chains of four or fewer, a tile of positions gives its part of the output in accumulators of its own,
// which are added up in fp32.  (One accumulator over 4000 positions came out low by some 2^-16 and moved one rounding to half in
// 33; so one in 700, a serial fp32 sum one in 370.  3 % of the time.)
//
// Bound: 20 heads of 128 over 1800 positions keep the tensor pipe busy for half of the active cycles and the chip active for
// 70 % of them (245 blocks of unequal length on 148 SMs).  A block per (head, token) that walks the positions serially, used
// before, re-read K and V once per head and token: 2176 us per chunk of 1024 or 776 tokens; this kernel 75 us, and 66 us since
// full tiles are not masked, a factor of one is not multiplied into the output and the weights are split two at a time.
// Two warps per 16 tokens (32 of a tile's positions each) and clusters of two blocks per 16 tokens (alternate tiles) measured
// the same or slower.
#include "fused_ops.cuh"

namespace spb {

namespace {

constexpr int kPaTile = 64;  // positions per K / V tile
constexpr int kPaRows = 16;  // tokens per warp
constexpr float kPaFactor = 32768.0f;  // of the weights: the largest, this, is a half

__device__ __forceinline__ void pa_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 2^x for x <= 0.  Like exp2f but for results below 2^-126, which come out as zero: next to the row's largest weight, 1, they
// are below every bit of the sums.
__device__ __forceinline__ float pa_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two weights as halves and the halves of what those miss
__device__ __forceinline__ void pa_split(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// A warp's 16 rows position by position, for a block whose outputs are not all finite: an infinity or a NaN of V is to reach the
// rows that see its position, but in a product on the tensor core a weight of zero makes NaN of it, and so do the two halves of
// a weight.  Out of line and not tuned: as a second turn of the kernel's own loop it made that loop 9 % slower.
template <int HD>
__device__ __noinline__ void pa_rows_one_by_one(const __half* __restrict__ Q, const __half* __restrict__ K, const __half* __restrict__ V,
                                                __half* __restrict__ out, int tok0, int T, int start, int num_heads, int head, float scale_log2) {
    constexpr int kDims = HD / 32;
    const int lane = threadIdx.x & 31;
    for (int t = tok0; t < min(tok0 + kPaRows, T); ++t) {
        const __half* q = Q + (static_cast<size_t>(t) * num_heads + head) * HD;
        const int n = start + t + 1;
        float m = -INFINITY, l = 0.0f, o[kDims];
#pragma unroll
        for (int i = 0; i < kDims; ++i) o[i] = 0.0f;
        for (int p0 = 0; p0 < n; p0 += 32) {
            const int p = p0 + lane;
            float s = -INFINITY;
            if (p < n) {
                s = 0.0f;
                const uint4* kr = reinterpret_cast<const uint4*>(K + static_cast<size_t>(p) * HD);
#pragma unroll 4
                for (int c = 0; c < HD / 8; ++c) {
                    const uint4 kv = kr[c], qv = reinterpret_cast<const uint4*>(q)[c];
                    const uint32_t kw[4] = {kv.x, kv.y, kv.z, kv.w}, qw[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&qw[i])), b = __half22float2(*reinterpret_cast<const __half2*>(&kw[i]));
                        s = fmaf(a.x, b.x, s);
                        s = fmaf(a.y, b.y, s);
                    }
                }
                s *= scale_log2;
            }
            float mn = s;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, off));
            mn = fmaxf(m, mn);
            const float corr = exp2f(m - mn), e = p < n ? exp2f(s - mn) : 0.0f;
            m = mn;
            l = l * corr + e;
#pragma unroll
            for (int i = 0; i < kDims; ++i) o[i] *= corr;
            const int seen = min(32, n - p0);
#pragma unroll 4
            for (int r = 0; r < seen; ++r) {
                const float w = __shfl_sync(0xFFFFFFFFu, e, r);
#pragma unroll
                for (int i = 0; i < kDims; ++i) o[i] = fmaf(w, __half2float(V[static_cast<size_t>(p0 + r) * HD + 32 * i + lane]), o[i]);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, off);
#pragma unroll
        for (int i = 0; i < kDims; ++i) out[(static_cast<size_t>(t) * num_heads + head) * HD + 32 * i + lane] = __float2half_rn(o[i] / l);
    }
}

template <int HD>
__global__ void __launch_bounds__(256) prefill_attention_kernel(
    const __half* __restrict__ Q, const __half* __restrict__ K, const __half* __restrict__ V, __half* __restrict__ out,
    int T, int num_heads, int G, int R, int max_seq_len, float scale_log2, const int* __restrict__ d_pos) {
    extern __shared__ __align__(128) uint8_t pa_sm[];  // K tile x 2, V tile x 2
    constexpr int kRowBytes = HD * 2, kTileBytes = kPaTile * kRowBytes;
    grid_dep_launch();
    grid_dep_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nthreads = blockDim.x;
    const int start = *d_pos;
    const int kvh = blockIdx.y, head = kvh * G + warp % G;
    const int btile = (gridDim.x - 1 - blockIdx.x) * R;  // the longest rows first
    const int tok0 = (btile + warp / G) * kPaRows;       // this warp's tokens
    const int last = min(T, (btile + R) * kPaRows) - 1;  // the block's last token
    const int npos = start + last + 1;
    const int ntiles = (npos + kPaTile - 1) / kPaTile;
    const uint32_t sm = static_cast<uint32_t>(__cvta_generic_to_shared(pa_sm));
    const uint8_t* kg = reinterpret_cast<const uint8_t*>(K + static_cast<size_t>(kvh) * max_seq_len * HD);
    const uint8_t* vg = reinterpret_cast<const uint8_t*>(V + static_cast<size_t>(kvh) * max_seq_len * HD);

    auto load_tile = [&](int j) {  // 16-byte pieces, piece c of row r at c ^ (r & 7); positions past the block's last: zero
        const uint32_t kb = sm + (j & 1) * kTileBytes, vb = kb + 2 * kTileBytes;
        for (int i = threadIdx.x; i < kPaTile * (HD / 8); i += nthreads) {
            const int r = i / (HD / 8), c = i % (HD / 8);
            const int p = j * kPaTile + r;
            const uint32_t dst = r * kRowBytes + ((c ^ (r & 7)) << 4);
            const size_t src = static_cast<size_t>(min(p, npos - 1)) * kRowBytes + c * 16;
            const int n = p < npos ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kb + dst), "l"(kg + src), "r"(n) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vb + dst), "l"(vg + src), "r"(n) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_tile(0);

    const int g = lane >> 2, t4 = lane & 3;
    const int ta = min(tok0 + g, T - 1), tb = min(tok0 + g + 8, T - 1);  // rows past the batch repeat its last token
    const int pa = start + ta, pb = start + tb;
    uint32_t qf[HD / 16][4];
    {
        const uint32_t* qa = reinterpret_cast<const uint32_t*>(Q + (static_cast<size_t>(ta) * num_heads + head) * HD) + t4;
        const uint32_t* qb = reinterpret_cast<const uint32_t*>(Q + (static_cast<size_t>(tb) * num_heads + head) * HD) + t4;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
            qf[k][0] = qa[k * 8];
            qf[k][1] = qb[k * 8];
            qf[k][2] = qa[k * 8 + 4];
            qf[k][3] = qb[k * 8 + 4];
        }
    }
    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[i][c] = 0.0f;
    float ma = -INFINITY, mb = -INFINITY, la = 0.0f, lb = 0.0f;

    for (int j = 0; j < ntiles; ++j) {
        if (j + 1 < ntiles) {
            load_tile(j + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t kb = sm + (j & 1) * kTileBytes, vb = kb + 2 * kTileBytes;
        if (tok0 < T && j * kPaTile <= start + min(tok0 + kPaRows, T) - 1) {  // else: every position is past the warp's rows
            float s[kPaTile / 8][4];
#pragma unroll
            for (int nb = 0; nb < kPaTile / 16; ++nb) {
                float c0[2][4] = {}, c1[2][4] = {};
#pragma unroll
                for (int k = 0; k < HD / 16; ++k) {
                    const int r = nb * 16 + (lane & 7) + ((lane >> 4) << 3), c = 2 * k + ((lane >> 3) & 1);
                    uint32_t b[4];
                    pa_ldsm4(b, kb + r * kRowBytes + ((c ^ (r & 7)) << 4));
                    pa_mma(c0[k & 1], qf[k], b[0], b[1]);
                    pa_mma(c1[k & 1], qf[k], b[2], b[3]);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[2 * nb][c] = c0[0][c] + c0[1][c];
                    s[2 * nb + 1][c] = c1[0][c] + c1[1][c];
                }
            }
            if ((j + 1) * kPaTile - 1 > start + tok0) {  // some of the tile's positions are past some of the warp's rows
#pragma unroll
                for (int i = 0; i < kPaTile / 8; ++i) {
                    const int p = j * kPaTile + i * 8 + 2 * t4;
                    if (p > pa) s[i][0] = -INFINITY;
                    if (p + 1 > pa) s[i][1] = -INFINITY;
                    if (p > pb) s[i][2] = -INFINITY;
                    if (p + 1 > pb) s[i][3] = -INFINITY;
                }
            }
            float na = -INFINITY, nb_ = -INFINITY;
#pragma unroll
            for (int i = 0; i < kPaTile / 8; ++i) {
                na = fmaxf(na, fmaxf(s[i][0], s[i][1]));
                nb_ = fmaxf(nb_, fmaxf(s[i][2], s[i][3]));
            }
#pragma unroll
            for (int off = 1; off < 4; off <<= 1) {
                na = fmaxf(na, __shfl_xor_sync(0xFFFFFFFFu, na, off));
                nb_ = fmaxf(nb_, __shfl_xor_sync(0xFFFFFFFFu, nb_, off));
            }
            na = fmaxf(ma, na * scale_log2);  // scale > 0
            nb_ = fmaxf(mb, nb_ * scale_log2);
            // position 0 is visible to every row, so the maxima are finite from the first tile on; past the first few tiles
            // they rarely move, and a factor of one is not multiplied
            if (__any_sync(0xFFFFFFFFu, !(na == ma && nb_ == mb))) {
                const float ca = exp2f(ma - na), cb = exp2f(mb - nb_);
                ma = na;
                mb = nb_;
                la *= ca;
                lb *= cb;
#pragma unroll
                for (int i = 0; i < HD / 8; ++i) {
                    o[i][0] *= ca;
                    o[i][1] *= ca;
                    o[i][2] *= cb;
                    o[i][3] *= cb;
                }
            }
            uint32_t hi[kPaTile / 16][4], lo[kPaTile / 16][4];
#pragma unroll
            for (int kk = 0; kk < kPaTile / 16; ++kk)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float* e = s[2 * kk + h];
                    e[0] = kPaFactor * pa_exp2(fmaf(e[0], scale_log2, -ma));
                    e[1] = kPaFactor * pa_exp2(fmaf(e[1], scale_log2, -ma));
                    e[2] = kPaFactor * pa_exp2(fmaf(e[2], scale_log2, -mb));
                    e[3] = kPaFactor * pa_exp2(fmaf(e[3], scale_log2, -mb));
                    la += e[0] + e[1];
                    lb += e[2] + e[3];
                    pa_split(e[0], e[1], hi[kk][2 * h], lo[kk][2 * h]);
                    pa_split(e[2], e[3], hi[kk][2 * h + 1], lo[kk][2 * h + 1]);
                }
#pragma unroll
            for (int nb = 0; nb < HD / 16; ++nb) {
                float d0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int kk = 0; kk < kPaTile / 16; ++kk) {
                    const int r = kk * 16 + (lane & 15), c = 2 * nb + (lane >> 4);
                    uint32_t b[4];
                    pa_ldsm4_t(b, vb + r * kRowBytes + ((c ^ (r & 7)) << 4));
                    pa_mma(d0, lo[kk], b[0], b[1]);
                    pa_mma(d1, lo[kk], b[2], b[3]);
                    pa_mma(d0, hi[kk], b[0], b[1]);
                    pa_mma(d1, hi[kk], b[2], b[3]);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    o[2 * nb][c] += d0[c];
                    o[2 * nb + 1][c] += d1[c];
                }
            }
        }
        __syncthreads();  // the tile's buffer is free for the load after next
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
        la += __shfl_xor_sync(0xFFFFFFFFu, la, off);
        lb += __shfl_xor_sync(0xFFFFFFFFu, lb, off);
    }
    float z = 0.0f;  // 0 times anything finite
#pragma unroll
    for (int i = 0; i < HD / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) z = fmaf(o[i][c], 0.0f, z);
    if (__syncthreads_or(z != 0.0f)) {
        pa_rows_one_by_one<HD>(Q, reinterpret_cast<const __half*>(kg), reinterpret_cast<const __half*>(vg), out, tok0, T, start, num_heads, head, scale_log2);
        return;
    }
    const float ia = 1.0f / la, ib = 1.0f / lb;
    const int ra = tok0 + g, rb = tok0 + g + 8;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
        const int d = i * 8 + 2 * t4;
        if (ra < T)
            *reinterpret_cast<__half2*>(out + (static_cast<size_t>(ra) * num_heads + head) * HD + d) =
                __halves2half2(__float2half_rn(o[i][0] * ia), __float2half_rn(o[i][1] * ia));
        if (rb < T)
            *reinterpret_cast<__half2*>(out + (static_cast<size_t>(rb) * num_heads + head) * HD + d) =
                __halves2half2(__float2half_rn(o[i][2] * ib), __float2half_rn(o[i][3] * ib));
    }
}

}  // namespace

bool prefill_attention_supported(int num_heads, int num_kv_heads, int head_dim) {
    return num_kv_heads > 0 && num_heads % num_kv_heads == 0 && num_heads / num_kv_heads <= 8 &&
           (head_dim == 64 || head_dim == 128);
}

// Q and out: T rows of num_heads * head_dim half, 16-byte aligned caches (num_kv_heads, max_seq_len, head_dim) half
int prefill_attention(const void* Q, const void* K, const void* V, void* out, int T, int num_heads, int num_kv_heads,
                      int head_dim, int max_seq_len, float scale, const int* d_pos, void* stream) {
    const int G = num_heads / num_kv_heads;
    const int R = max(1, 4 / G);  // four warps or more share a K / V tile, three where G = 3
    const float scale_log2 = scale * 1.44269504088896340736f;
    const size_t smem = 4 * static_cast<size_t>(kPaTile) * head_dim * 2;
    auto kernel = head_dim == 64 ? prefill_attention_kernel<64> : prefill_attention_kernel<128>;
    if (int rc = ensure_dynamic_smem("prefill_attention", kernel, smem)) return rc;
    return launch("prefill_attention", kernel, dim3((T + R * kPaRows - 1) / (R * kPaRows), num_kv_heads), dim3(32 * G * R),
                  smem, stream, static_cast<const __half*>(Q), static_cast<const __half*>(K), static_cast<const __half*>(V),
                  static_cast<__half*>(out), T, num_heads, G, R, max_seq_len, scale_log2, d_pos);
}

}  // namespace spb

extern "C" int spb_debug_prefill_attention(const void* Q, const void* K, const void* V, void* out, int T, int num_heads,
                                           int num_kv_heads, int head_dim, int max_seq_len, float scale, const int* d_pos,
                                           void* stream) {
    using namespace spb;
    const char* name = "spb_debug_prefill_attention";
    if (!Q || !K || !V || !out || !d_pos || T < 1 || max_seq_len < T || !(scale > 0.0f)) return fail(SPB_E_INVALID, "%s: bad arguments", name);
    if (!prefill_attention_supported(num_heads, num_kv_heads, head_dim) ||
        ((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(V) | reinterpret_cast<uintptr_t>(out)) & 15u))
        return fail(SPB_E_UNSUPPORTED, "%s: shape", name);
    return prefill_attention(Q, K, V, out, T, num_heads, num_kv_heads, head_dim, max_seq_len, scale, d_pos, stream);
}
