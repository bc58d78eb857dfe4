// Decode attention of many vectors (one new token of each of B independent sequences): attention_scores_gpu + softmax_gpu +
// attention_output_gpu (src/kernels/inference_kernels.cu:241-371) over the positions up to the token's own.
//
// A block takes one KV head of one sequence, a warp one of its G query heads, so that K and V cross into shared memory once
// for the group: tiles of 32 positions, two in flight.  A lane forms the score of one position, then holds head_dim / 32 of
// the output's dims while the tile's weights go round by shuffles.  Scores, running maximum, sum and output are fp32.
//
// Bound: the caches through HBM with one query head per KV head and blocks enough (64 sequences of 4000 positions, 20 heads of
// 128: 422 us, 6.2 TB/s); the arithmetic of a block's warps with groups (8 KV heads of 8: 578 us, 1.8 TB/s); a block's tiles one
// after the other where KV heads times sequences leave SMs idle (two sequences of 4000 at 5 KV heads of 4: 141 us); two barriers
// and one tile's chain for short sequences.  One block per (query head, sequence), a warp per position with 2-byte loads, used
// before, was slower by 1.3 to 4.6 over 1, 2, 3, 4 and 8 heads per KV head, head dims 64 and 128, 2 to 64 sequences of 1 to 4000
// positions: 1270, 2379 and 291 us for the three above, 24.2 against 6.2 for 64 sequences of 16 positions at 8 KV heads of 8.
#include "fused_ops.cuh"

namespace spb {

namespace {

constexpr int kAbTile = 32;

__device__ __forceinline__ float ab_max(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
    return v;
}

template <int HD>
__global__ void __launch_bounds__(256) batch_attention_kernel(const __half* __restrict__ Q, const __half* __restrict__ K,
                                                              const __half* __restrict__ V, __half* __restrict__ out,
                                                              int num_heads, int max_seq_len, float scale,
                                                              const int* __restrict__ d_pos, size_t seq_stride) {
    constexpr int kRowBytes = HD * 2, kTileBytes = kAbTile * kRowBytes, kDims = HD / 32;
    extern __shared__ __align__(128) uint8_t ab_sm[];  // K tile x 2, V tile x 2, q as fp32: G x HD
    grid_dep_launch();
    grid_dep_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = blockDim.x >> 5;
    const int seq_len = *d_pos + (seq_stride ? 0 : blockIdx.y) + 1;
    const int ntiles = (seq_len + kAbTile - 1) / kAbTile;
    const int head = blockIdx.x * G + warp;
    const uint8_t* kg = reinterpret_cast<const uint8_t*>(K + seq_stride * blockIdx.y + static_cast<size_t>(blockIdx.x) * max_seq_len * HD);
    const uint8_t* vg = reinterpret_cast<const uint8_t*>(V + seq_stride * blockIdx.y + static_cast<size_t>(blockIdx.x) * max_seq_len * HD);
    const size_t qoff = (static_cast<size_t>(blockIdx.y) * num_heads + head) * HD;
    const uint32_t sm = static_cast<uint32_t>(__cvta_generic_to_shared(ab_sm));
    float* qs = reinterpret_cast<float*>(ab_sm + 4 * kTileBytes) + warp * HD;

    auto load_tile = [&](int j) {  // 16-byte pieces, piece c of row r at c ^ (r & 7); positions past the sequence: zero
        const uint32_t kb = sm + (j & 1) * kTileBytes, vb = kb + 2 * kTileBytes;
        for (int i = threadIdx.x; i < kAbTile * (HD / 8); i += blockDim.x) {
            const int r = i / (HD / 8), c = i % (HD / 8), p = j * kAbTile + r;
            const uint32_t dst = r * kRowBytes + ((c ^ (r & 7)) << 4);
            const size_t src = static_cast<size_t>(min(p, seq_len - 1)) * kRowBytes + c * 16;
            const int n = p < seq_len ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kb + dst), "l"(kg + src), "r"(n) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vb + dst), "l"(vg + src), "r"(n) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_tile(0);
#pragma unroll
    for (int i = 0; i < kDims; ++i) qs[i * 32 + lane] = __half2float(Q[qoff + i * 32 + lane]);
    __syncwarp();

    float o[kDims];
#pragma unroll
    for (int i = 0; i < kDims; ++i) o[i] = 0.0f;
    float m = -INFINITY, l = 0.0f;
    for (int j = 0; j < ntiles; ++j) {
        if (j + 1 < ntiles) {
            load_tile(j + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint8_t* kb = ab_sm + (j & 1) * kTileBytes;
        const uint8_t* vb = kb + 2 * kTileBytes;
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
        for (int c = 0; c < HD / 8; ++c) {
            const uint4 kv = *reinterpret_cast<const uint4*>(kb + lane * kRowBytes + ((c ^ (lane & 7)) << 4));
            const float4 qa = *reinterpret_cast<const float4*>(qs + 8 * c), qb = *reinterpret_cast<const float4*>(qs + 8 * c + 4);
            const float2 k0 = __half22float2(*reinterpret_cast<const __half2*>(&kv.x)), k1 = __half22float2(*reinterpret_cast<const __half2*>(&kv.y));
            const float2 k2 = __half22float2(*reinterpret_cast<const __half2*>(&kv.z)), k3 = __half22float2(*reinterpret_cast<const __half2*>(&kv.w));
            a0 = fmaf(qa.x, k0.x, a0); a1 = fmaf(qa.y, k0.y, a1);
            a0 = fmaf(qa.z, k1.x, a0); a1 = fmaf(qa.w, k1.y, a1);
            a0 = fmaf(qb.x, k2.x, a0); a1 = fmaf(qb.y, k2.y, a1);
            a0 = fmaf(qb.z, k3.x, a0); a1 = fmaf(qb.w, k3.y, a1);
        }
        const bool seen = j * kAbTile + lane < seq_len;
        const float s = seen ? (a0 + a1) * scale : -INFINITY;
        const float mn = fmaxf(m, ab_max(s));  // the first tile holds a position of the sequence
        const float corr = expf(m - mn), e = seen ? expf(s - mn) : 0.0f;
        m = mn;
        l = l * corr + e;
#pragma unroll
        for (int i = 0; i < kDims; ++i) o[i] *= corr;
        const int rows = min(kAbTile, seq_len - j * kAbTile);
        for (int r0 = 0; r0 < rows; r0 += 4) {  // rows past the sequence: zero weights and zero V
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + q;
                const float w = __shfl_sync(0xFFFFFFFFu, e, r);
                const uint8_t* vr = vb + r * kRowBytes;
                if (kDims == 4) {
                    const uint2 vv = *reinterpret_cast<const uint2*>(vr + (((lane >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8);
                    const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(&vv.x)), v1 = __half22float2(*reinterpret_cast<const __half2*>(&vv.y));
                    o[0] = fmaf(w, v0.x, o[0]); o[1] = fmaf(w, v0.y, o[1]);
                    o[kDims - 2] = fmaf(w, v1.x, o[kDims - 2]); o[kDims - 1] = fmaf(w, v1.y, o[kDims - 1]);
                } else {
                    const uint32_t vv = *reinterpret_cast<const uint32_t*>(vr + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
                    const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(&vv));
                    o[0] = fmaf(w, v0.x, o[0]); o[1] = fmaf(w, v0.y, o[1]);
                }
            }
        }
        __syncthreads();  // the tile's buffer is free for the load after next
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, off);
    const float inv = 1.0f / l;
    __half2* dst = reinterpret_cast<__half2*>(out + qoff + lane * kDims);
#pragma unroll
    for (int i = 0; i < kDims / 2; ++i) dst[i] = __floats2half2_rn(o[2 * i] * inv, o[2 * i + 1] * inv);
}

}  // namespace

// head dims 64 and 128, whole groups of up to 8 heads, 16-byte aligned caches a multiple of 16 bytes apart
bool batch_attention_supported(const void* K, const void* V, const void* out, int num_heads, int num_kv_heads, int head_dim,
                               size_t seq_stride) {
    return (head_dim == 64 || head_dim == 128) && num_kv_heads > 0 && num_heads % num_kv_heads == 0 &&
           num_heads / num_kv_heads <= 8 && seq_stride % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(V)) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 3u) == 0;
}

int batch_attention(const void* Q, const void* K, const void* V, void* out, int num_heads, int num_kv_heads, int head_dim,
                    int max_seq_len, float scale, const int* d_pos, void* stream, int vectors, size_t seq_stride) {
    const int G = num_heads / num_kv_heads;
    const size_t smem = 4 * static_cast<size_t>(kAbTile) * head_dim * 2 + sizeof(float) * G * head_dim;
    auto kernel = head_dim == 64 ? batch_attention_kernel<64> : batch_attention_kernel<128>;
    if (int rc = ensure_dynamic_smem("batch_attention", kernel, smem)) return rc;
    return launch("batch_attention", kernel, dim3(num_kv_heads, vectors), dim3(32 * G), smem, stream,
                  static_cast<const __half*>(Q), static_cast<const __half*>(K), static_cast<const __half*>(V),
                  static_cast<__half*>(out), num_heads, max_seq_len, scale, d_pos, seq_stride);
}

}  // namespace spb
