// The vector ops of a batch of rows (prompt tokens, sequences), one block per row, the row in registers: each operand is
// read once with 16-byte loads, all of a thread's loads in flight before the first reduction, and nothing goes through
// shared memory but the warps' partial sums.  The rounding points are those of the scalar kernels in fused_ops.cu and
// prefill.cu, which take what these do not (lengths that are no multiple of 8, unaligned operands, rows above 32768).
//
// Bound: bytes through L2.  The scalar forms walked a row element by element in up to 1024 threads, with a trip through
// shared memory between passes.  Measured for 1024 rows, us before -> now: residual + norm + quantise of 2560 19.9 -> 7.5,
// relu2 + norm + quantise of 6912 29.8 -> 12.9, absmax + quantise of 2560 9.2 -> 4.5, rotation + scatter of 20 + 5 heads of
// 128 20.1 -> 7.0 (a thread per pair evaluated powf, cosf and sinf for every head; here once per token and pair).
//
// Threads and pieces per thread follow from the row length alone, never from the number of rows: the order of a row's sums
// does not depend on how a prompt is cut into calls.
#include "fused_ops.cuh"
#include "row_ops.cuh"

namespace spb {

namespace {

__device__ __forceinline__ float row_sum(float v, float* sh, int warps) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
    const int lane = threadIdx.x & 31;
    if (lane == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = lane < warps ? sh[lane] : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
    return v;
}
__device__ __forceinline__ float row_max(float v, float* sh, int warps) {  // values >= 0
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
    const int lane = threadIdx.x & 31;
    if (lane == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = lane < warps ? sh[lane] : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
    return v;
}

__device__ __forceinline__ void unpack8(const uint4& p, float (&f)[8]) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {  // of values that are halves already
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 t = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&t);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ uint2 quantize8(const float (&f)[8], float qs) {
    uint32_t w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        w[i] = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) w[i] |= (static_cast<uint32_t>(quantize_one(f[4 * i + j], qs)) & 0xFFu) << (8 * j);
    }
    return make_uint2(w[0], w[1]);
}

// residual_norm_quant (fused_ops.cu) of a row of 8 * pieces elements
template <int P>
__global__ void __launch_bounds__(1024) rows_residual_norm_quant_kernel(
    const __half* __restrict__ delta, const float* __restrict__ sub_w, __half* __restrict__ x, const float* __restrict__ w,
    __half* __restrict__ xn_out, int8_t* __restrict__ xq, float* __restrict__ d_absmax, int pieces, float eps) {
    __shared__ float sh[3 * 32];
    grid_dep_launch();
    grid_dep_wait();
    const int tid = threadIdx.x, nt = blockDim.x, warps = nt >> 5;
    const size_t row = static_cast<size_t>(blockIdx.x) * pieces;
    const float n = static_cast<float>(8 * pieces);
    uint4* xr = reinterpret_cast<uint4*>(x) + row;
    float v[P][8];
    {
        uint4 px[P], pd[P];
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int i = tid + k * nt;
            px[k] = i < pieces ? xr[i] : make_uint4(0, 0, 0, 0);
            pd[k] = delta && i < pieces ? reinterpret_cast<const uint4*>(delta)[row + i] : make_uint4(0, 0, 0, 0);
        }
        float sub_scale = 1.0f;
        if (delta && sub_w) {
            float s = 0.0f;
#pragma unroll
            for (int k = 0; k < P; ++k) {
                float d[8];
                unpack8(pd[k], d);
#pragma unroll
                for (int j = 0; j < 8; ++j) s += d[j] * d[j];
            }
            sub_scale = rsqrtf(row_sum(s, sh, warps) / n + eps);
        }
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int i = tid + k * nt;
            unpack8(px[k], v[k]);
            if (delta && i < pieces) {
                float d[8];
                unpack8(pd[k], d);
                if (sub_w) {
                    float sw[8];
                    load8(sub_w + 8 * i, sw);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        d[j] = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(d[j], sub_scale), sw[j])));
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) v[k][j] = __half2float(__float2half_rn(d[j] + v[k][j]));
                xr[i] = pack8(v[k]);
            }
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < P; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[k][j] * v[k][j];
    const float scale = rsqrtf(row_sum(s, sh + 32, warps) / n + eps);
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        if (i < pieces) {
            float wv[8];
            load8(w + 8 * i, wv);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[k][j] = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(v[k][j], scale), wv[j])));
                m = fmaxf(m, fabsf(v[k][j]));
            }
            if (xn_out) reinterpret_cast<uint4*>(xn_out)[row + i] = pack8(v[k]);
        }
    }
    const float absmax = row_max(m, sh + 64, warps);
    if (tid == 0) d_absmax[blockIdx.x] = absmax;
    const float qs = quant_scale(absmax);
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        if (i < pieces) reinterpret_cast<uint2*>(xq)[row + i] = quantize8(v[k], qs);
    }
}

// relu2_norm_quant (fused_ops.cu) of a row of 8 * pieces elements
template <int P>
__global__ void __launch_bounds__(1024) rows_relu2_norm_quant_kernel(
    const __half* __restrict__ gate, const __half* __restrict__ up, const float* __restrict__ sub_w, __half* __restrict__ h_out,
    int8_t* __restrict__ hq, float* __restrict__ d_absmax, int pieces, float eps) {
    __shared__ float sh[2 * 32];
    grid_dep_launch();
    grid_dep_wait();
    const int tid = threadIdx.x, nt = blockDim.x, warps = nt >> 5;
    const size_t row = static_cast<size_t>(blockIdx.x) * pieces;
    float v[P][8], s = 0.0f;
    {
        uint4 pg[P], pu[P];
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int i = tid + k * nt;
            pg[k] = i < pieces ? reinterpret_cast<const uint4*>(gate)[row + i] : make_uint4(0, 0, 0, 0);
            pu[k] = i < pieces ? reinterpret_cast<const uint4*>(up)[row + i] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int k = 0; k < P; ++k) {
            float g[8], u[8];
            unpack8(pg[k], g);
            unpack8(pu[k], u);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float r = fmaxf(0.0f, g[j]);
                v[k][j] = __fmul_rn(__fmul_rn(r, r), u[j]);
                s += v[k][j] * v[k][j];
            }
        }
    }
    float scale = 1.0f;
    if (sub_w) scale = rsqrtf(row_sum(s, sh, warps) / static_cast<float>(8 * pieces) + eps);
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        if (i < pieces) {
            float sw[8];
            if (sub_w) load8(sub_w + 8 * i, sw);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float t = sub_w ? __fmul_rn(__fmul_rn(v[k][j], scale), sw[j]) : v[k][j];
                v[k][j] = __half2float(__float2half_rn(t));
                m = fmaxf(m, fabsf(v[k][j]));
            }
            if (h_out) reinterpret_cast<uint4*>(h_out)[row + i] = pack8(v[k]);
        }
    }
    const float absmax = row_max(m, sh + 32, warps);
    if (tid == 0) d_absmax[blockIdx.x] = absmax;
    const float qs = quant_scale(absmax);
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        if (i < pieces) reinterpret_cast<uint2*>(hq)[row + i] = quantize8(v[k], qs);
    }
}

// absmax_quantize_rows (prefill.cu) of a row of 8 * pieces elements
template <int P>
__global__ void __launch_bounds__(1024) rows_absmax_quantize_kernel(const __half* __restrict__ in, int8_t* __restrict__ out,
                                                                    float* __restrict__ d_absmax, int pieces) {
    __shared__ float sh[32];
    grid_dep_launch();
    grid_dep_wait();
    const int tid = threadIdx.x, nt = blockDim.x;
    const size_t row = static_cast<size_t>(blockIdx.x) * pieces;
    uint4 p[P];
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        p[k] = i < pieces ? reinterpret_cast<const uint4*>(in)[row + i] : make_uint4(0, 0, 0, 0);
    }
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        float f[8];
        unpack8(p[k], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(f[j]));
    }
    const float absmax = row_max(m, sh, nt >> 5);
    if (tid == 0) d_absmax[blockIdx.x] = absmax;
    const float qs = quant_scale(absmax);
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int i = tid + k * nt;
        float f[8];
        unpack8(p[k], f);
        if (i < pieces) reinterpret_cast<uint2*>(out)[row + i] = quantize8(f, qs);
    }
}

constexpr int kRopeThreads = 256;

// rope_scatter (fused_ops.cu): blockIdx.y = token, 256 pieces of 8 elements per block, q heads first, then k, then v.  The
// head_dim / 2 rotations of the token are evaluated once per block into shared memory.
__global__ void __launch_bounds__(kRopeThreads) rows_rope_scatter_kernel(
    __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, __half* __restrict__ kcache,
    __half* __restrict__ vcache, int num_heads, int num_kv_heads, int head_dim, int max_seq_len, float theta,
    const int* __restrict__ d_pos, size_t seq_stride) {
    extern __shared__ __align__(16) float2 rot[];  // head_dim / 2 of (cos, sin)
    grid_dep_launch();
    grid_dep_wait();
    const int pos = *d_pos + (seq_stride ? 0 : blockIdx.y);
    const int ppr = head_dim >> 3;  // pieces per head
    const int nq = num_heads * ppr, nk = num_kv_heads * ppr;
    const int t = blockIdx.x * kRopeThreads + threadIdx.x;
    const size_t tok = blockIdx.y;
    const bool is_q = t < nq, is_k = !is_q && t < nq + nk, is_v = !is_q && !is_k && t < nq + 2 * nk;
    const int kt = t - nq - (is_v ? nk : 0);  // piece of k or v
    uint4* src = nullptr;
    if (is_q) src = reinterpret_cast<uint4*>(q) + tok * nq + t;
    if (is_k) src = const_cast<uint4*>(reinterpret_cast<const uint4*>(k)) + tok * nk + kt;
    if (is_v) src = const_cast<uint4*>(reinterpret_cast<const uint4*>(v)) + tok * nk + kt;
    uint4 p = make_uint4(0, 0, 0, 0);
    if (src) p = *src;
    if (blockIdx.x * kRopeThreads < nq + nk)
        for (int i = threadIdx.x; i < head_dim / 2; i += kRopeThreads) {
            float c, s;
            rope_angle(pos, i, head_dim, theta, c, s);
            rot[i] = make_float2(c, s);
        }
    __syncthreads();
    if (!src) return;
    if (!is_v) {
        const int pair0 = ((is_q ? t : kt) % ppr) * 4;
        float f[8];
        unpack8(p, f);
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 cs = rot[pair0 + j];
            __half y0, y1;
            rope_apply(f[2 * j], f[2 * j + 1], cs.x, cs.y, y0, y1);
            w[j] = static_cast<uint32_t>(__half_as_ushort(y0)) | (static_cast<uint32_t>(__half_as_ushort(y1)) << 16);
        }
        p = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (is_q) {
        *src = p;
    } else {
        const int head = kt / ppr;
        __half* cache = (is_k ? kcache : vcache) + seq_stride * tok + (static_cast<size_t>(head) * max_seq_len + pos) * head_dim;
        reinterpret_cast<uint4*>(cache)[kt % ppr] = p;
    }
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Pieces per thread: more for longer rows, so that a block keeps few warps at its barriers and a thread several loads in
// flight, up to 1024 threads of four pieces.
int pieces_per_thread(int pieces) { return pieces <= 128 ? 1 : pieces <= 512 ? 2 : 4; }
dim3 row_threads(int pieces, int per) { return dim3(((pieces + per - 1) / per + 31) & ~31); }

}  // namespace

bool row_ops_take(int n, const void* a, const void* b, const void* c, const void* d, const void* e, const void* q) {
    return n > 0 && n % 8 == 0 && n <= 8 * 4 * 1024 && al16(a) && al16(b) && al16(c) && al16(d) && al16(e) && al16(q);
}

#define SPB_ROW_CASES(name, kernel, vectors, ...)                                                                        \
    switch (pieces_per_thread(n / 8)) {                                                                                  \
        case 1: return launch(name, kernel<1>, dim3(vectors), row_threads(n / 8, 1), 0, stream, __VA_ARGS__);           \
        case 2: return launch(name, kernel<2>, dim3(vectors), row_threads(n / 8, 2), 0, stream, __VA_ARGS__);           \
        default: return launch(name, kernel<4>, dim3(vectors), row_threads(n / 8, 4), 0, stream, __VA_ARGS__);          \
    }

int rows_residual_norm_quant(const __half* delta, const float* sub_w, __half* x, const float* w, __half* xn_out, int8_t* xq,
                             float* d_absmax, int n, float eps, void* stream, int vectors) {
    SPB_ROW_CASES("residual_norm_quant", rows_residual_norm_quant_kernel, vectors, delta, sub_w, x, w, xn_out, xq, d_absmax, n / 8, eps)
}
int rows_relu2_norm_quant(const __half* gate, const __half* up, const float* sub_w, __half* h_out, int8_t* hq, float* d_absmax,
                          int n, float eps, void* stream, int vectors) {
    SPB_ROW_CASES("relu2_norm_quant", rows_relu2_norm_quant_kernel, vectors, gate, up, sub_w, h_out, hq, d_absmax, n / 8, eps)
}
int rows_absmax_quantize(const __half* in, int8_t* out, float* d_absmax, int n, void* stream, int vectors) {
    SPB_ROW_CASES("absmax_quantize_rows", rows_absmax_quantize_kernel, vectors, in, out, d_absmax, n / 8)
}
#undef SPB_ROW_CASES

bool rows_rope_scatter_takes(const void* q, const void* k, const void* v, const void* kcache, const void* vcache, int head_dim,
                             size_t seq_stride) {
    return head_dim > 0 && head_dim % 8 == 0 && head_dim <= 4096 && seq_stride % 8 == 0 && al16(q) && al16(k) && al16(v) &&
           al16(kcache) && al16(vcache);
}
int rows_rope_scatter(__half* q, const __half* k, const __half* v, __half* kcache, __half* vcache, int num_heads,
                      int num_kv_heads, int head_dim, int max_seq_len, float theta, const int* d_pos, void* stream, int vectors,
                      size_t seq_stride) {
    const int pieces = (num_heads + 2 * num_kv_heads) * (head_dim / 8);
    return launch("rope_scatter", rows_rope_scatter_kernel, dim3((pieces + kRopeThreads - 1) / kRopeThreads, vectors),
                  dim3(kRopeThreads), sizeof(float2) * (head_dim / 2), stream, q, k, v, kcache, vcache, num_heads, num_kv_heads,
                  head_dim, max_seq_len, theta, d_pos, seq_stride);
}

}  // namespace spb
