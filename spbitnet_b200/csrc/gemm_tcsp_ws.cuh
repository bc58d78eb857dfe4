// Host interface of the tcgen05 sparse product (gemm_tcsp_ws.cu); library-internal.
#pragma once
#include "spb_common.cuh"

namespace spb {

constexpr int kWsMaxMats = 3;

// One weight matrix of a launch: its packed rows and where its n rows of `rows` results go.
struct TcspMat {
    const uint32_t* meta;
    const uint32_t* values;
    void* out;  // int32 sums, or half when the launch has row scales
    float gamma;
    int rows, meta_stride, values_stride;
};

// out = X W^T for up to kWsMaxMats matrices of the same width on the same n activation rows, one launch.  With absmax (n
// row scales, device) the outputs are half(float(sum) * dequant_scale(gamma, absmax[row])).  Any layout the packed format
// has; meta and values at their natural 4-byte alignment.
int gemm_tcsp_ws_launch(const TcspMat* mats, int nmat, const int8_t* X, const float* absmax, int cols, int n, void* stream);

// gemm_mmasp.cu: the same on the warp-level sparse MMA; where it applies, and where it is the faster form
bool gemm_mmasp_supported(const TcspMat* mats, int nmat, const int8_t* X, int cols, int n);
bool gemm_mmasp_preferred(const TcspMat* mats, int nmat, int cols, int n, bool half_out);
int gemm_mmasp_launch(const TcspMat* mats, int nmat, const int8_t* X, const float* absmax, int cols, int n, void* stream);

// gemm.cu: BitLinear layers of one width on n quantised rows (scaled half outputs); acc_workspace: n * max rows int32, for the
// forms that need it
int bitlinear_gemm_group(const TcspMat* mats, int nmat, const int8_t* Xq, const float* absmax, int cols, int n,
                         int32_t* acc_workspace, void* stream);

}  // namespace spb
