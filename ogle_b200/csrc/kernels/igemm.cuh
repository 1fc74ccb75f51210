// Arguments of the CUDA-core fp32 contraction (igemm.cu): convolution as implicit GEMM, and gemm.
#pragma once
#include "conv_args.cuh"

namespace ogle {

// D[m][n] = sum_r A[m][r] * B[r][n]. A is gathered from an NHWC4 tensor (a row-major matrix is the 1x1 case with one
// pixel per row), B is [R][ldb] or, transposed, [N][ldb].
struct IgemmArgs {
    const float* x;          // A: pixels of Cs floats
    const float* w;          // B
    const float* bias;
    float* y;
    long M;                  // output pixels (rows)
    int H, W, Ho, Wo, Cs;    // input extent and pixel stride; fewer than 2^31 input pixels, or one image
    int kernel, stride, pad, dil;
    int Cp;                  // reduction elements per filter tap
    int R;                   // kernel * kernel * Cp
    int ldb, n_b;            // row stride of B; columns of B that hold data
    int N;                   // output channels
    int n_store;             // columns written (lanes N..n_store-1 as zeros)
    int ldy, yoff;           // floats per output row, first column
    int act;
    float lo, hi;
    float alpha, beta;       // gemm: alpha * sum + beta * bias
    int bias_mode;           // 0 none, 1 matrix [M][ldc], 2 row [N]
    int ldc;
};

// name: not null = nothing is launched (y is null), and *name says which kernel would be.
int launch_igemm(const IgemmArgs& a, bool trans_b, cudaStream_t s, const char** name = nullptr);

}  // namespace ogle
