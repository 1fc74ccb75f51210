// Arguments of the contraction of few rows with packed filters (few_rows.cu).
#pragma once
#include "conv_args.cuh"

namespace ogle {

// D[m][n] = sum over taps and channels of A and B. B as the tensor-core kernels take it: `hi` [>= N rows][kernel^2][Cp32],
// `lo` the cross section beside it (null: one pass, `hi` alone). A is a matrix of M rows of C elements, ldx floats apart
// (kernel 1, H 0), or the windows of a convolution over pixels of ldx floats.
struct FewRowsArgs {
    const float *x, *hi, *lo, *bias, *res;
    float *y, *y2;
    int M, N;                          // rows; columns (stacked, with two outputs)
    int C, Cp32, kernel;
    int H, W, Ho, Wo, stride, pad, dil;
    int ldx, ldy, ldy2, ldc, res_ld;   // floats a row (of y, y2 from their first column on)
    int split_col, N1;                 // two outputs: columns [0, N1) to y, [split_col, N) to y2 (split_col 0: one)
    float alpha, beta;
    int bias_mode;                     // 0 none, 1 matrix [M][ldc], 2 row [N]
    int act;
    float lo_clip, hi_clip;
    int kw;                            // set by the launch
};

int launch_few_rows(FewRowsArgs a, cudaStream_t s);

// Warps that share a column and a reduction of `total` elements: as many as fill the GPU, with two steps each.
inline int few_rows_warps(int N, int total) {
    int kw = 1;
    while (kw < 8 && (long)up4(N) * kw * 2 <= 16 * kNumSMs && total >= kw * 256) kw *= 2;
    return kw;
}
// Columns of a warp: four where one each is more than the GPU holds at once.
inline int few_rows_cols(int N) { return N > 32 * kNumSMs ? 4 : 1; }
// Rows of a warp.
inline int few_rows_rows(long M) { return M == 1 ? 1 : (M == 2 ? 2 : 4); }

}  // namespace ogle
