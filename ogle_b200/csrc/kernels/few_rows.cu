// Contractions of few rows - a classifier's last layer for an image or a few, the last maps of a detector, of a few pixels -
// with the filters as they are packed for the tensor cores: bound by fetching the filters once, and, at a few megabytes of
// them, by the launch and a trip to L2, of which the tensor-core kernel makes several (1 x 512 x 1000, waited for: 30 us a
// call, 22 here). A warp takes kCols columns, 128 reduction elements a step, every lane four of each; where the columns do
// not fill the GPU, kw warps share them and a reduction. Multiply-adds are fp32 on the operand as the pack holds it - its
// high part, in split mode plus the bfloat16 of the rest, an exact sum -: nothing is dropped that the tensor-core passes
// keep, and nothing of the other operand is.
#include <cuda_bf16.h>

#include "few_rows.cuh"

namespace ogle {
namespace {

template <int kRows, int kCols, bool kSplit, bool kWindow>
__global__ void __launch_bounds__(256)
few_rows_kernel(const FewRowsArgs a) {
    __shared__ float s_part[8][kRows * kCols];
    grid_dependency_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / a.kw, part = warp - group * a.kw, groups = 8 / a.kw;
    const int n0 = ((int)blockIdx.x * groups + group) * kCols, m0 = (int)blockIdx.y * kRows;
    const int Np = (a.N + 3) / 4 * 4, taps = kWindow ? a.kernel * a.kernel : 1;
    // a row's pixel: its number in the tensor, and where its window starts
    long at[kRows];
    int iy0[kRows], ix0[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int m = m0 + r < a.M ? m0 + r : 0;
        at[r] = m;
        iy0[r] = ix0[r] = 0;
        if (kWindow) {
            const int line = m / a.Wo, n = line / a.Ho;
            iy0[r] = (line - n * a.Ho) * a.stride - a.pad;
            ix0[r] = (m - line * a.Wo) * a.stride - a.pad;
            at[r] = (long)n * a.H * a.W;
        }
    }
    grid_dependency_wait();
    float acc[kRows][kCols];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) acc[r][c] = 0.f;
    if (n0 < Np) {                                   // (rows of the pack past N are zeros, up to a multiple of 128)
        const int total = taps * a.Cp32;
        const __nv_bfloat16* cross = reinterpret_cast<const __nv_bfloat16*>(a.lo);
        auto step = [&](int k) {
            float b[kCols][4];
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const long row = (long)(n0 + c) * total;
                const float4 h = __ldg(reinterpret_cast<const float4*>(a.hi + row + k));
                b[c][0] = h.x; b[c][1] = h.y; b[c][2] = h.z; b[c][3] = h.w;
                if (kSplit) {
                    const uint2 l = __ldg(reinterpret_cast<const uint2*>(cross + (row + (k & ~31)) * 2 + (k & 31)));
                    b[c][0] += __uint_as_float(l.x << 16); b[c][1] += __uint_as_float(l.x & 0xffff0000u);
                    b[c][2] += __uint_as_float(l.y << 16); b[c][3] += __uint_as_float(l.y & 0xffff0000u);
                }
            }
            int ch = k, dy = 0, dx = 0;
            if (kWindow) {
                const int tap = k / a.Cp32, ky = tap / a.kernel;
                ch = k - tap * a.Cp32;
                dy = ky * a.dil;
                dx = (tap - ky * a.kernel) * a.dil;
            }
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                long pixel = at[r];
                bool there = m0 + r < a.M;
                if (kWindow) {
                    const int iy = iy0[r] + dy, ix = ix0[r] + dx;
                    there = there && (unsigned)iy < (unsigned)a.H && (unsigned)ix < (unsigned)a.W;
                    pixel += (long)iy * a.W + ix;
                }
                if (there) {
                    const float* from = a.x + pixel * a.ldx + ch;
                    if (ch + 4 <= a.C) {
                        const float4 q = *reinterpret_cast<const float4*>(from);
                        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
                    } else {                         // what lies past the end of a row is not to be read
#pragma unroll
                        for (int l = 0; l < 3; ++l)
                            if (ch + l < a.C) v[l] = from[l];
                    }
                }
#pragma unroll
                for (int c = 0; c < kCols; ++c)
#pragma unroll
                    for (int l = 0; l < 4; ++l) acc[r][c] = fmaf(v[l], b[c][l], acc[r][c]);
            }
        };
        // Several rows: all lanes take as many steps, but for one by itself at the end. In one loop to the end of the reduction
        // some lanes went once more through its unrolled part while the others took its remainder, one after the other:
        // 4 x 448 x 1500 8.7 us (8.3 on the tensor cores), 5.9 so; 6 x 864 x 700 8.9 -> 6.1; 260 convolutions of few pixels 3 %.
        // (One row has less in its steps, and the last by itself costs more: a pixel of 5x5 607 -> 40 5.9 us, 7.0 that way. In
        // long reductions it is one of many: 2 x 3092 x 2558 16.1, 17.0 that way; with four columns a warp both loops want the
        // registers of two blocks: 8 x 64 x 5000 3.9, 5.7.)
        constexpr int kAtOnce = kRows * kCols == 1 ? 8 : (kRows * kCols <= 4 ? 4 : 2);
        if (kRows > 1 && kCols == 1 && total < 2048) {
            int k0 = part * 128;
#pragma unroll(kAtOnce)
            for (; k0 + 128 <= total; k0 += a.kw * 128) step(k0 + lane * 4);
            if (k0 + lane * 4 < total) step(k0 + lane * 4);
        } else {
#pragma unroll(kAtOnce)
            for (int k = part * 128 + lane * 4; k < total; k += a.kw * 128) step(k);
        }
    }
    float mine = 0.f;                                // lane r * kCols + c keeps that sum
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            float v = acc[r][c];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == r * kCols + c) mine = v;
        }
    if (a.kw > 1) {
        if (lane < kRows * kCols) s_part[warp][lane] = mine;
        __syncthreads();
        if (part != 0) return;
        if (lane < kRows * kCols)
            for (int p = 1; p < a.kw; ++p) mine += s_part[warp + p][lane];
    }
    const int m = m0 + lane / kCols, n = n0 + lane % kCols;
    if (lane >= kRows * kCols || m >= a.M || n >= Np) return;
    // which output the column belongs to, and its place there; padded columns are zero
    const bool second = a.split_col > 0 && n >= a.split_col;
    const int col = second ? n - a.split_col : n, real = second ? a.N - a.split_col : (a.split_col > 0 ? a.N1 : a.N);
    if (col >= (real + 3) / 4 * 4) return;           // between the two outputs
    float v = 0.f;
    if (col < real) {
        if (a.bias_mode == 1) v = fmaf(a.beta, a.bias[(long)m * a.ldc + n], a.alpha * mine);
        else v = fmaf(a.alpha, mine, a.bias_mode == 2 ? a.beta * a.bias[n] : 0.f);
        if (a.res) v += a.res[(long)m * a.res_ld + n];
        v = apply_act(v, a.act, a.lo_clip, a.hi_clip);
    }
    if (second) a.y2[(long)m * a.ldy2 + col] = v;
    else a.y[(long)m * a.ldy + col] = v;
}

template <int kRows, int kCols>
void (*kernel_for(const FewRowsArgs& a))(FewRowsArgs) {
    if (a.H > 0) return a.lo ? few_rows_kernel<kRows, kCols, true, true> : few_rows_kernel<kRows, kCols, false, true>;
    return a.lo ? few_rows_kernel<kRows, kCols, true, false> : few_rows_kernel<kRows, kCols, false, false>;
}

}  // namespace

int launch_few_rows(FewRowsArgs a, cudaStream_t s) {
    a.kw = few_rows_warps(a.N, a.kernel * a.kernel * a.Cp32);
    const int rows = few_rows_rows(a.M), cols = few_rows_cols(a.N), per_block = 8 / a.kw * cols;
    const bool wide = cols > 1;
    const dim3 grid((unsigned)((up4(a.N) + per_block - 1) / per_block), (unsigned)((a.M + rows - 1) / rows));
    const auto kernel = rows == 1   ? (wide ? kernel_for<1, 4>(a) : kernel_for<1, 1>(a))
                        : rows == 2 ? (wide ? kernel_for<2, 4>(a) : kernel_for<2, 1>(a))
                                    : (wide ? kernel_for<4, 4>(a) : kernel_for<4, 1>(a));
    const bool overlapped = overlapped_launches_enabled();
    note_contraction(8, a.kw, cols, overlapped);
    launch_overlapped_if(overlapped, kernel, grid, dim3(256), 0, s, a);
    return finish_launch();
}

}  // namespace ogle
