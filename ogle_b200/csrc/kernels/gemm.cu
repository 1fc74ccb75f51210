// Gemm: Y[M,N] = alpha * A[M,K] * (transB ? B[N,K]^T : B[K,N]) + beta * C.
// OGLE_MATH_FP32 runs the CUDA-core kernel of igemm.cu; the TF32 modes
// go to the tcgen05 path when the shape allows it.
#include <cuda_bf16.h>

#include "igemm.cuh"

namespace ogle {

int launch_gemm_tc(const OgleGemmParams& p, const float* A, const float* B, const float* C,
                   float* Y, cudaStream_t s);
bool gemm_tc_supported(const OgleGemmParams& p, const float* A, const float* B);
int launch_gemm_tc_packed(const OgleGemmParams& p, const float* A, const float* Bhi, const float* Blo,
                          const float* C, float* Y, cudaStream_t s, bool overlapped);

// B [K][ldb] (or [N][ldb] when transB) -> two K-major sections of [round_up(N,128)][round_up(K,32)]
// 4-byte slots each: the fp32 values with the low 13 mantissa bits cleared (operand of the TF32
// pass), and per 32-element chunk of a row the 64 bf16 values [b_lo x 32 | b x 32] (operand of
// the BF16 cross-term pass, against [a_hi | a_lo]).
// Bound by latency and L2: a tile of 32 reduction elements x 64 columns at a time; a row-major B is read along its rows
// and turned over in shared memory (read down its columns, 1500 x 700 took 8.4 us against 4.8), and a thread writes
// four elements of a row as 16 and 2 x 8 bytes.
template <bool kTransB>
__global__ void __launch_bounds__(256)
gemm_pack_b_kernel(const float* __restrict__ B, float* __restrict__ hi, __nv_bfloat16* __restrict__ cross,
                   int K, int N, int ldb, int Kp32, int tiles_n, long tiles) {
    __shared__ float s_tile[32][65];
    grid_dependency_trigger();
    grid_dependency_wait();
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int k0 = (int)(tile / tiles_n) * 32, n0 = (int)(tile % tiles_n) * 64;
        if (!kTransB) {
            __syncthreads();                       // the tile before has been read
#pragma unroll
            for (int i = threadIdx.x; i < 32 * 64; i += 256) {
                const int k = k0 + (i >> 6), n = n0 + (i & 63);
                s_tile[i >> 6][i & 63] = k < K && n < N ? B[(long)k * ldb + n] : 0.f;
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = threadIdx.x; i < 64 * 8; i += 256) {
            const int n = n0 + (i >> 3), kk = (i & 7) * 4;
            float v[4], h[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (kTransB) v[l] = k0 + kk + l < K && n < N ? B[(long)n * ldb + k0 + kk + l] : 0.f;
                else v[l] = s_tile[kk + l][i >> 3];
                h[l] = __uint_as_float(__float_as_uint(v[l]) & 0xffffe000u);
            }
            const long chunk = (long)n * Kp32 + k0;              // first slot of this 32-element chunk
            *reinterpret_cast<float4*>(hi + chunk + kk) = make_float4(h[0], h[1], h[2], h[3]);
            const __nv_bfloat162 lo01 = __floats2bfloat162_rn(v[0] - h[0], v[1] - h[1]), lo23 = __floats2bfloat162_rn(v[2] - h[2], v[3] - h[3]);
            const __nv_bfloat162 v01 = __floats2bfloat162_rn(v[0], v[1]), v23 = __floats2bfloat162_rn(v[2], v[3]);
            uint2 lo, all;
            lo.x = *reinterpret_cast<const uint32_t*>(&lo01); lo.y = *reinterpret_cast<const uint32_t*>(&lo23);
            all.x = *reinterpret_cast<const uint32_t*>(&v01); all.y = *reinterpret_cast<const uint32_t*>(&v23);
            *reinterpret_cast<uint2*>(cross + chunk * 2 + kk) = lo;
            *reinterpret_cast<uint2*>(cross + chunk * 2 + 32 + kk) = all;
        }
    }
}

// A product of a few rows and a packed B: bound by fetching B once, and, at a few megabytes of it, by the launch and a trip
// to L2, of which the tensor-core kernel makes several (1 x 512 x 1000, waited for: 30 us a call, 22). A warp takes kCols columns, 128 reduction
// elements a step, every lane four of each; where the columns do not fill the GPU, kw warps share them and a reduction.
// Multiply-adds are fp32 on the operand as the pack holds it - its high part, in split mode plus the bfloat16 of the rest,
// an exact sum -: nothing is dropped that the tensor-core passes keep.
struct RowsArgs {
    const float *A, *hi, *bias;
    const __nv_bfloat16* cross;
    float* Y;
    int M, K, N, lda, ldy, ldc, Kp32;
    float alpha, beta;
    int bias_mode, kw;
};

template <int kRows, int kCols, bool kSplit>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const RowsArgs a) {
    __shared__ float s_part[8][kRows * kCols];
    grid_dependency_trigger();
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / a.kw, part = warp - group * a.kw, groups = 8 / a.kw;
    const int n0 = ((int)blockIdx.x * groups + group) * kCols, m0 = (int)blockIdx.y * kRows;
    const int Np = (a.N + 3) / 4 * 4;
    float acc[kRows][kCols];
#pragma unroll
    for (int m = 0; m < kRows; ++m)
#pragma unroll
        for (int c = 0; c < kCols; ++c) acc[m][c] = 0.f;
    if (n0 < Np) {                                   // (rows of the pack past N are zeros, up to a multiple of 128)
#pragma unroll(kRows * kCols == 1 ? 8 : (kRows * kCols <= 4 ? 4 : 2))
        for (int k = part * 128 + lane * 4; k < a.Kp32; k += a.kw * 128) {
            float b[kCols][4];
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const long row = (long)(n0 + c) * a.Kp32;
                const float4 h = __ldg(reinterpret_cast<const float4*>(a.hi + row + k));
                b[c][0] = h.x; b[c][1] = h.y; b[c][2] = h.z; b[c][3] = h.w;
                if (kSplit) {
                    const uint2 l = __ldg(reinterpret_cast<const uint2*>(a.cross + (row + (k & ~31)) * 2 + (k & 31)));
                    b[c][0] += __uint_as_float(l.x << 16); b[c][1] += __uint_as_float(l.x & 0xffff0000u);
                    b[c][2] += __uint_as_float(l.y << 16); b[c][3] += __uint_as_float(l.y & 0xffff0000u);
                }
            }
#pragma unroll
            for (int m = 0; m < kRows; ++m) {
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                if (m0 + m < a.M) {
                    const float* from = a.A + (long)(m0 + m) * a.lda + k;
                    if (k + 4 <= a.K) {
                        const float4 q = *reinterpret_cast<const float4*>(from);
                        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
                    } else {                         // what lies past the end of a row is not to be read
#pragma unroll
                        for (int l = 0; l < 3; ++l)
                            if (k + l < a.K) v[l] = from[l];
                    }
                }
#pragma unroll
                for (int c = 0; c < kCols; ++c)
#pragma unroll
                    for (int l = 0; l < 4; ++l) acc[m][c] = fmaf(v[l], b[c][l], acc[m][c]);
            }
        }
    }
    float mine = 0.f;                                // lane m * kCols + c keeps that sum
#pragma unroll
    for (int m = 0; m < kRows; ++m)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            float v = acc[m][c];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == m * kCols + c) mine = v;
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
    float v = 0.f;                                   // padded columns are zero
    if (n < a.N) {
        if (a.bias_mode == 1) v = fmaf(a.beta, a.bias[(long)m * a.ldc + n], a.alpha * mine);
        else v = fmaf(a.alpha, mine, a.bias_mode == 2 ? a.beta * a.bias[n] : 0.f);
    }
    a.Y[(long)m * a.ldy + n] = v;
}

template <int kRows>
static int launch_rows(const RowsArgs& a, bool split, bool overlapped, cudaStream_t s) {
    // four columns a warp where one each is more than the GPU holds at once
    const bool wide = a.N > 8 * 8 * kNumSMs / 2;
    const int per_block = 8 / a.kw * (wide ? 4 : 1);
    const dim3 grid((unsigned)((up4(a.N) + per_block - 1) / per_block), (unsigned)((a.M + kRows - 1) / kRows));
    auto kernel = wide ? (split ? gemm_rows_kernel<kRows, 4, true> : gemm_rows_kernel<kRows, 4, false>)
                       : (split ? gemm_rows_kernel<kRows, 1, true> : gemm_rows_kernel<kRows, 1, false>);
    launch_overlapped_if(overlapped_launches_enabled(overlapped), kernel, grid, dim3(256), 0, s, a);
    return finish_launch();
}

}  // namespace ogle

using namespace ogle;

static int normalize_gemm(OgleGemmParams* p) {
    if (p->M <= 0 || p->K <= 0 || p->N <= 0) return OGLE_ERR_INVALID;
    if (p->lda == 0) p->lda = up4(p->K);
    if (p->ldb == 0) p->ldb = p->transB ? up4(p->K) : up4(p->N);
    if (p->ldy == 0) p->ldy = up4(p->N);
    if (p->ldc == 0) p->ldc = up4(p->N);
    if (p->lda < p->K || p->ldy < p->N || p->ldb < (p->transB ? p->K : p->N)) return OGLE_ERR_INVALID;
    if ((p->lda & 3) || (p->ldb & 3) || (p->ldy & 3)) return OGLE_ERR_ALIGNMENT;
    if (p->bias_mode < 0 || p->bias_mode > 2) return OGLE_ERR_INVALID;
    if (p->bias_mode == 1 && p->ldc < p->N) return OGLE_ERR_INVALID;
    if (p->math_mode < OGLE_MATH_FP32 || p->math_mode > OGLE_MATH_TF32X3) return OGLE_ERR_INVALID;
    return OGLE_OK;
}

extern "C" size_t ogle_cuda_gemm_packed_b_bytes(const OgleGemmParams* pp) {
    if (!pp) return 0;
    OgleGemmParams p = *pp;
    if (normalize_gemm(&p) != OGLE_OK) return 0;
    const size_t half = size_t((p.N + 127) / 128 * 128) * size_t((p.K + 31) / 32 * 32) * sizeof(float);
    return 2 * ((half + 255) / 256 * 256);
}

extern "C" int ogle_cuda_gemm_pack_b(const OgleGemmParams* pp, const float* B, void* packed, ogle_stream_t stream) {
    if (!pp || !B || !packed) return OGLE_ERR_INVALID;
    OgleGemmParams p = *pp;
    int rc = normalize_gemm(&p);
    if (rc != OGLE_OK) return rc;
    if (!aligned16(packed)) return OGLE_ERR_ALIGNMENT;
    const int Kp32 = (p.K + 31) / 32 * 32, Np128 = (p.N + 127) / 128 * 128;
    const size_t half = (size_t(Np128) * Kp32 * sizeof(float) + 255) / 256 * 256;
    float* hi = static_cast<float*>(packed);
    float* lo = reinterpret_cast<float*>(static_cast<char*>(packed) + half);
    const int tiles_n = Np128 / 64;
    const long tiles = (long)(Kp32 / 32) * tiles_n;
    const dim3 grid((unsigned)(tiles < 16L * kNumSMs ? tiles : 16L * kNumSMs));
    launch_overlapped(p.transB ? gemm_pack_b_kernel<true> : gemm_pack_b_kernel<false>, grid, dim3(256), 0, (cudaStream_t)stream, B, hi,
                      reinterpret_cast<__nv_bfloat16*>(lo), p.K, p.N, p.ldb, Kp32, tiles_n, tiles);
    return finish_launch();
}

static int gemm_packed(const OgleGemmParams* pp, const float* A, const void* packed_b, const float* C, float* Y,
                       ogle_stream_t stream, bool overlapped) {
    if (!pp || !A || !packed_b || !Y) return OGLE_ERR_INVALID;
    OgleGemmParams p = *pp;
    int rc = normalize_gemm(&p);
    if (rc != OGLE_OK) return rc;
    if (p.bias_mode && !C) return OGLE_ERR_INVALID;
    if (p.math_mode == OGLE_MATH_FP32) return OGLE_ERR_INVALID;
    if (!aligned16(A) || !aligned16(Y) || !aligned16(packed_b)) return OGLE_ERR_ALIGNMENT;
    const int Kp32 = (p.K + 31) / 32 * 32, Np128 = (p.N + 127) / 128 * 128;
    const size_t half = (size_t(Np128) * Kp32 * sizeof(float) + 255) / 256 * 256;
    const float* hi = static_cast<const float*>(packed_b);
    const float* lo = reinterpret_cast<const float*>(static_cast<const char*>(packed_b) + half);
    // A row at a time is always quicker without the tensor cores (1 x 4096 x 4096 70 us, 31; in one pass 19, 13); up to eight rows while there is
    // little to multiply (4 x 679 x 2536 13.9 us, 13.1; 3 x 2516 x 2240 in one pass 14.9, 19.1), further where split-mode
    // reductions are too long to be cut (2 x 3430 x 700 42 us, 13; 3 x 3784 x 3257 62, 52). Not behind a packing pass, whose
    // B it would wait for no less.
    const bool split = p.math_mode == OGLE_MATH_TF32X3;
    const double products = (double)p.M * p.N * p.K;
    if (!overlapped && (p.M == 1 || (p.M <= 8 && products <= 8e6) || (split && p.M <= 4 && p.K >= 2048 && products <= 4e7))) {
        RowsArgs r = {A, hi, C, reinterpret_cast<const __nv_bfloat16*>(lo), Y, p.M, p.K, p.N, p.lda, p.ldy, p.ldc, Kp32, p.alpha, p.beta, p.bias_mode, 1};
        const long warps = up4(p.N);
        while (r.kw < 8 && warps * r.kw * 2 <= 8 * kNumSMs * 2 && Kp32 >= r.kw * 256) r.kw *= 2;
        cudaStream_t s = (cudaStream_t)stream;
        if (p.M == 1) return launch_rows<1>(r, split, overlapped, s);
        if (p.M == 2) return launch_rows<2>(r, split, overlapped, s);
        if (p.M <= 4) return launch_rows<4>(r, split, overlapped, s);
        return launch_rows<8>(r, split, overlapped, s);
    }
    return launch_gemm_tc_packed(p, A, hi, lo, C, Y, (cudaStream_t)stream, overlapped);
}

extern "C" int ogle_cuda_gemm_packed(const OgleGemmParams* pp, const float* A, const void* packed_b, const float* C,
                                     float* Y, ogle_stream_t stream) {
    return gemm_packed(pp, A, packed_b, C, Y, stream, false);
}

extern "C" int ogle_cuda_gemm_ws(const OgleGemmParams* pp, const float* A, const float* B, const float* C, float* Y,
                                 void* workspace, size_t workspace_bytes, ogle_stream_t stream) {
    if (!pp) return OGLE_ERR_INVALID;
    if (pp->math_mode == OGLE_MATH_FP32) return ogle_cuda_gemm(pp, A, B, C, Y, stream);
    const size_t need = ogle_cuda_gemm_packed_b_bytes(pp);
    if (need == 0) return OGLE_ERR_INVALID;
    if (!workspace || workspace_bytes < need) return OGLE_ERR_INVALID;
    int rc = ogle_cuda_gemm_pack_b(pp, B, workspace, stream);
    if (rc != OGLE_OK) return rc;
    // the product's blocks set up while the packing pass drains, and wait for it before they read anything
    return gemm_packed(pp, A, workspace, C, Y, stream, true);
}

extern "C" int ogle_cuda_gemm(const OgleGemmParams* pp, const float* A, const float* B, const float* C,
                              float* Y, ogle_stream_t stream) {
    if (!pp || !A || !B || !Y) return OGLE_ERR_INVALID;
    OgleGemmParams p = *pp;
    int rc0 = normalize_gemm(&p);
    if (rc0 != OGLE_OK) return rc0;
    if (p.bias_mode && !C) return OGLE_ERR_INVALID;
    if (!aligned16(A) || !aligned16(B) || !aligned16(Y)) return OGLE_ERR_ALIGNMENT;
    cudaStream_t s = (cudaStream_t)stream;
    if (p.math_mode != OGLE_MATH_FP32 && gemm_tc_supported(p, A, B)) return launch_gemm_tc(p, A, B, C, Y, s);
    IgemmArgs g = {};
    g.x = A; g.w = B; g.bias = C; g.y = Y;
    g.M = p.M; g.H = 1; g.W = 1; g.Ho = 1; g.Wo = 1; g.Cs = p.lda;      // (a pixel per row)
    g.kernel = 1; g.stride = 1; g.dil = 1;
    g.Cp = p.K; g.R = p.K;
    g.ldb = p.ldb; g.n_b = p.N; g.N = p.N; g.n_store = p.ldy; g.ldy = p.ldy;
    g.alpha = p.alpha; g.beta = p.beta; g.bias_mode = p.bias_mode; g.ldc = p.ldc;
    return launch_igemm(g, p.transB != 0, s);
}
