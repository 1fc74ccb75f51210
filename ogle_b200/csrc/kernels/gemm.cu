// Gemm: Y[M,N] = alpha * A[M,K] * (transB ? B[N,K]^T : B[K,N]) + beta * C.
// OGLE_MATH_FP32 runs the CUDA-core kernel of igemm.cu; the TF32 modes
// go to the tcgen05 path when the shape allows it.
#include <cuda_bf16.h>

#include "few_rows.cuh"
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
    // A row at a time is always quicker without the tensor cores (in graphs: 1 x 512 x 1000 8.6 -> 3.2 us; 1 x 4096 x 4096 70 ->
    // 31, in one pass 19 -> 13), up to eight rows while there is little to multiply (8 x 512 x 1000 8.7 -> 5.0; 6 x 911 x
    // 1257 9.5 -> 13), further where split-mode reductions are too long to be cut (2 x 3430 x 700 42 -> 13, 3 x 3784 x 3257
    // 62 -> 52), or nearly so: from 2660 elements on ranges in clusters would move the result too far (choose_cluster). Below,
    // four rows over columns that give each SM less than two blocks of a warp a column are no better off (4 x 2500 x 1500
    // 19.4 -> 22), nor is a warp of four columns (3 x 2500 x 5000 26 -> 41). Not behind a packing pass, whose B it would wait for no less.
    const bool split = p.math_mode == OGLE_MATH_TF32X3;
    const double products = (double)p.M * p.N * p.K;
    const bool cut = p.K <= 2660 && (few_rows_cols(p.N) > 1 || (p.M == 4 && p.N < 16 * kNumSMs && few_rows_warps(p.N, Kp32) == 1));
    if (!overlapped && (p.M == 1 || (p.M <= 8 && products <= 6e6) || (split && p.M <= 4 && p.K >= 2048 && products <= 4e7 && !cut))) {
        FewRowsArgs r = {};
        r.x = A; r.hi = hi; r.lo = split ? lo : nullptr; r.bias = C; r.y = Y;
        r.M = p.M; r.N = p.N; r.C = p.K; r.Cp32 = Kp32; r.ldx = p.lda; r.ldy = p.ldy; r.ldc = p.ldc;
        r.kernel = 1;
        r.alpha = p.alpha; r.beta = p.beta; r.bias_mode = p.bias_mode;
        return launch_few_rows(r, (cudaStream_t)stream);
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
