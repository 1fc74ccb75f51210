// CUDA-core (fp32 FMA) conv2d kernels:
//   - depthwise 3x3 (stride 1 or 2) and a generic depthwise loop: HBM-bound, one
//     thread owns a float4 of channels for a 2x2 patch of output pixels so the
//     overlapping input rows are reused from registers;
//   - grouped (non-depthwise) direct convolution: scalar, rarely used;
// and the dispatch of the dense ones that the tensor cores do not serve (OGLE_MATH_FP32 mode, too few input
// channels) to the small-channel kernel (conv_stem.cu) or the implicit GEMM (igemm.cu).
#include "igemm.cuh"

namespace ogle {

bool dw_tma_supported(const ConvArgs& a);
int launch_dw_tma(const ConvArgs& a, const float* x, const float* w, const float* bias, float* y, cudaStream_t s);

// Bias holds exactly K floats; lanes past K read as zero.
__device__ __forceinline__ float4 load_bias4(const float* bias, int c, int K, int has_bias) {
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has_bias) {
        if (c + 0 < K) b.x = bias[c + 0];
        if (c + 1 < K) b.y = bias[c + 1];
        if (c + 2 < K) b.z = bias[c + 2];
        if (c + 3 < K) b.w = bias[c + 3];
    }
    return b;
}

// ---------------------------------------------------------------- depthwise
template <int S>
__global__ void __launch_bounds__(128)
dw3x3_kernel(const float4* __restrict__ x, const float4* __restrict__ w, const float* __restrict__ bias,
             float4* __restrict__ y, ConvArgs a) {
    constexpr int K = 3, TY = 2, TX = 2;
    constexpr int PH = (TY - 1) * S + K, PW = (TX - 1) * S + K;
    const int C4 = a.Kp >> 2, in_q = a.Cs >> 2, out_q = a.Ks >> 2, off_q = a.koff >> 2;
    const int gy = (a.Ho + TY - 1) / TY, gx = (a.Wo + TX - 1) / TX;
    const long total = (long)a.N * gy * gx * C4;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        long t = i;
        const int c4 = int(t % C4); t /= C4;
        const int px = int(t % gx); t /= gx;
        const int py = int(t % gy); t /= gy;
        const int n = int(t);
        const int oy0 = py * TY, ox0 = px * TX;
        const int iy0 = oy0 * S - a.pad, ix0 = ox0 * S - a.pad;
        float4 wk[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) wk[k] = w[k * C4 + c4];
        const float4 b = load_bias4(bias, c4 * 4, a.K, a.has_bias);
        float4 acc[TY][TX];
#pragma unroll
        for (int ty = 0; ty < TY; ++ty)
#pragma unroll
            for (int tx = 0; tx < TX; ++tx) acc[ty][tx] = b;
#pragma unroll
        for (int r = 0; r < PH; ++r) {
            const int iy = iy0 + r;
            if (iy < 0 || iy >= a.H) continue;  // zero padding: skipped taps add nothing
            const float4* row = x + ((long)n * a.H + iy) * a.W * in_q + c4;
            float4 v[PW];
#pragma unroll
            for (int c = 0; c < PW; ++c) {
                const int ix = ix0 + c;
                v[c] = (ix >= 0 && ix < a.W) ? row[(long)ix * in_q] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int ty = 0; ty < TY; ++ty) {
                if (r < ty * S || r >= ty * S + K) continue;
                const int ky = r - ty * S;
#pragma unroll
                for (int tx = 0; tx < TX; ++tx)
#pragma unroll
                    for (int kx = 0; kx < K; ++kx) {
                        const float4 f = wk[ky * 3 + kx];
                        const float4 u = v[tx * S + kx];
                        acc[ty][tx].x = fmaf(f.x, u.x, acc[ty][tx].x);
                        acc[ty][tx].y = fmaf(f.y, u.y, acc[ty][tx].y);
                        acc[ty][tx].z = fmaf(f.z, u.z, acc[ty][tx].z);
                        acc[ty][tx].w = fmaf(f.w, u.w, acc[ty][tx].w);
                    }
            }
        }
#pragma unroll
        for (int ty = 0; ty < TY; ++ty)
#pragma unroll
            for (int tx = 0; tx < TX; ++tx) {
                const int oy = oy0 + ty, ox = ox0 + tx;
                if (oy >= a.Ho || ox >= a.Wo) continue;
                float4 r = apply_act4(acc[ty][tx], a.act, a.lo, a.hi);
                // lanes past K stay zero (their weights and bias are zero; a clip
                // with lo > 0 must not lift them)
                const int c = c4 * 4;
                if (c >= a.K) r.x = 0.f;
                if (c + 1 >= a.K) r.y = 0.f;
                if (c + 2 >= a.K) r.z = 0.f;
                if (c + 3 >= a.K) r.w = 0.f;
                y[(((long)n * a.Ho + oy) * a.Wo + ox) * out_q + off_q + c4] = r;
            }
    }
}


// Any kernel size / dilation / stride, depthwise.
__global__ void dw_generic_kernel(const float4* __restrict__ x, const float4* __restrict__ w,
                                  const float* __restrict__ bias, float4* __restrict__ y, ConvArgs a) {
    const int C4 = a.Kp >> 2, in_q = a.Cs >> 2, out_q = a.Ks >> 2, off_q = a.koff >> 2;
    const long total = a.M * C4;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        long t = i;
        const int c4 = int(t % C4); t /= C4;
        const int ox = int(t % a.Wo); t /= a.Wo;
        const int oy = int(t % a.Ho); t /= a.Ho;
        const int n = int(t);
        float4 acc = load_bias4(bias, c4 * 4, a.K, a.has_bias);
        for (int ky = 0; ky < a.kernel; ++ky)
            for (int kx = 0; kx < a.kernel; ++kx) {
                const int iy = oy * a.stride + ky * a.dil - a.pad, ix = ox * a.stride + kx * a.dil - a.pad;
                if (iy < 0 || iy >= a.H || ix < 0 || ix >= a.W) continue;
                const float4 u = x[(((long)n * a.H + iy) * a.W + ix) * in_q + c4];
                const float4 f = w[(ky * a.kernel + kx) * C4 + c4];
                acc.x = fmaf(f.x, u.x, acc.x); acc.y = fmaf(f.y, u.y, acc.y);
                acc.z = fmaf(f.z, u.z, acc.z); acc.w = fmaf(f.w, u.w, acc.w);
            }
        float4 r = apply_act4(acc, a.act, a.lo, a.hi);
        const int c = c4 * 4;
        if (c >= a.K) r.x = 0.f;
        if (c + 1 >= a.K) r.y = 0.f;
        if (c + 2 >= a.K) r.z = 0.f;
        if (c + 3 >= a.K) r.w = 0.f;
        y[(((long)n * a.Ho + oy) * a.Wo + ox) * out_q + off_q + c4] = r;
    }
}

// ------------------------------------------------------------------ grouped
// One thread per output scalar; packed filter [tap][Cp][Kp] with Cp = round_up(C/group,4).
__global__ void grouped_kernel(const float* __restrict__ x, const float* __restrict__ w,
                               const float* __restrict__ bias, float* __restrict__ y, ConvArgs a) {
    const long total = a.M * a.Kp;
    const int Cg = a.C / a.group, Kg = a.K / a.group;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        long t = i;
        const int k = int(t % a.Kp); t /= a.Kp;
        const int ox = int(t % a.Wo); t /= a.Wo;
        const int oy = int(t % a.Ho); t /= a.Ho;
        const int n = int(t);
        float r = 0.f;
        if (k < a.K) {
            const int g = k / Kg;
            float acc = 0.f;
            for (int ky = 0; ky < a.kernel; ++ky)
                for (int kx = 0; kx < a.kernel; ++kx) {
                    const int iy = oy * a.stride + ky * a.dil - a.pad, ix = ox * a.stride + kx * a.dil - a.pad;
                    if (iy < 0 || iy >= a.H || ix < 0 || ix >= a.W) continue;
                    const float* px = x + (((long)n * a.H + iy) * a.W + ix) * a.Cs + g * Cg;
                    const float* pw = w + (long)(ky * a.kernel + kx) * a.Cp * a.Kp + k;
                    for (int c = 0; c < Cg; ++c) acc = fmaf(px[c], pw[(long)c * a.Kp], acc);
                }
            acc += a.has_bias ? bias[k] : 0.f;
            r = apply_act(acc, a.act, a.lo, a.hi);
        }
        y[(((long)n * a.Ho + oy) * a.Wo + ox) * a.Ks + a.koff + k] = r;
    }
}

bool conv_smallc_supported(const ConvArgs& a);
int launch_conv_smallc(const ConvArgs& a, const float* x, const float* w_tap_major, const float* bias, float* y,
                       cudaStream_t s);

static IgemmArgs igemm_args(const ConvArgs& a, const float* x, const float* w, const float* bias, float* y) {
    IgemmArgs g = {};
    g.x = x; g.w = w; g.bias = bias; g.y = y;
    g.M = a.M; g.H = a.H; g.W = a.W; g.Ho = a.Ho; g.Wo = a.Wo; g.Cs = a.Cs;
    g.kernel = a.kernel; g.stride = a.stride; g.pad = a.pad; g.dil = a.dil;
    g.Cp = a.Cp; g.R = a.kernel * a.kernel * a.Cp;
    g.ldb = a.Kp; g.n_b = a.Kp; g.N = a.K; g.n_store = a.Kp;
    g.ldy = a.Ks; g.yoff = a.koff;
    g.act = a.act; g.lo = a.lo; g.hi = a.hi;
    g.alpha = 1.f; g.beta = 1.f; g.bias_mode = a.has_bias ? 2 : 0;
    return g;
}

int launch_conv_simt(const ConvArgs& a, int variant, const float* x, const float* w,
                     const float* bias, float* y, cudaStream_t s) {
    if (variant == CONV_DEPTHWISE) {
        const float4* x4 = reinterpret_cast<const float4*>(x);
        const float4* w4 = reinterpret_cast<const float4*>(w);
        const float* b4 = bias;
        float4* y4 = reinterpret_cast<float4*>(y);
        const int C4 = a.Kp / 4;
        if (dw_tma_supported(a)) {
            return launch_dw_tma(a, x, w, bias, y, s);
        } else if (a.kernel == 3 && a.dil == 1 && (a.stride == 1 || a.stride == 2)) {
            const long items = (long)a.N * ((a.Ho + 1) / 2) * ((a.Wo + 1) / 2) * C4;
            if (a.stride == 1) dw3x3_kernel<1><<<grid_for(items, 128, 16), 128, 0, s>>>(x4, w4, b4, y4, a);
            else dw3x3_kernel<2><<<grid_for(items, 128, 16), 128, 0, s>>>(x4, w4, b4, y4, a);
        } else {
            dw_generic_kernel<<<grid_for(a.M * C4, 256), 256, 0, s>>>(x4, w4, b4, y4, a);
        }
        return finish_launch();
    }
    if (variant == CONV_GROUPED) {
        grouped_kernel<<<grid_for(a.M * a.Kp, 256), 256, 0, s>>>(x, w, bias, y, a);
        return finish_launch();
    }
    if (variant == CONV_GENERAL && conv_smallc_supported(a)) return launch_conv_smallc(a, x, w, bias, y, s);
    // the kernel numbers input pixels in 32 bits: larger batches go in groups of images (a single image that is
    // larger goes alone, numbered in 64)
    const long pixels = (long)a.H * a.W;
    long group = pixels * a.N < 0x7fffffffL ? a.N : 0x7fffffffL / pixels;
    if (group < 1) group = 1;
    if (group < a.N) {
        for (int n = 0; n < a.N; n += (int)group) {
            ConvArgs part = a;
            part.N = a.N - n < group ? a.N - n : (int)group;
            part.M = (long)part.N * a.Ho * a.Wo;
            const int rc = launch_conv_simt(part, variant, x + n * pixels * a.Cs, w, bias, y + (long)n * a.Ho * a.Wo * a.Ks, s);
            if (rc != OGLE_OK) return rc;
        }
        return OGLE_OK;
    }
    return launch_igemm(igemm_args(a, x, w, bias, y), false, s);
}

const char* conv_igemm_name(const ConvArgs& a) {
    const long pixels = (long)a.H * a.W;
    ConvArgs part = a;                               // of a batch that goes in groups, the first
    if (pixels * a.N >= 0x7fffffffL) {
        part.N = pixels < 0x7fffffffL ? (int)(0x7fffffffL / pixels) : 1;
        part.M = (long)part.N * a.Ho * a.Wo;
    }
    const char* name = "";
    launch_igemm(igemm_args(part, nullptr, nullptr, nullptr, nullptr), false, nullptr, &name);
    return name;
}

}  // namespace ogle
