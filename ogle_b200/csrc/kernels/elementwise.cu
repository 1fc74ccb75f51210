// Elementwise kernels (relu, clip, add, batchnorm): HBM-bound, 128-bit accesses,
// grid-stride over a grid that is a multiple of the SM count.
#include "common.cuh"

namespace ogle {

enum { EW_RELU = 0, EW_CLIP = 1, EW_ADD = 2, EW_ADD_RELU = 3, EW_ADD_CLIP = 4 };

template <int OP>
__device__ __forceinline__ float4 elementwise_op(float4 v, float4 w, float lo, float hi) {
    if (OP == EW_ADD || OP == EW_ADD_RELU || OP == EW_ADD_CLIP) {
        // binary.glsl then relu.glsl / clip.glsl in one pass: the sum is rounded to fp32 before the
        // activation exactly as when it goes through memory, so the result is bit-identical
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    if (OP == EW_RELU || OP == EW_ADD_RELU) {
        v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
    } else if (OP == EW_CLIP || OP == EW_ADD_CLIP) {
        // clip.glsl:8-9: min(hi, max(lo, v))
        v.x = fminf(hi, fmaxf(lo, v.x)); v.y = fminf(hi, fmaxf(lo, v.y));
        v.z = fminf(hi, fmaxf(lo, v.z)); v.w = fminf(hi, fmaxf(lo, v.w));
    }
    return v;
}

// WIDE: four independent loads (eight with two operands) before the first store, for tensors that give a thread more than
// three elements. Smaller ones are the launch and one trip to memory, and the loop that is never entered costs them its
// instruction fetch: 1.6-2.0 us, 1.8-2.2 with it.
template <int OP, bool WIDE>
__global__ void elementwise_kernel(const float4* __restrict__ a, const float4* __restrict__ b,
                                   float4* __restrict__ y, long n4, float lo, float hi) {
    constexpr bool kBinary = OP >= EW_ADD;
    grid_dependency_trigger();
    grid_dependency_wait();
    const long step = (long)gridDim.x * blockDim.x;
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (; WIDE && i + 3 * step < n4; i += 4 * step) {
        float4 v[4], w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { v[u] = a[i + u * step]; w[u] = kBinary ? b[i + u * step] : zero; }
#pragma unroll
        for (int u = 0; u < 4; ++u) y[i + u * step] = elementwise_op<OP>(v[u], w[u], lo, hi);
    }
    for (; i < n4; i += step) y[i] = elementwise_op<OP>(a[i], kBinary ? b[i] : zero, lo, hi);
}

// (x-mean)/sqrt(var+eps)*gamma+beta, evaluated in that order with IEEE divide and
// sqrt as batchnorm.glsl:31 writes it (not folded into scale/shift), so results
// match the reference's to the last bit per operation.
struct BnChannels { float mean[4], d[4], gamma[4], beta[4]; int real; };

__device__ __forceinline__ BnChannels bn_channels(const float* gamma, const float* beta, const float* mean, const float* var,
                                                  int c, int C, float eps) {
    BnChannels p;
    p.real = C - c;                      // lanes from here on are padding
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const bool ok = l < p.real;
        p.mean[l] = ok ? mean[c + l] : 0.f;
        p.d[l] = ok ? __fsqrt_rn(__fadd_rn(var[c + l], eps)) : 1.f;
        p.gamma[l] = ok ? gamma[c + l] : 0.f;
        p.beta[l] = ok ? beta[c + l] : 0.f;
    }
    return p;
}

__device__ __forceinline__ float4 bn_apply(float4 v, const BnChannels& p) {
    const float in[4] = {v.x, v.y, v.z, v.w};
    float out[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const float t = __fdiv_rn(__fsub_rn(in[l], p.mean[l]), p.d[l]);
        out[l] = l < p.real ? __fadd_rn(__fmul_rn(t, p.gamma[l]), p.beta[l]) : 0.f;
    }
    return make_float4(out[0], out[1], out[2], out[3]);
}

// The grid's stride is a multiple of the channel quads of a pixel, so a thread meets the same four channels in every
// step: their parameters (and the square roots) are taken once and the loop holds no index arithmetic. 32 x 38 x 38 x
// 384 channels: 59 us with the parameters taken per element, 24 us with them hoisted (HBM floor 22 us).
__global__ void __launch_bounds__(256)
batchnorm_kernel(const float4* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                 const float* __restrict__ mean, const float* __restrict__ var, float4* __restrict__ y,
                 long total, int C, int q, float eps) {
    const long step = (long)gridDim.x * blockDim.x;
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= total) return;
    const BnChannels p = bn_channels(gamma, beta, mean, var, int(i % q) * 4, C, eps);
    for (; i + 3 * step < total; i += 4 * step) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = x[i + u * step];
#pragma unroll
        for (int u = 0; u < 4; ++u) y[i + u * step] = bn_apply(v[u], p);
    }
    for (; i < total; i += step) y[i] = bn_apply(x[i], p);
}

// Tensors of one element a thread, whose time is the launch, one trip to memory and the fetch of the kernel's
// instructions (9 x 28 x 32 x 6: 2.6 us, 3.3 by the kernel above; at two elements a thread 7.9 against 6.8), and pixels of
// so many channels that no grid keeps a thread on its own.
__global__ void batchnorm_each_kernel(const float4* __restrict__ x, const float* __restrict__ gamma,
                                      const float* __restrict__ beta, const float* __restrict__ mean,
                                      const float* __restrict__ var, float4* __restrict__ y,
                                      long total, int C, int q, float eps) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        const int c = int(i % q) * 4;
        const float4 v = x[i];
        float in[4] = {v.x, v.y, v.z, v.w};
        float out[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (c + l < C) {
                const float d = __fsqrt_rn(__fadd_rn(var[c + l], eps));
                const float t = __fdiv_rn(__fsub_rn(in[l], mean[c + l]), d);
                out[l] = __fadd_rn(__fmul_rn(t, gamma[c + l]), beta[c + l]);
            } else {
                out[l] = 0.f;
            }
        }
        y[i] = make_float4(out[0], out[1], out[2], out[3]);
    }
}

}  // namespace ogle

using namespace ogle;

template <int OP>
static int launch_elementwise(const float* a, const float* b, float* y, long n, float lo, float hi,
                              ogle_stream_t stream) {
    if (n < 0 || (n & 3)) return OGLE_ERR_INVALID;
    if (n == 0) return OGLE_OK;
    if (!a || !y || (OP >= EW_ADD && !b)) return OGLE_ERR_INVALID;
    if (!aligned16(a) || !aligned16(y) || (b && !aligned16(b))) return OGLE_ERR_ALIGNMENT;
    const int grid = grid_for(n / 4, 256);
    launch_overlapped(n / 4 > 3L * 256 * grid ? elementwise_kernel<OP, true> : elementwise_kernel<OP, false>, dim3(grid), dim3(256), 0,
                      (cudaStream_t)stream, reinterpret_cast<const float4*>(a), reinterpret_cast<const float4*>(b),
                      reinterpret_cast<float4*>(y), n / 4, lo, hi);
    return finish_launch();
}

extern "C" {

int ogle_cuda_relu(const float* x, float* y, long n, ogle_stream_t stream) {
    return launch_elementwise<EW_RELU>(x, nullptr, y, n, 0.f, 0.f, stream);
}
int ogle_cuda_clip(const float* x, float* y, long n, float lo, float hi, ogle_stream_t stream) {
    return launch_elementwise<EW_CLIP>(x, nullptr, y, n, lo, hi, stream);
}
int ogle_cuda_add(const float* a, const float* b, float* y, long n, ogle_stream_t stream) {
    return launch_elementwise<EW_ADD>(a, b, y, n, 0.f, 0.f, stream);
}

int ogle_cuda_add_act(const float* a, const float* b, float* y, long n, int act, float lo, float hi,
                      ogle_stream_t stream) {
    if (act == OGLE_ACT_NONE) return launch_elementwise<EW_ADD>(a, b, y, n, 0.f, 0.f, stream);
    if (act == OGLE_ACT_RELU) return launch_elementwise<EW_ADD_RELU>(a, b, y, n, 0.f, 0.f, stream);
    if (act == OGLE_ACT_CLIP) return launch_elementwise<EW_ADD_CLIP>(a, b, y, n, lo, hi, stream);
    return OGLE_ERR_INVALID;
}

int ogle_cuda_batchnorm(const float* x, const float* gamma, const float* beta, const float* mean,
                        const float* var, float* y, long pixels, int C, int channel_stride,
                        float eps, ogle_stream_t stream) {
    if (pixels < 0 || C <= 0) return OGLE_ERR_INVALID;
    if (channel_stride == 0) channel_stride = up4(C);
    if (channel_stride < C || (channel_stride & 3)) return OGLE_ERR_INVALID;
    if (pixels == 0) return OGLE_OK;
    if (!x || !y || !gamma || !beta || !mean || !var) return OGLE_ERR_INVALID;
    if (!aligned16(x) || !aligned16(y)) return OGLE_ERR_ALIGNMENT;
    const int q = channel_stride / 4;
    const long total = pixels * q;
    int grid = grid_for(total, 256);
    // blocks in multiples of m keep a thread on its channels (see the kernel); a pixel of more quads than the
    // grid has blocks times 256 (over a million channels) takes the other form
    int m = q, r = 256;
    while (r) { const int t = m % r; m = r; r = t; }          // greatest common divisor of q and 256
    m = q / m;
    const bool fixed = m <= kNumSMs * 8 && total > 256L * grid;
    if (fixed) grid = grid < m ? m : grid / m * m;
    if (fixed)
        batchnorm_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4*>(x), gamma, beta, mean, var, reinterpret_cast<float4*>(y), total, C, q, eps);
    else
        batchnorm_each_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4*>(x), gamma, beta, mean, var, reinterpret_cast<float4*>(y), total, C, q, eps);
    return finish_launch();
}

}  // extern "C"
