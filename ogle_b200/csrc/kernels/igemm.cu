// fp32 contraction on the CUDA cores (OGLE_MATH_FP32, and convolutions with too few input channels for the tensor
// cores): convolution as implicit GEMM and gemm, one kernel.
//
//  * A block computes a BM x BN tile, a thread 8 x 8 of it. The multiply-adds are packed (fma.rn.f32x2 over two
//    adjacent output columns): the same IEEE fma per lane in the same order as scalar code, in half the issue slots,
//    which leaves room for the shared-memory loads and operand moves between them.
//  * Both operands come through a ring of three stages filled by 16-byte asynchronous copies (zero-filled outside the
//    image and past the ends). A keeps its channels contiguous - no transposition on the way - in rows of 20 floats,
//    so that the rows a warp reads together start in different banks.
//  * A launch with few tiles splits the reduction over the blocks of a cluster (2, 4 or 8): every block leaves its
//    partial tile in its own shared memory, and each adds up a band of rows over the cluster, in rank order, through
//    distributed shared memory: no scratch memory, no second launch, the same bits every time.
//
// Large layers run at 46-47 TFLOP/s (3x3 256 -> 256 at 38 x 38 x 32 images: 1658 -> 1183 us); packed and scalar
// multiply-adds measure within 5 % of each other there, so it is the FP32 pipe and its operand reads, not issue slots
// or shared memory (42 % busy), that set the pace. At 8 images the gain is in filling the SMs: ResNet's 512-channel
// 3x3 layers at 7 x 7 were 32 blocks (407 us, now 69), the 256-channel ones at 14 x 14 205 us, now 55; the network
// 3010 -> 957 us.
#include "igemm.cuh"

namespace ogle {
namespace {

constexpr int kBK = 16;
constexpr int kALd = kBK + 4;        // floats per row of a k-contiguous tile
constexpr int kStages = 3;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16 bytes from global to shared memory, of which the first `bytes` are read and the rest zeros.
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ float4 load_cluster(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four output columns of row m from column n on: bias, activation, zeros past N.
__device__ __forceinline__ void store4(const IgemmArgs& a, long m, int n, float4 acc) {
    if (m >= a.M || n >= a.n_store) return;
    float v[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (n + l >= a.N) { v[l] = 0.f; continue; }
        v[l] *= a.alpha;
        if (a.bias_mode == 2) v[l] = fmaf(a.beta, a.bias[n + l], v[l]);
        else if (a.bias_mode == 1) v[l] = fmaf(a.beta, a.bias[m * a.ldc + n + l], v[l]);
        v[l] = apply_act(v[l], a.act, a.lo, a.hi);
    }
    *reinterpret_cast<float4*>(a.y + m * a.ldy + a.yoff + n) = make_float4(v[0], v[1], v[2], v[3]);
}

// Pixel: the type that numbers input pixels.
template <int BM, int BN, bool TRANSB, typename Pixel>
__global__ void __launch_bounds__(BM * BN / 64, BM * BN / 64 >= 256 ? 2 : (BM * BN / 64 >= 128 ? 3 : 6))
conv_igemm_kernel(const IgemmArgs a) {
    constexpr int NT = BM * BN / 64, TX = BN / 8, TY = BM / 8;
    constexpr int A_FLOATS = BM * kALd, B_FLOATS = TRANSB ? BN * kALd : kBK * BN;
    constexpr int A_COPIES = BM * (kBK / 4) / NT, B_COPIES = BN * (kBK / 4) / NT;
    static_assert(A_COPIES * NT == BM * (kBK / 4) && B_COPIES * NT == BN * (kBK / 4), "copies divide over the threads");
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x;
    const long m0 = (long)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    const int splits = gridDim.z, rank = blockIdx.z;
    // this block's share of the reduction, in steps of kBK
    const int steps = (a.R + kBK - 1) / kBK, per = (steps + splits - 1) / splits;
    const int first = min(rank * per, steps), count = min(first + per, steps) - first;

    // Copies of A: this thread always moves the same 4 reduction elements (kq) of the same rows.
    const int kq = (tid & 3) * 4;
    int iy0[A_COPIES], ix0[A_COPIES];
    Pixel pix[A_COPIES];
#pragma unroll
    for (int j = 0; j < A_COPIES; ++j) {
        const long m = m0 + (tid >> 2) + j * (NT / 4);
        const long mm = m < a.M ? m : 0;
        const int ox = int(mm % a.Wo);
        const long t = mm / a.Wo;
        const int oy = int(t % a.Ho);
        iy0[j] = m < a.M ? oy * a.stride - a.pad : -0x40000000;       // a row past the end lies outside every image
        ix0[j] = ox * a.stride - a.pad;
        pix[j] = (Pixel)(t / a.Ho) * a.H * a.W + (Pixel)(oy * a.stride - a.pad) * a.W + ix0[j];
    }
    int c, ky, kx;                   // the elements' channel and filter tap, carried from step to step
    {
        const int r = first * kBK + kq, tap = r / a.Cp;
        c = r - tap * a.Cp;
        ky = tap / a.kernel;
        kx = tap - ky * a.kernel;
    }
    int r_next = first * kBK;        // first reduction index of the next step to be loaded
    auto load_step = [&](int stage) {
        float* sa = smem + stage * (A_FLOATS + B_FLOATS);
        const uint32_t da = smem_addr(sa), db = smem_addr(sa + A_FLOATS);
        const int tail_a = min(4, a.Cp - c) * 4;                       // a matrix row may end between 16-byte pieces
#pragma unroll
        for (int j = 0; j < A_COPIES; ++j) {
            const int iy = iy0[j] + ky * a.dil, ix = ix0[j] + kx * a.dil;
            const bool ok = r_next + kq < a.R && (unsigned)iy < (unsigned)a.H && (unsigned)ix < (unsigned)a.W;
            const float* src = ok ? a.x + (long)(pix[j] + ((Pixel)ky * a.W + kx) * a.dil) * a.Cs + c : a.x;
            copy16(da + (((tid >> 2) + j * (NT / 4)) * kALd + kq) * 4, src, ok ? tail_a : 0);
        }
#pragma unroll
        for (int j = 0; j < B_COPIES; ++j) {
            if (TRANSB) {
                const int n = n0 + (tid >> 2) + j * (NT / 4), r = r_next + kq;
                const bool ok = n < a.n_b && r < a.R;
                copy16(db + (((tid >> 2) + j * (NT / 4)) * kALd + kq) * 4, ok ? a.w + (long)n * a.ldb + r : a.w,
                       ok ? min(4, a.R - r) * 4 : 0);
            } else {
                const int idx = tid + j * NT, kr = idx / (BN / 4), nc = idx % (BN / 4) * 4;
                const int n = n0 + nc, r = r_next + kr;
                const bool ok = n < a.n_b && r < a.R;
                copy16(db + (kr * BN + nc) * 4, ok ? a.w + (long)r * a.ldb + n : a.w, ok ? min(4, a.n_b - n) * 4 : 0);
            }
        }
        r_next += kBK;
        c += kBK;
        while (c >= a.Cp) { c -= a.Cp; if (++kx == a.kernel) { kx = 0; ++ky; } }
    };

    const int tx = tid % TX, ty = tid / TX;      // rows ty + i * TY; columns tx * 4 and BN / 2 + tx * 4
    unsigned long long acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

#pragma unroll
    for (int p = 0; p < kStages - 1; ++p) {
        if (p < count) load_step(p);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    for (int t = 0; t < count; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();             // this step's tiles are complete, and everyone is done with the stage refilled next
        if (t + kStages - 1 < count) load_step(stage == 0 ? kStages - 1 : stage - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* sa = smem + stage * (A_FLOATS + B_FLOATS);
        const float* sb = sa + A_FLOATS;
#pragma unroll
        for (int k2 = 0; k2 < kBK; k2 += 2) {
            float2 av[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float2*>(sa + (ty + i * TY) * kALd + k2);
            float2 bt[8];
            if (TRANSB) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    bt[j] = *reinterpret_cast<const float2*>(sb + ((j >> 2) * (BN / 2) + tx * 4 + (j & 3)) * kALd + k2);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                unsigned long long b[4];
                if (TRANSB) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        b[j] = k ? pack2(bt[2 * j].y, bt[2 * j + 1].y) : pack2(bt[2 * j].x, bt[2 * j + 1].x);
                } else {
                    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(sb + (k2 + k) * BN + tx * 4);
                    const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(sb + (k2 + k) * BN + BN / 2 + tx * 4);
                    b[0] = b0.x; b[1] = b0.y; b[2] = b1.x; b[3] = b1.y;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float u = k ? av[i].y : av[i].x;
                    const unsigned long long uu = pack2(u, u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(acc[i][j], uu, b[j]);
                }
            }
        }
        if (++stage == kStages) stage = 0;
    }

    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 p = unpack2(acc[i][h * 2]), q = unpack2(acc[i][h * 2 + 1]);
                store4(a, m0 + ty + i * TY, n0 + h * (BN / 2) + tx * 4, make_float4(p.x, p.y, q.x, q.y));
            }
        return;
    }
    // split reduction: the ring is idle now and takes the partial tile
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float4* part = reinterpret_cast<float4*>(smem);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 p = unpack2(acc[i][h * 2]), q = unpack2(acc[i][h * 2 + 1]);
            part[(ty + i * TY) * (BN / 4) + h * (BN / 8) + tx] = make_float4(p.x, p.y, q.x, q.y);
        }
    cluster_sync();
    const int band = BM / splits * (BN / 4);     // float4s of this block's rows
    for (int i = tid; i < band; i += NT) {
        const int at = rank * band + i;
        const uint32_t addr = smem_addr(part + at);
        float4 sum = load_cluster(addr, 0);
        for (int p = 1; p < splits; ++p) {
            const float4 v = load_cluster(addr, (uint32_t)p);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        store4(a, m0 + at / (BN / 4), n0 + at % (BN / 4) * 4, sum);
    }
    cluster_sync();                              // no block leaves while another still reads its partial tile
}

template <int BM, int BN, bool TRANSB, typename Pixel = int>
int launch(const IgemmArgs& a, int splits, cudaStream_t s) {
    constexpr size_t ring = (size_t)kStages * (BM * kALd + (TRANSB ? BN * kALd : kBK * BN)) * sizeof(float);
    constexpr size_t tile = (size_t)BM * BN * sizeof(float);
    const size_t smem = splits > 1 && tile > ring ? tile : ring;
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        cudaError_t e = cudaFuncSetAttribute(conv_igemm_kernel<BM, BN, TRANSB, Pixel>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(tile > ring ? tile : ring));
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(div_up(a.M, BM), div_up(a.n_store, BN), splits);
    cfg.blockDim = dim3(BM * BN / 64);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = splits;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, conv_igemm_kernel<BM, BN, TRANSB, Pixel>, a);
    if (e != cudaSuccess) { set_last_error(e); (void)cudaGetLastError(); return OGLE_ERR_CUDA; }
    return finish_launch();
}

}  // namespace

// Tile and split. The large tiles read the least through L2 per multiply-add and are taken where they alone give
// every SM its two (128 x 128) or four (128 x 64) resident blocks; 128 x 32 serves narrow outputs over many rows.
// Everything else runs on 64 x 64 tiles with the reduction split so that the SMs fill: the cost of a split is
// (blocks on the busiest SM, at least the four that keep its FP32 pipes busy) x (steps of a block, plus about six
// for its start, its partial tile and the cluster's barriers).
int launch_igemm(const IgemmArgs& a, bool trans_b, cudaStream_t s) {
    const long m128 = (a.M + 127) / 128, m64 = (a.M + 63) / 64;
    if (m64 > 0x7fffffffL || (a.n_store + 63) / 64 > 65535) return OGLE_ERR_UNSUPPORTED;
    const bool large = a.M / ((long)a.Ho * a.Wo) * a.H * a.W > 0x7fffffffL;       // (one image of 2^31 pixels or more)
    if (!trans_b && !large) {
        if (a.n_store > 64 && m128 * ((a.n_store + 127) / 128) >= 2 * kNumSMs && (a.n_store % 128 == 0 || a.n_store % 128 > 64))
            return launch<128, 128, false>(a, 1, s);
        if (a.n_store > 32 && m128 * ((a.n_store + 63) / 64) >= 4 * kNumSMs) return launch<128, 64, false>(a, 1, s);
        if (a.n_store <= 32 && m128 >= 4 * kNumSMs) return launch<128, 32, false>(a, 1, s);
    }
    const long tiles = m64 * ((a.n_store + 63) / 64);
    const int steps = (a.R + kBK - 1) / kBK;
    int best = 1;
    double best_cost = -1.0;
    for (int k = 1; k <= 8 && k <= steps; k *= 2) {
        const double blocks = (double)((tiles * k + kNumSMs - 1) / kNumSMs);
        const double cost = (blocks < 4 ? 4.0 : blocks) * ((steps + k - 1) / k + 6.0);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = k; }
    }
    if (large) return launch<64, 64, false, long>(a, best, s);
    return trans_b ? launch<64, 64, true>(a, best, s) : launch<64, 64, false>(a, best, s);
}

}  // namespace ogle
