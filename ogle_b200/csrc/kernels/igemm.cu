// fp32 contraction on the CUDA cores (OGLE_MATH_FP32, and convolutions with too few input channels for the tensor
// cores): convolution as implicit GEMM and gemm, one kernel.
//
//  * A block computes a BM x BN tile, a thread TM x 8 of it: 8 x 8 where the reduction is long, 2 x 8 - four times the
//    threads, each with a quarter of the instructions - where a launch is over before a warp has worked off 64 outputs
//    (455 pixels, 16 -> 9 channels: 6.4 us by two warps a block, 3.3 by four; 7020 x 84 x 216: 18.3, 16.4). The multiply-adds are packed (fma.rn.f32x2 over two
//    adjacent output columns): the same IEEE fma per lane in the same order as scalar code, in half the issue slots,
//    which leaves room for the shared-memory loads and operand moves between them.
//  * Both operands come through a ring of three stages filled by 16-byte asynchronous copies (zero-filled outside the
//    image and past the ends), but for a transposed B, which is turned over through registers (read as it lies, its rows
//    put four lanes on a bank: 2001 x 1613 x 3423 984 us, now 532). A keeps its channels contiguous - no transposition on the way - in rows of 20 floats,
//    so that the rows a warp reads together start in different banks.
//  * A launch with few tiles splits the reduction over the blocks of a cluster (2, 4 or 8): every block leaves its
//    partial tile in its own shared memory, and each adds up a band of rows over the cluster, in rank order, through
//    distributed shared memory: no scratch memory, no second launch, the same bits every time.
//  * Longer reductions of more than 32 columns take conv_igemm_tma_kernel where that is the faster (launch_igemm): both
//    operands by the copy engine, 4 x 16 outputs a thread. A thread's own copies and their addresses were an eighth of the
//    instructions, and 8 x 8 outputs move 16 multiplicands a step into pairs where 4 x 16 move 8: in registers and shared
//    memory alone the two reach 56 and 60 TFLOP/s (a multiply-add by itself 65), as kernels 46 and 54.
//  * Bias and activation are applied on the way out of a tile in shared memory, row by row, not to 64 registers.
//
// Large layers run at 46-47 TFLOP/s (3x3 256 -> 256 at 38 x 38 x 32 images: 1658 -> 1183 us); packed and scalar
// multiply-adds measure within 5 % of each other there, so it is the FP32 pipe and its operand reads, not issue slots
// or shared memory (42 % busy), that set the pace. At 8 images the gain is in filling the SMs: ResNet's 512-channel
// 3x3 layers at 7 x 7 were 32 blocks (407 us, then 69), the 256-channel ones at 14 x 14 205 us, then 55; the network
// 3010 -> 942 us, and 882 with conv_igemm_tma_kernel.
#include "igemm.cuh"
#include "tc_common.cuh"
#include "tma_host.h"

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

// Bias of four output columns (row bias).
__device__ __forceinline__ float4 row_bias(const IgemmArgs& a, int n) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.bias_mode == 2) {
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (n + l < a.N) v[l] = __ldg(a.bias + n + l);
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// One value of row m, column n: bias, activation, zero past N.
__device__ __forceinline__ float finish(const IgemmArgs& a, long m, int n, float v, float bias) {
    if (n >= a.N) return 0.f;
    v *= a.alpha;
    if (a.bias_mode == 2) v = fmaf(a.beta, bias, v);
    else if (a.bias_mode == 1) v = fmaf(a.beta, __ldg(a.bias + m * a.ldc + n), v);
    return apply_act(v, a.act, a.lo, a.hi);
}
// Four output columns of row m from column n on.
__device__ __forceinline__ void store4(const IgemmArgs& a, long m, int n, float4 acc, float4 bias) {
    if (m >= a.M || n >= a.n_store) return;
    if (n + 4 <= a.N && a.bias_mode != 1) {
        acc = make_float4(acc.x * a.alpha, acc.y * a.alpha, acc.z * a.alpha, acc.w * a.alpha);
        if (a.bias_mode == 2)
            acc = make_float4(fmaf(a.beta, bias.x, acc.x), fmaf(a.beta, bias.y, acc.y), fmaf(a.beta, bias.z, acc.z), fmaf(a.beta, bias.w, acc.w));
        *reinterpret_cast<float4*>(a.y + m * a.ldy + a.yoff + n) = apply_act4(acc, a.act, a.lo, a.hi);
        return;
    }
    *reinterpret_cast<float4*>(a.y + m * a.ldy + a.yoff + n) =
        make_float4(finish(a, m, n, acc.x, bias.x), finish(a, m, n + 1, acc.y, bias.y), finish(a, m, n + 2, acc.z, bias.z),
                    finish(a, m, n + 3, acc.w, bias.w));
}

// TM: rows of a thread's outputs. Pixel: the type that numbers pixels (unsigned, or long where those are not enough).
template <int BM, int BN, int TM, bool TRANSB, typename Pixel>
__global__ void __launch_bounds__(BM * BN / (8 * TM), TM == 8 ? (BM * BN >= 16384 ? 2 : (BM * BN >= 8192 ? 3 : 6)) : (TM == 4 ? 8 : 1024 / (BM * BN / (8 * TM))))
conv_igemm_kernel(const IgemmArgs a) {
    constexpr int NT = BM * BN / (8 * TM), TX = BN / 8, TY = BM / TM;
    constexpr int A_FLOATS = BM * kALd, B_FLOATS = kBK * BN;
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
        const Pixel m = (Pixel)m0 + (tid >> 2) + j * (NT / 4);
        const Pixel mm = m < (Pixel)a.M ? m : 0;
        const Pixel t = mm / (Pixel)a.Wo;
        const int ox = int(mm - t * (Pixel)a.Wo);
        const int oy = int(t % (Pixel)a.Ho);
        iy0[j] = m < (Pixel)a.M ? oy * a.stride - a.pad : -0x40000000;       // a row past the end lies outside every image
        ix0[j] = ox * a.stride - a.pad;
        pix[j] = t / (Pixel)a.Ho * a.H * a.W + (Pixel)(oy * a.stride - a.pad) * a.W + ix0[j];
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
        for (int j = 0; j < (TRANSB ? 0 : B_COPIES); ++j) {
            const int idx = tid + j * NT, kr = idx / (BN / 4), nc = idx % (BN / 4) * 4;
            const int n = n0 + nc, r = r_next + kr;
            const bool ok = n < a.n_b && r < a.R;
            copy16(db + (kr * BN + nc) * 4, ok ? a.w + (long)r * a.ldb + n : a.w, ok ? min(4, a.n_b - n) * 4 : 0);
        }
        r_next += kBK;
        c += kBK;
        while (c >= a.Cp) { c -= a.Cp; if (++kx == a.kernel) { kx = 0; ++ky; } }
    };

    // A transposed B is turned over on its way into the ring: this thread's 16-byte pieces (four reduction elements of a
    // column) wait in registers for a step and are then stored down their columns; columns trade places in groups of
    // eight with the reduction index, so that a warp stores to different banks.
    float4 held[TRANSB ? B_COPIES : 1];
    auto fetch_b = [&](int step) {
#pragma unroll
        for (int j = 0; j < (TRANSB ? B_COPIES : 0); ++j) {
            const int n = n0 + ((tid + j * NT) >> 2), r = (first + step) * kBK + kq;
            held[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* src = a.w + (long)n * a.ldb + r;
            if (n < a.n_b && r + 3 < a.R) {
                held[j] = __ldg(reinterpret_cast<const float4*>(src));
            } else if (n < a.n_b) {                              // what lies past the end of a row is not ours to read
                if (r < a.R) held[j].x = __ldg(src);
                if (r + 1 < a.R) held[j].y = __ldg(src + 1);
                if (r + 2 < a.R) held[j].z = __ldg(src + 2);
            }
        }
    };
    auto put_b = [&](int stage) {
        float* sb = smem + stage * (A_FLOATS + B_FLOATS) + A_FLOATS + kq * BN;
#pragma unroll
        for (int j = 0; j < (TRANSB ? B_COPIES : 0); ++j) {
            const int col = ((tid + j * NT) >> 2) ^ (2 * kq);
            sb[col] = held[j].x; sb[BN + col] = held[j].y; sb[2 * BN + col] = held[j].z; sb[3 * BN + col] = held[j].w;
        }
    };

    // rows ty + i * TY; columns tx * 4 and BN / 2 + tx * 4, four each
    const int tx = tid % TX, ty = tid / TX;
    unsigned long long acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

#pragma unroll
    for (int p = 0; p < kStages - 1; ++p) {
        if (p < count) {
            load_step(p);
            if (TRANSB) { fetch_b(p); put_b(p); }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (TRANSB && kStages - 1 < count) fetch_b(kStages - 1);
    int stage = 0;
    for (int t = 0; t < count; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();             // this step's tiles are complete, and everyone is done with the stage refilled next
        if (t + kStages - 1 < count) {
            const int free = stage == 0 ? kStages - 1 : stage - 1;
            load_step(free);
            if (TRANSB) {
                put_b(free);
                if (t + kStages < count) fetch_b(t + kStages);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* sa = smem + stage * (A_FLOATS + B_FLOATS);
        const float* sb = sa + A_FLOATS;
#pragma unroll
        for (int k2 = 0; k2 < kBK; k2 += 2) {
            float2 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float2*>(sa + (ty + i * TY) * kALd + k2);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int swap = TRANSB ? (k2 + k) / 4 * 8 : 0;
                const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(sb + (k2 + k) * BN + ((tx * 4) ^ swap));
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(sb + (k2 + k) * BN + ((BN / 2 + tx * 4) ^ swap));
                const unsigned long long b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float u = k ? av[i].y : av[i].x;
                    const unsigned long long uu = pack2(u, u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(acc[i][j], uu, b[j]);
                }
            }
        }
        if (++stage == kStages) stage = 0;
    }

    // Few rows a thread: finished and stored from registers.
    if (TM == 2 && splits == 1) {
        const float4 bias[2] = {row_bias(a, n0 + tx * 4), row_bias(a, n0 + BN / 2 + tx * 4)};
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 p = unpack2(acc[i][h * 2]), q = unpack2(acc[i][h * 2 + 1]);
                store4(a, m0 + ty + i * TY, n0 + h * (BN / 2) + tx * 4, make_float4(p.x, p.y, q.x, q.y), bias[h]);
            }
        return;
    }
    // Else the ring, idle now, takes the partial tile, from which bands of rows - the whole tile, or of a split reduction
    // this block's share of it, summed over the cluster - are finished and stored row by row: from registers, the 64 copies
    // of bias and activation were more instructions than a short reduction.
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float4* part = reinterpret_cast<float4*>(smem);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 p = unpack2(acc[i][h * 2]), q = unpack2(acc[i][h * 2 + 1]);
            part[(ty + i * TY) * (BN / 4) + h * (BN / 8) + tx] = make_float4(p.x, p.y, q.x, q.y);
        }
    static_assert(NT % (BN / 4) == 0, "a thread stays on its columns");
    const int n = n0 + tid % (BN / 4) * 4, band = BM / splits;
    const float4 bias = row_bias(a, n);
    if (splits == 1) __syncthreads();
    else cluster_sync();
#pragma unroll 2
    for (int i = tid / (BN / 4); i < band; i += NT / (BN / 4)) {
        const int row = rank * band + i;
        const float4* at = part + row * (BN / 4) + tid % (BN / 4);
        float4 sum;
        if (splits == 1) {
            sum = *at;
        } else {
            const uint32_t addr = smem_addr(at);
            sum = load_cluster(addr, 0);
            for (int p = 1; p < splits; ++p) {
                const float4 v = load_cluster(addr, (uint32_t)p);
                sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
        }
        store4(a, m0 + row, n, sum, bias);
    }
    if (splits > 1) cluster_sync();                              // no block leaves while another still reads its partial tile
}

// The same contraction with both operands fetched by the copy engine: 32 reduction elements a stage, of A as 128-byte rows in
// the 128-byte swizzle (im2col copies walk rows and images, so that a tile has as many pixels as suits it), of B as rows of
// 64 columns. A thread computes 4 x 16 outputs and reads A four reduction elements at a time. Sums are taken in the order of
// conv_igemm_kernel. Bound by the FP32 pipe where SMs have several blocks (1.42 us a step of 128 x 64 x 32, 1.3 at its full
// rate); two stages are enough for that, more gave nothing. Launched after its predecessor, not beside it: blocks that
// wait on SMs that happen to have room are then not spread evenly (ResNet-18, 8 images, 882 us; 1068 overlapped).
constexpr int kTmaBN = 64, kTmaTX = 4, kTmaK = 32, kTmaStages = 2;

struct IgemmTile {
    int im2col;                      // 0: the rows of A follow one another
    int chunks, per_tap;             // steps of kTmaK reduction elements: all, and of one filter tap
    uint32_t spin_limit;             // polls of a wait before it gives up
};

template <int TY>
__global__ void __launch_bounds__(kTmaTX * TY, 512 / (kTmaTX * TY))
conv_igemm_tma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const IgemmArgs a,
                      const IgemmTile tl, int* err_flag) {
    constexpr int TM = 4, BM = TY * TM, BN = kTmaBN, NT = kTmaTX * TY;
    constexpr uint32_t kBytesA = BM * 128, kBytesB = kTmaK * BN * 4, kStage = kBytesA + kBytesB;
    extern __shared__ __align__(1024) unsigned char ring[];
    __shared__ __align__(8) uint64_t full[kTmaStages];
    // the tile's first pixel; whether somebody gave up, and the step at which thread 0, which asks for the copies, did (here
    // and not in its registers, which all are short of: eight of them went to the stack)
    __shared__ int s_at[3], s_abort, s_stop;
    const int tid = threadIdx.x, tx = tid % kTmaTX, ty = tid / kTmaTX;
    const long m0 = (long)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN, splits = gridDim.z, rank = blockIdx.z;
    const int first = (int)((long)tl.chunks * rank / splits), count = (int)((long)tl.chunks * (rank + 1) / splits) - first;
    const uint32_t base = smem_addr(ring);
    if (tid == 0) {
        for (int i = 0; i < kTmaStages; ++i) tc::mbar_init(&full[i], 1);
        s_abort = 0;
        s_stop = count;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int ky = 0, kx = 0, cc = 0;                                // thread 0: next step
    if (tid == 0) {
        const long line = m0 / a.Wo, an = line / a.Ho;
        s_at[0] = (int)(m0 - line * a.Wo) * a.stride - a.pad;
        s_at[1] = (int)(line - an * a.Ho) * a.stride - a.pad;
        s_at[2] = (int)an;
        const int tap = first / tl.per_tap;
        cc = first - tap * tl.per_tap;
        ky = tap / a.kernel;
        kx = tap - ky * a.kernel;
    }
    auto issue = [&](int stage) {
        const uint32_t to = base + (uint32_t)stage * kStage;
        tc::mbar_expect_tx(&full[stage], kStage);
        if (tl.im2col) tc::tma_load_im2col(to, &tmA, &full[stage], cc * kTmaK, s_at[0], s_at[1], s_at[2], kx * a.dil, ky * a.dil);
        else tc::tma_load_2d(to, &tmA, &full[stage], cc * kTmaK, (int)m0);
        tc::tma_load_3d(to + kBytesA, &tmB, &full[stage], n0, cc * kTmaK, ky * a.kernel + kx);
        if (++cc == tl.per_tap) { cc = 0; if (++kx == a.kernel) { kx = 0; ++ky; } }
    };
    if (tid == 0)
        for (int i = 0; i < kTmaStages && i < count; ++i) issue(i);
    unsigned long long acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    bool came = true;
    int stage = 0;
    uint32_t phase = 0;
    for (int t = 0; t < count; ++t) {
        if (came && !tc::wait_turn(&full[stage], phase, &s_abort, tl.spin_limit)) {
            came = false;                                      // (a thread that gives up goes on to the barriers all the same)
            s_abort = 1;
            if (tid == 0) s_stop = t;
            tc::record_error(err_flag, 8);
        }
        const float* sa = reinterpret_cast<const float*>(ring + stage * kStage) + ty * 32;
        const float* sb = reinterpret_cast<const float*>(ring + stage * kStage + kBytesA) + tx * 4;
#pragma unroll
        for (int k4 = 0; k4 < kTmaK / 4; ++k4) {
            float4 av[TM];
            const float* row = sa + ((k4 ^ (ty & 7)) << 2);
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(row + i * TY * 32);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unsigned long long b[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sb + (k4 * 4 + k) * BN + j * kTmaTX * 4);
                    b[2 * j] = v.x; b[2 * j + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float u = k == 0 ? av[i].x : (k == 1 ? av[i].y : (k == 2 ? av[i].z : av[i].w));
                    const unsigned long long uu = pack2(u, u);
#pragma unroll
                    for (int j = 0; j < 8; ++j) fma2(acc[i][j], uu, b[j]);
                }
            }
        }
        __syncthreads();                                       // everyone is done with the stage
        if (tid == 0 && came && t + kTmaStages < count) issue(stage);
        if (++stage == kTmaStages) { stage = 0; phase ^= 1u; }
    }
    if (tid == 0)                                              // no copy may land in a block that has retired
        for (int t = s_stop; t < count && t < s_stop + kTmaStages; ++t)
            tc::mbar_wait(&full[t % kTmaStages], (uint32_t)(t / kTmaStages) & 1u);

    if (splits == 1) {
        // 64 bytes of eight rows a store instruction: whole sectors, and no pass through shared memory
        float4 bias[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bias[j] = row_bias(a, n0 + j * 16 + tx * 4);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 p = unpack2(acc[i][j * 2]), q = unpack2(acc[i][j * 2 + 1]);
                store4(a, m0 + ty + i * TY, n0 + j * 16 + tx * 4, make_float4(p.x, p.y, q.x, q.y), bias[j]);
            }
        return;
    }
    float4* part = reinterpret_cast<float4*>(ring);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 p = unpack2(acc[i][j * 2]), q = unpack2(acc[i][j * 2 + 1]);
            part[(ty + i * TY) * (BN / 4) + j * kTmaTX + tx] = make_float4(p.x, p.y, q.x, q.y);
        }
    const int n = n0 + tid % (BN / 4) * 4;
    const float4 bias = row_bias(a, n);
    cluster_sync();
    const int r1 = BM * (rank + 1) / splits;
    for (int row = BM * rank / splits + tid / (BN / 4); row < r1; row += NT / (BN / 4)) {
        const uint32_t addr = smem_addr(part + row * (BN / 4) + tid % (BN / 4));
        float4 v[8];
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < splits) v[p] = load_cluster(addr, (uint32_t)p);
        float4 sum = v[0];
#pragma unroll
        for (int p = 1; p < 8; ++p)
            if (p < splits) { sum.x += v[p].x; sum.y += v[p].y; sum.z += v[p].z; sum.w += v[p].w; }
        store4(a, m0 + row, n, sum, bias);
    }
    cluster_sync();                                            // no block leaves while another still reads its partial tile
}

template <int TY>
int launch_tma(const IgemmArgs& a, const CUtensorMap& mA, const CUtensorMap& mB, const IgemmTile& tl, int splits, cudaStream_t s) {
    constexpr int BM = TY * 4;
    constexpr size_t stage = (size_t)(BM * 128 + kTmaK * kTmaBN * 4);
    constexpr size_t smem = stage * kTmaStages;
    static_assert(smem >= (size_t)BM * kTmaBN * 4, "the partial tile takes the ring's place");
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        cudaError_t e = cudaFuncSetAttribute(conv_igemm_tma_kernel<TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(div_up(a.M, BM), div_up(a.n_store, kTmaBN), splits);
    cfg.blockDim = dim3(kTmaTX * TY);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = splits;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, conv_igemm_tma_kernel<TY>, mA, mB, a, tl, error_flag_ptr());
    if (e != cudaSuccess) { set_last_error(e); (void)cudaGetLastError(); return OGLE_ERR_CUDA; }
    return finish_launch();
}

// How this form would lay a contraction out, and about how long it would take (microseconds, launch included): the busiest
// SM's tiles x steps, 1.42 us a step for every four warps of 128 x 64 outputs - 1.8 for four alone, which do not cover their
// own waits -, and 8.5 to 12.5 us of start, first copies and way out. The parts of the GPU that clusters are placed in hold no whole number
// of larger ones: 128 blocks in clusters of 8 were seen to put two on some SMs, 400 to put four on some. Of 130 layers drawn
// from 3e7 to 2e10 operations all but a dozen that take over 40 us took within 5 % of the estimate.
struct TmaPlan { int ty, splits; double us; };

// least: ranges the reduction has in the other form; with fewer, sums are longer and errors larger (by up to a quarter). At the
// same number the longest may be up to 24 elements longer than there, since a step is 32 elements of one tap.
TmaPlan plan_tma(const IgemmArgs& a, int least) {
    const int chunks = a.kernel * a.kernel * ((a.Cp + kTmaK - 1) / kTmaK);
    TmaPlan best = {0, 1, 1e30};
    static const int kSplits[] = {1, 2, 4, 5, 6, 8};
    for (int ty = 32; ty >= 16; ty -= 16)
        for (int k : kSplits) {
            if (k < least || k > chunks || (k > least && 2 * k > chunks)) continue;
            const long blocks = (a.M + ty * 4 - 1) / (ty * 4) * ((a.n_store + kTmaBN - 1) / kTmaBN) * k;
            const int sms = k <= 2 ? kNumSMs : (k >= 5 && (ty == 32 || blocks <= kNumSMs) ? 120 : (blocks <= kNumSMs ? 132 : 136));
            const long busiest = (blocks + sms - 1) / sms;
            const double load = 1.42 * (double)(ty == 32 ? busiest : (busiest + 1) / 2);    // (a warp to each of four schedulers)
            const int per = (chunks + k - 1) / k;
            const double body = (load < 1.8 ? 1.8 : load) * (per + 0.6 / per);          // (short ranges are mostly start and end)
            const double us = body + 8.5 + (body < 50 ? 0.08 * body : 4.0) + (k > 1 ? 0.5 : 0.0);
            if (us < best.us) best = {ty, k, us};
        }
    return best;
}

// Whether the copy engine's maps can say it: corners of a map with two image extents have eight bits, offsets of a copy as many.
bool tma_can_serve(const IgemmArgs& a) {
    const int far = a.pad - (a.kernel - 1) * a.dil;
    return a.pad <= 127 && far >= -128 && far <= 127 && (a.kernel - 1) * a.dil <= 255 && a.stride <= 8;
}

// OGLE_ERR_UNSUPPORTED: no map of these tensors.
int launch_igemm_tma(const IgemmArgs& a, const TmaPlan& plan, cudaStream_t s) {
    IgemmTile tl = {};
    tl.per_tap = (a.Cp + kTmaK - 1) / kTmaK;
    tl.chunks = a.kernel * a.kernel * tl.per_tap;
    tl.im2col = a.kernel == 1 && a.stride == 1 && a.pad == 0 ? 0 : 1;
    tl.spin_limit = tc::role_wait_limit();
    const int BM = plan.ty * 4;
    CUtensorMap mA, mB;
    if (!tl.im2col) {
        const cuuint64_t dims[2] = {(cuuint64_t)a.Cp, (cuuint64_t)a.M};
        const cuuint64_t str[1] = {(cuuint64_t)a.Cs * 4};
        const cuuint32_t box[2] = {kTmaK, (cuuint32_t)BM}, es[2] = {1, 1};
        if (!make_map(&mA, a.x, 2, dims, str, box, es)) return OGLE_ERR_UNSUPPORTED;
    } else {
        const int far = a.pad - (a.kernel - 1) * a.dil;
        const cuuint64_t row = (cuuint64_t)a.Cs * 4 * a.W;
        const cuuint64_t dims[4] = {(cuuint64_t)a.Cp, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)(a.M / ((long)a.Ho * a.Wo))};
        const cuuint64_t str[3] = {(cuuint64_t)a.Cs * 4, row, row * a.H};
        const int lower[2] = {-a.pad, -a.pad}, upper[2] = {far, far};
        if (!make_map_im2col(&mA, a.x, dims, str, lower, upper, kTmaK, BM, a.stride)) return OGLE_ERR_UNSUPPORTED;
    }
    const cuuint64_t dims[3] = {(cuuint64_t)a.n_b, (cuuint64_t)a.Cp, (cuuint64_t)(a.kernel * a.kernel)};
    const cuuint64_t str[2] = {(cuuint64_t)a.ldb * 4, (cuuint64_t)a.ldb * 4 * a.Cp};
    const cuuint32_t box[3] = {kTmaBN, kTmaK, 1}, es[3] = {1, 1, 1};
    if (!make_map_sw(CU_TENSOR_MAP_SWIZZLE_NONE, &mB, a.w, 3, dims, str, box, es)) return OGLE_ERR_UNSUPPORTED;
    return plan.ty == 32 ? launch_tma<32>(a, mA, mB, tl, plan.splits, s) : launch_tma<16>(a, mA, mB, tl, plan.splits, s);
}

template <int BM, int BN, int TM, bool TRANSB, typename Pixel = unsigned>
int launch(const IgemmArgs& a, int splits, cudaStream_t s) {
    if (!a.y) return OGLE_OK;                        // (asked for the kernel's name only)
    constexpr size_t ring = (size_t)kStages * (BM * kALd + kBK * BN) * sizeof(float);
    constexpr size_t tile = (size_t)BM * BN * sizeof(float);
    constexpr size_t smem = tile > ring ? tile : ring;
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        cudaError_t e = cudaFuncSetAttribute(conv_igemm_kernel<BM, BN, TM, TRANSB, Pixel>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(div_up(a.M, BM), div_up(a.n_store, BN), splits);
    cfg.blockDim = dim3(BM * BN / (8 * TM));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = splits;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, conv_igemm_kernel<BM, BN, TM, TRANSB, Pixel>, a);
    if (e != cudaSuccess) { set_last_error(e); (void)cudaGetLastError(); return OGLE_ERR_CUDA; }
    return finish_launch();
}

}  // namespace

// Tile and split. Reductions of up to 64 elements are bound by their instructions before and after the multiplies and take
// the 2 x 8 form; up to 128 it pays where it gives an SM one to three tiles (fewer are better split, 126 x 116 x 24 4.5 us
// against 9.0; more make better large tiles, 52288 x 108 x 508 177 against 214). The large tiles read the least through L2
// per multiply-add and are taken where they alone give every SM its two (128 x 128) or four (128 x 64) resident blocks,
// the larger only where the SM with the most of them ends no later (1419 x 557 x 3436: 324 of them, two on most SMs and
// three on some, 190 us, 153 in halves); 128 x 32 serves narrow outputs over many rows. Everything else runs on 64 x 64
// tiles, 64 x 32 for narrow outputs, with the reduction split so that the SMs fill: the cost of a split is (blocks on the
// busiest SM, at least the four that keep its FP32 pipes busy) x (steps of a block, plus about six for its start, its
// partial tile and the cluster's barriers).
int launch_igemm(const IgemmArgs& a, bool trans_b, cudaStream_t s, const char** name) {
    if (name) *name = "conv_igemm_kernel";
    const long m128 = (a.M + 127) / 128, m64 = (a.M + 63) / 64;
    if (m64 > 0x7fffffffL || (a.n_store + 63) / 64 > 65535) return OGLE_ERR_UNSUPPORTED;
    const bool large = a.M > 0x7fffffffL || a.M / ((long)a.Ho * a.Wo) * a.H * a.W > 0x7fffffffL;
    const long tiles64 = m64 * ((a.n_store + 63) / 64);
    if (!large && (a.R <= 64 || (a.R <= 128 && tiles64 >= kNumSMs && tiles64 <= 3 * kNumSMs))) {
        if (trans_b) return launch<64, 64, 2, true>(a, 1, s);
        return a.n_store <= 32 ? launch<64, 32, 2, false>(a, 1, s) : launch<64, 64, 2, false>(a, 1, s);
    }
    // The copy engine's form, where it is the faster by what both were measured to take (below): 3x3 256 -> 256 at 38 x 38
    // x 32 images 1169 -> 1003 us, 5776 x 512 x 512 pointwise 87 -> 71, ResNet's 3x3 layers at 8 images 54 -> 50. It wants
    // steps that are mostly full and half of its 64 columns.
    auto by_copy_engine = [&](double us, int least) {
        if (large || trans_b || a.n_store <= 32 || a.Cp < 28 || !tma_can_serve(a)) return (int)OGLE_ERR_UNSUPPORTED;
        const TmaPlan plan = plan_tma(a, least);
        if (plan.us >= us) return (int)OGLE_ERR_UNSUPPORTED;
        if (name) { *name = "conv_igemm_tma_kernel"; return (int)OGLE_OK; }
        return launch_igemm_tma(a, plan, s);
    };
    const int steps = (a.R + kBK - 1) / kBK;
    if (!large) {
        const long wide = m128 * ((a.n_store + 127) / 128), half = m128 * ((a.n_store + 63) / 64);
        const long wide_sm = (wide + kNumSMs - 1) / kNumSMs, half_sm = (half + kNumSMs - 1) / kNumSMs;
        // (the SM with the most tiles sets the time)
        if (a.n_store > 64 && wide >= 2 * kNumSMs && 2 * wide_sm <= half_sm) {
            const int rc = by_copy_engine(1.7 * (double)wide_sm * steps + 8.0, 1);
            if (rc != OGLE_ERR_UNSUPPORTED) return rc;
            return trans_b ? launch<128, 128, 8, true>(a, 1, s) : launch<128, 128, 8, false>(a, 1, s);
        }
        if (a.n_store > 32 && half >= 4 * kNumSMs) {
            const int rc = by_copy_engine(0.86 * (double)half_sm * steps + 8.0, 1);
            if (rc != OGLE_ERR_UNSUPPORTED) return rc;
            return trans_b ? launch<128, 64, 8, true>(a, 1, s) : launch<128, 64, 8, false>(a, 1, s);
        }
        if (a.n_store <= 32 && m128 >= 4 * kNumSMs && !trans_b) return launch<128, 32, 8, false>(a, 1, s);
    }
    const bool narrow = a.n_store <= 32 && !trans_b && !large;
    const long tiles = narrow ? m64 : tiles64;
    int best = 1;
    double best_cost = -1.0, us = 0.0;
    for (int k = 1; k <= 8 && k <= steps; k *= 2) {
        const double blocks = (double)((tiles * k + kNumSMs - 1) / kNumSMs);
        const double cost = (blocks < 4 ? 4.0 : blocks) * ((steps + k - 1) / k + 6.0);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = k;
            // (Two or three blocks an SM come out ahead of what they are counted as above, and so do five and a part, of which the
            // last two run beside each other alone: 3 images of 40 x 28, 3x3 87 -> 220, 5.7 blocks, 40.1 us where six take
            // 46.7, and the other form 43.8. Five images of 61 x 23, 3x3 315 -> 92, 5.95 blocks, 155 and 117.)
            const double exact = (double)(tiles * k) / kNumSMs;
            us = 0.41 * (blocks < 2.7 ? 2.55 : (exact > 5.0 && exact < 5.75 ? exact + 0.1 : blocks)) * ((steps + k - 1) / k + 6.0);
        }
    }
    const int rc = by_copy_engine(us, best);
    if (rc != OGLE_ERR_UNSUPPORTED) return rc;
    if (large) return launch<64, 64, 8, false, long>(a, best, s);
    if (narrow) return launch<64, 32, 4, false>(a, best, s);
    return trans_b ? launch<64, 64, 8, true>(a, best, s) : launch<64, 64, 8, false>(a, best, s);
}

}  // namespace ogle
