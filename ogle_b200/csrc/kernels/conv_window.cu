// Convolutions of 5 x 5 and 7 x 7 filters over images of at most four channels (an RGB stem: 16-byte pixels) into at most 64
// channels, on the tensor cores, with the input window itself as the operand: nothing is gathered.
//
// A pixel is half of a K = 8 step of TF32 (four values), and - as [bf16 high x 4 | bf16 low x 4] - half of a K = 16 step of the
// BF16 pass that adds the cross terms of the split mode. Without swizzle an operand is made of pieces of eight rows x 16
// bytes, and two byte distances say where the next piece along the reduction and the next eight rows are. With a tile of 8 x 16 output
// pixels eight rows are eight neighbouring pixels of one row of the window (of every second one at stride 2: the window is
// kept as two planes, even and odd columns), the next eight rows lie one output row further down, and the next piece is the
// next tap: any pair of taps at a constant distance is one step. (At stride 1 a tile may be 128 x 1 pixels, for flat maps.) Taps pair up along the filter row; the last column's pair
// up downwards, and since their number is odd too the last but one is in two pairs with half its filter value in each: a
// zero in the filter instead would multiply a pixel outside the window, which may be infinite.
//
// The form that gathers rows of 147 values (conv_tc2.cu) is bound by building them, 12 copies of every value with a split
// each: 128 images of 224 x 224, 7 x 7 / 2, 3 -> 64 channels take 257 us, 279 in one pass. Here a value is split once a tile:
// 226 us, 135 in one pass (HBM 78). What bounds it is the multiplies: one of 128 pixels x 64 channels x 32 bytes takes 88
// cycles (75 for 16 channels: it is the reads of the window's pieces), wherever the pieces begin - at multiples of 128 bytes it
// would be 214 and 130 us -, 50 a tile, 25 in one pass.
//
// Warps: copies, multiplies, four that split the window, two groups of four that finish and store 32 channels of the tile each
// (one group: 279 us in split mode, 164 in one pass).
#include "tc_common.cuh"
#include "tma_host.h"

namespace ogle {

namespace {

using namespace tc;

constexpr int kThreadsW = 448;
constexpr int kAccCols = 64;                       // tensor-memory columns of an accumulator (two of them)
constexpr int kSlabBytes = 128 * 128;              // 128 pixels x 32 channels

// Geometry of a tile's window and of the pairs of taps.
template <int kK, int kS, int kTileW>
struct Window {
    static constexpr int kTileH = 128 / kTileW;
    static constexpr int kW = (kTileW - 1) * kS + kK, kH = (kTileH - 1) * kS + kK;
    static constexpr int kPlaneW = (kW + kS - 1) / kS;              // columns of a plane (stride 2: even and odd ones apart)
    static constexpr int kPairs = kK / 2, kSteps = kK * kPairs + kPairs + 1;
    static constexpr uint32_t kPlane = kPlaneW * kH * 16, kOperand = (kPlane * kS + 127u) & ~127u, kRaw = (kW * kH * 16 + 127u) & ~127u;
};

struct WindowArgs {
    int Ho, Wo, K, Kp, C, pad;
    int tiles_w, tiles_h, total;
    int np;                      // columns of the multiply
    uint32_t filters;            // bytes of one pass's filters
    int has_bias, act;
    float lo, hi;
    int passes;
    const float* res;
    int res_ld;
    uint32_t spin_limit;
};

// K-major operand of pieces of 8 rows x 16 bytes: `lead` bytes to the next piece along the reduction, `next8` to the next eight rows.
__device__ __forceinline__ uint64_t plain_desc(uint32_t lead, uint32_t next8) {
    return (uint64_t)(lead >> 4) << 16 | (uint64_t)(next8 >> 4) << 32 | (uint64_t)1 << 46;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// kK x kK filters, stride kS: every operand's place is known when this is compiled (worked out step by step: 285 us).
template <int kK, int kS, int kTileW>
__global__ void __launch_bounds__(kThreadsW, 1)
conv_window_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const float* __restrict__ w, const float* __restrict__ bias, const WindowArgs a, int* err_flag) {
    using W = Window<kK, kS, kTileW>;
    constexpr int kPairs = W::kPairs, kSteps = W::kSteps, kTileH = W::kTileH;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t bar_raw_full[2], bar_raw_empty[2], bar_op_full[2], bar_op_empty[2], bar_acc_full[2], bar_acc_empty[2],
        bar_filters, bar_drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    __shared__ float s_bias[kAccCols];
    unsigned char* base_ptr = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    const uint32_t base = smem_u32(base_ptr);
    const int sections = a.passes == 3 ? 2 : 1;                   // operands of a pass each
    const uint32_t off_filters = 2 * kSlabBytes, off_op = off_filters + (uint32_t)sections * a.filters,
                   off_raw = off_op + 2u * (uint32_t)sections * W::kOperand;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_flag = &s_abort;

    grid_dependency_trigger();
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_raw_full[i], 1);
            mbar_init(&bar_raw_empty[i], 128);
            mbar_init(&bar_op_full[i], 128);
            mbar_init(&bar_op_empty[i], 1);
            mbar_init(&bar_acc_full[i], 1);
            mbar_init(&bar_acc_empty[i], a.K > 32 ? 256 : 128);
        }
        mbar_init(&bar_filters, 384);
        mbar_init(&bar_drain, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(2u * kAccCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = tmem_slot;
    grid_dependency_wait();         // nothing from global memory before this point

    if (warp >= 2) {
        // Filters: step m's two taps of channel n are 16 bytes each, at [m][tap][n].
        const int t = threadIdx.x - 64;
        constexpr int kPieces = (2 * kSteps * kAccCols + 383) / 384;
        float v[kPieces][4];
        int to[kPieces];
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {              // (all loads in flight at once)
            const int i = t + j * 384, n = i % kAccCols, m = i / kAccCols >> 1, second = i / kAccCols & 1;
            const bool down = m >= kK * kPairs;
            const int e = m - kK * kPairs, row = down ? (e < kPairs ? 2 * e : kK - 2) + second : m / kPairs,
                      col = down ? kK - 1 : m % kPairs * 2 + second;
            const float scale = down && row == kK - 2 ? 0.5f : 1.f;
            to[j] = m < kSteps && n < a.np ? ((m * 2 + second) * a.np + n) * 16 : -1;
#pragma unroll
            for (int c = 0; c < 4; ++c) v[j][c] = m < kSteps && n < a.K && c < a.C ? scale * w[((row * kK + col) * 4 + c) * a.Kp + n] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
            if (to[j] < 0) continue;
            float h[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) h[c] = __uint_as_float(__float_as_uint(v[j][c]) & 0xffffe000u);
            unsigned char* dst = base_ptr + off_filters + to[j];
            *reinterpret_cast<float4*>(dst) = make_float4(h[0], h[1], h[2], h[3]);
            if (sections == 2)
                *reinterpret_cast<uint4*>(dst + a.filters) =
                    make_uint4(bf16_pair(v[j][0] - h[0], v[j][1] - h[1]), bf16_pair(v[j][2] - h[2], v[j][3] - h[3]), bf16_pair(v[j][0], v[j][1]),
                               bf16_pair(v[j][2], v[j][3]));
        }
        if (t >= 128 && t - 128 < kAccCols) s_bias[t - 128] = a.has_bias && t - 128 < a.K ? bias[t - 128] : 0.f;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(&bar_filters);
    }

    if (warp == 0) {
        // ------------------------------------------------------------ copies
        if (elect_one()) {
            int issued = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < a.total; tile += gridDim.x) {
                const int s = issued & 1;
                if (issued >= 2) ok = wait_turn(&bar_raw_empty[s], (uint32_t)((issued >> 1) - 1) & 1u, abort_flag, a.spin_limit);
                if (!ok) { record_error(err_flag, 1); s_abort = 1; break; }
                const int q = tile / a.tiles_w, tx = tile - q * a.tiles_w, n = q / a.tiles_h, ty = q - n * a.tiles_h;
                mbar_expect_tx(&bar_raw_full[s], (uint32_t)(W::kW * W::kH * 16));
                const int x = tx * kTileW * kS - a.pad, y = ty * kTileH * kS - a.pad;
                const uint32_t to = base + off_raw + (uint32_t)s * W::kRaw;
                if (W::kW <= 128) tma_load_4d(to, &tmX, &bar_raw_full[s], 2 * x, y, n, 0);
                else tma_load_4d(to, &tmX, &bar_raw_full[s], 0, x, y, n);
                ++issued;
            }
            // what is in flight lands before the block ends: others may have given up on it after the last was asked for
            for (int i = issued < 2 ? 0 : issued - 2; i < issued; ++i) (void)mbar_wait(&bar_raw_full[i & 1], (uint32_t)(i >> 1) & 1u);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ multiplies
        if (elect_one()) {
            const uint32_t shape = ((uint32_t)(a.np >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24) | (1u << 4);
            const uint32_t idesc = shape | (2u << 7) | (2u << 10), idesc_bf16 = shape | (1u << 7) | (1u << 10);
            // (eight rows on: a row of the tile, or eight pixels of a tile one row high)
            constexpr uint32_t kNext8 = kTileW == 8 ? kS * W::kPlaneW * 16 : 128, kPair = kS == 2 ? 1 : 2;              // (a pair of taps on: in 16 bytes)
            const uint64_t along = plain_desc(kS == 2 ? W::kPlane : 16u, kNext8), down = plain_desc(W::kPlaneW * 16u, kNext8);
            const uint64_t bdesc = plain_desc((uint32_t)a.np * 16u, 128u) + ((base + off_filters) >> 4);
            bool ok = wait_turn(&bar_filters, 0, abort_flag, a.spin_limit);
            int it = 0;
            for (int tile = blockIdx.x; tile < a.total && ok; tile += gridDim.x, ++it) {
                const int s = it & 1;
                const uint32_t use = (uint32_t)(it >> 1);
                ok = (it < 2 || wait_turn(&bar_acc_empty[s], (use - 1) & 1u, abort_flag, a.spin_limit)) &&
                     wait_turn(&bar_op_full[s], use & 1u, abort_flag, a.spin_limit);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem_d + (uint32_t)(s * kAccCols);
                uint32_t any = 0;
                // the small terms first
                for (int pass = sections - 1; pass >= 0; --pass) {
                    const uint32_t op = (base + off_op + (uint32_t)(s * sections + pass) * W::kOperand) >> 4;
                    uint64_t b = bdesc + ((uint32_t)pass * a.filters >> 4);
                    auto multiply = [&](uint64_t ad) {
                        if (pass) umma_bf16(d, ad, b, idesc_bf16, any);
                        else umma_tf32(d, ad, b, idesc, any);
                        any = 1;
                        b += (uint32_t)a.np * 2u;
                    };
#pragma unroll
                    for (int m = 0; m < kK * kPairs; ++m) multiply(along + op + (uint32_t)(m / kPairs * W::kPlaneW + m % kPairs * kPair));
#pragma unroll
                    for (int e = 0; e <= kPairs; ++e)
                        multiply(down + op + (uint32_t)((e < kPairs ? 2 * e : kK - 2) * W::kPlaneW + (kS == 2 ? kPairs : kK - 1)));
                }
                umma_commit(&bar_op_empty[s]);
                umma_commit(&bar_acc_full[s]);
            }
            if (!ok) { record_error(err_flag, 2); s_abort = 1; }
            umma_commit(&bar_drain);
            (void)mbar_wait(&bar_drain, 0);
        }
    } else if (warp < 6) {
        // ------------------------------------------------------------ operands: the window as planes, and its split
        const int t = threadIdx.x - 64;
        constexpr int kPixels = W::kW * W::kH, kMine = (kPixels + 127) / 128;
        uint32_t to[kMine];                            // where this thread's pixels go, the same in every tile
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
            const int i = t + j * 128, y = i / W::kW, x = i % W::kW;
            to[j] = (uint32_t)(x % kS) * W::kPlane + (uint32_t)(y * W::kPlaneW + x / kS) * 16u;
        }
        int it = 0;
        for (int tile = blockIdx.x; tile < a.total; tile += gridDim.x, ++it) {
            const int s = it & 1;
            const uint32_t use = (uint32_t)(it >> 1);
            const bool ok = wait_turn(&bar_raw_full[s], use & 1u, abort_flag, a.spin_limit) &&
                            (it < 2 || wait_turn(&bar_op_empty[s], (use - 1) & 1u, abort_flag, a.spin_limit));
            if (!ok) { record_error(err_flag, 3); s_abort = 1; break; }
            const float4* raw = reinterpret_cast<const float4*>(base_ptr + off_raw + (size_t)s * W::kRaw);
            unsigned char* op = base_ptr + off_op + (size_t)(s * sections) * W::kOperand;
#pragma unroll
            for (int j = 0; j < kMine; ++j) {
                if (t + j * 128 >= kPixels) continue;
                float4 v = raw[t + j * 128];
                if (a.C < 4) v.w = 0.f;                // whatever the lanes behind the channels hold
                if (a.C < 3) v.z = 0.f;
                if (a.C < 2) v.y = 0.f;
                *reinterpret_cast<float4*>(op + to[j]) = v;
                if (a.passes == 3) {
                    float h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) h[c] = __uint_as_float(__float_as_uint(h[c]) & 0xffffe000u);
                    *reinterpret_cast<uint4*>(op + W::kOperand + to[j]) =
                        make_uint4(bf16_pair(h[0], h[1]), bf16_pair(h[2], h[3]), bf16_pair(v.x - h[0], v.y - h[1]), bf16_pair(v.z - h[2], v.w - h[3]));
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(&bar_op_full[s]);
            mbar_arrive(&bar_raw_empty[s]);
        }
    } else {
        // ------------------------------------------------------------ finish and store
        const int eg = (warp - 6) >> 2, t = (threadIdx.x - 192) & 127, q = warp & 3, row = q * 32 + lane, slabs = a.K > 32 ? 2 : 1;
        auto all = [&](bool mine) {                    // (also the barrier in front of what the others read)
            uint32_t r;
            mine = __all_sync(0xffffffffu, mine);
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "=r"(r) : "r"((uint32_t)mine), "r"(1 + eg) : "memory");
            return r != 0;
        };
        const float lo = a.act == OGLE_ACT_CLIP ? a.lo : 0.f, hi = a.act == OGLE_ACT_CLIP ? a.hi : INFINITY;
        bool ok = all(wait_turn(&bar_filters, 0, abort_flag, a.spin_limit));         // the bias
        if (!ok) { record_error(err_flag, 4); s_abort = 1; }
        // two slabs a tile: one each; one: every other tile
        int it = slabs > 1 ? 0 : eg;
        const int by = slabs > 1 ? 1 : 2, g = slabs > 1 ? eg : 0;
        const bool full = g * 32 + 32 <= a.K;
        unsigned char* slab = base_ptr + (size_t)eg * kSlabBytes;
        float4* dst = reinterpret_cast<float4*>(slab + (size_t)row * 128);
        for (int tile = blockIdx.x + it * (int)gridDim.x; tile < a.total && ok; tile += by * (int)gridDim.x, it += by) {
            const int s = it & 1;
            const int tq = tile / a.tiles_w, tx = tile - tq * a.tiles_w, n = tq / a.tiles_h, ty = tq - n * a.tiles_h;
            ok = all(wait_turn(&bar_acc_full[s], (uint32_t)(it >> 1) & 1u, abort_flag, a.spin_limit));
            if (!ok) { record_error(err_flag, 4); s_abort = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int oy = ty * kTileH + row / kTileW, ox = tx * kTileW + row % kTileW;
            const float* res = a.res && oy < a.Ho && ox < a.Wo ? a.res + (((long)n * a.Ho + oy) * a.Wo + ox) * a.res_ld : nullptr;
            uint32_t r[32];
            const uint32_t taddr = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * kAccCols + g * 32);
#pragma unroll
            for (int half = 0; half < 2; ++half)
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                    : "=r"(r[half * 16]), "=r"(r[half * 16 + 1]), "=r"(r[half * 16 + 2]), "=r"(r[half * 16 + 3]), "=r"(r[half * 16 + 4]),
                      "=r"(r[half * 16 + 5]), "=r"(r[half * 16 + 6]), "=r"(r[half * 16 + 7]), "=r"(r[half * 16 + 8]), "=r"(r[half * 16 + 9]),
                      "=r"(r[half * 16 + 10]), "=r"(r[half * 16 + 11]), "=r"(r[half * 16 + 12]), "=r"(r[half * 16 + 13]),
                      "=r"(r[half * 16 + 14]), "=r"(r[half * 16 + 15])
                    : "r"(taddr + (uint32_t)(half * 16)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&bar_acc_empty[s]);
            float v[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) v[c] = __uint_as_float(r[c]) + s_bias[g * 32 + c];
            if (res) {
#pragma unroll
                for (int c4 = 0; c4 < 8; ++c4) {
                    if (g * 32 + c4 * 4 >= a.Kp) continue;
                    const float4 x = *reinterpret_cast<const float4*>(res + g * 32 + c4 * 4);
                    v[c4 * 4] += x.x; v[c4 * 4 + 1] += x.y; v[c4 * 4 + 2] += x.z; v[c4 * 4 + 3] += x.w;
                }
            }
            if (a.act != OGLE_ACT_NONE) {              // (rectified: clipped to [0, inf))
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] = fminf(fmaxf(v[c], lo), hi);
            }
            if (!full) {
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    if (g * 32 + c >= a.K) v[c] = 0.f;                   // padded lanes stay zero
            }
            // the slab is free once the store from it has been read
            if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            asm volatile("bar.sync %0, 128;" ::"r"(1 + eg) : "memory");
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4)             // 128-byte swizzle
                dst[c4 ^ (row & 7)] = make_float4(v[c4 * 4], v[c4 * 4 + 1], v[c4 * 4 + 2], v[c4 * 4 + 3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync %0, 128;" ::"r"(1 + eg) : "memory");
            if (t == 0) {
                asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                             ::"l"(&tmY), "r"(smem_u32(slab)), "r"(g * 32), "r"(tx * kTileW), "r"(ty * kTileH), "r"(n) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(2u * kAccCols));
}

bool make_map_wide_pixels(CUtensorMap* m, const float* x, const ConvArgs& a, int cols, int rows) {
    const cuuint64_t dims[4] = {4, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.N};
    const cuuint64_t str[3] = {16, (cuuint64_t)a.W * 16, (cuuint64_t)a.W * 16 * a.H};
    const cuuint32_t box[4] = {4, (cuuint32_t)cols, (cuuint32_t)rows, 1}, es[4] = {1, 1, 1, 1};
    return make_map_sw(CU_TENSOR_MAP_SWIZZLE_NONE, m, x, 4, dims, str, box, es);
}

template <int kK, int kS, int kTileW>
int launch(const ConvArgs& a, int passes, const float* x, const float* w, const float* bias, float* y, const float* residual, int res_ld,
           cudaStream_t s) {
    using W = Window<kK, kS, kTileW>;
    constexpr int kTileH = W::kTileH;
    WindowArgs t = {};
    t.Ho = a.Ho; t.Wo = a.Wo; t.K = a.K; t.Kp = a.Kp; t.C = a.C; t.pad = a.pad;
    t.tiles_w = (a.Wo + kTileW - 1) / kTileW;
    t.tiles_h = (a.Ho + kTileH - 1) / kTileH;
    const long total = (long)t.tiles_w * t.tiles_h * a.N;
    if (total > 0x7fffffffL - 2 * kNumSMs || a.K > kAccCols || a.Cp != 4) return OGLE_ERR_UNSUPPORTED;      // (tile + 2 grids stays below 2^31)
    t.total = (int)total;
    t.np = (a.K + 15) / 16 * 16;
    t.filters = (uint32_t)(W::kSteps * t.np * 32);
    t.has_bias = a.has_bias; t.act = a.act; t.lo = a.lo; t.hi = a.hi;
    t.passes = passes;
    t.res = residual; t.res_ld = res_ld;
    t.spin_limit = role_wait_limit();
    CUtensorMap mX, mY;
    const cuuint32_t es[4] = {1, 1, 1, 1}, yb[4] = {kChunk, kTileW, kTileH, 1};
    const cuuint64_t yd[4] = {(cuuint64_t)a.Kp, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)a.N};
    const cuuint64_t ys[3] = {(cuuint64_t)a.Ks * 4, (cuuint64_t)a.Ks * 4 * a.Wo, (cuuint64_t)a.Ks * 4 * a.Wo * a.Ho};
    if (W::kW <= 128 ? !make_map_pixels(&mX, x, a.W, a.H, a.N, W::kW, W::kH) : !make_map_wide_pixels(&mX, x, a, W::kW, W::kH)) return OGLE_ERR_CUDA;
    if (!make_map(&mY, y + a.koff, 4, yd, ys, yb, es)) return OGLE_ERR_CUDA;
    const uint32_t sections = passes == 3 ? 2 : 1;
    const size_t smem = 1024 + 2 * kSlabBytes + sections * t.filters + 2 * sections * W::kOperand + 2 * W::kRaw;
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        const cudaError_t e = cudaFuncSetAttribute(conv_window_kernel<kK, kS, kTileW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
        if (e != cudaSuccess) { set_last_error(e); (void)cudaGetLastError(); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    const int blocks = t.total < kNumSMs ? t.total : kNumSMs;
    const bool overlapped = overlapped_launches_enabled();
    note_contraction(9, 1, t.np, overlapped);
    launch_overlapped_if(overlapped, conv_window_kernel<kK, kS, kTileW>, dim3((unsigned)blocks), dim3(kThreadsW), smem, s, mX, mY, w, bias, t,
                         error_flag_ptr());
    return finish_launch();
}

}  // namespace

// x: dense 16-byte pixels; w: tap-major filters; row_tiles: tiles of 128 x 1 pixels (stride 1), else of 8 x 16.
int launch_conv_window(const ConvArgs& a, int passes, bool row_tiles, const float* x, const float* w, const float* bias, float* y,
                       const float* residual, int res_ld, cudaStream_t s) {
    auto with = [&](auto run) { return run(a, passes, x, w, bias, y, residual, res_ld, s); };
    if (a.kernel == 7) return a.stride == 2 ? with(launch<7, 2, 8>) : row_tiles ? with(launch<7, 1, 128>) : with(launch<7, 1, 8>);
    if (a.kernel == 5) return a.stride == 2 ? with(launch<5, 2, 8>) : row_tiles ? with(launch<5, 1, 128>) : with(launch<5, 1, 8>);
    return OGLE_ERR_UNSUPPORTED;
}

}  // namespace ogle
