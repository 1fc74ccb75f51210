// Device helpers shared by the tcgen05 kernels: mbarrier, TMA, UMMA descriptors.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "conv_args.cuh"

namespace ogle {

namespace tc {

constexpr int kTileM = 128;
constexpr int kChunk = 32;              // reduction elements per pipeline stage (128 bytes)
constexpr int kABytes = kTileM * 128;   // one A tile
constexpr int kTapsPixels = kTileM - 2; // output pixels of a tile whose taps lie side by side: their neighbours are rows of it too
constexpr uint32_t kSpinLimit = 1u << 22;

constexpr int kMaxGatherK = 224;     // reduction indices of the gather form (k * k * C rounded up to 32); offsets fit 16 bits

struct TcArgs {
    int flat;                 // 1: rows are a flat range of pixels (pointwise / gemm)
    int tn, th, tw;           // output pixels per tile along n, h, w (tn*th*tw <= 128)
    int tiles_w, tiles_h;     // tile grid along w and h (n follows)
    int N, Ho, Wo;            // output extent (flat: rows = Wo)
    int stride, pad, dil, kernel;
    // 1 (3x3 windows of stride 1 and padding 1; flat): the taps of a filter row side by side along the multiply's column side
    // (kTaps form of conv_tc2.cu). A tile is kTapsPixels consecutive output pixels, which run on over rows and images of
    // oH x oW - an im2col map fetches them -, and BN counts its output channels, of which the accumulator has three sets.
    int taps, oH, oW;
    int chunks_per_tap, Cp32;
    int K, Kp, Ks, koff;      // output channels, padded to 4, row stride, first channel
    int BN, n_tiles;          // N tile and how many cover Kp
    int act;
    float lo, hi;
    float alpha, beta;
    int bias_mode;            // 0 none, 1 full matrix C[m][ldc], 2 per-column vector
    int ldc;
    int passes;               // 1 (TF32) or 3 (split mode: a TF32 pass + a BF16 pass of the cross terms)
    int stages;
    int ta;                   // split mode: 1 = A operands in tensor memory (64 columns per stage, after the accumulators), 2 = the BF16 one (32)
    int tmem_cols;
    int n_acc;                // accumulator buffers in tensor memory (2 or 4)
    int total_tiles;          // m_tiles * n_tiles (persistent kernel)
    int epi_groups, xf_groups; // persistent kernel: warp groups per role (1 or 2)
    int epi_share;            // one-SM form: the epilogue groups take alternate slabs of every tile (else alternate tiles)
    int epi_slabs;            // staging slabs (128 rows x 32 columns) per epilogue group (1 or 2)
    // Two outputs from one pass (sibling convolutions over the same input, filters stacked):
    // columns [0, K1) go to the first tensor, columns [split_col, K) to the second.
    // split_col is a multiple of 32 (0 = single output).
    int split_col, K1;
    // Split reduction: each tile is computed by split_k work items over consecutive ranges of
    // chunks_per_split reduction chunks; their partial tiles are combined by TMA reduce-add
    // stores into an output the host zeroed. Used (activation none only) when the tiles alone
    // would leave most SMs idle or a last round mostly empty. total_work = total_tiles * split_k.
    int split_k, chunks_per_split, total_work;
    // Split reduction through a workspace (ws_mode = 1; any number of ranges, any activation): work item
    // (tile, ks) stores its raw partial tile - no bias, no activation - into slice ks of a scratch tensor
    // of ws_cols columns through the first output map (which then describes the scratch tensor: slices
    // follow one another along its outermost extent, ws_slice rows (flat form) or images apart), and
    // a second, small kernel adds the slices in a fixed order, then bias and activation. Results do not
    // depend on which block finishes first.
    int ws_mode, ws_cols, ws_slice;
    // Split reduction inside a cluster (cluster = 1): the split_k <= 8 blocks of a cluster hold one tile's ranges, leave
    // their partial tiles in shared memory and each adds up and stores a band of the tile's rows: one launch, no
    // scratch, any activation, a residual operand. Stores go straight to y (first channel; y_ld floats a pixel) and,
    // with two outputs, y2.
    int cluster;
    float *y, *y2;
    int y_ld, y2_ld;
    // Gather form (k x k convolution over at most four input channels, e.g. an RGB stem): the
    // activation "tile" that TMA delivers is the tile's input window of 16-byte pixels
    // (g_iw x g_ih of them, halo included), once per reduction chunk; the operand-split warps
    // build the 128 x 32 operand of the chunk from it, row r = window values of output pixel r
    // at reduction indices k = (ky * g_k + kx) * g_C + c, zero padded to a multiple of 32
    // (chunks_per_tap chunks; kernel = 1 in this form). g_C = input channels, g_k = filter
    // size, g_bytes = window bytes rounded up to 1 KB (its slot at the end of every stage). The map of windows more than 128
    // pixels wide has pixels as an extent of their own, that of narrower ones rows of them.
    int gather, g_iw, g_ih, g_C, g_bytes, g_k;
    // Residual operand (one-SM form, reduction unsplit or split inside a cluster): res[pixel * res_ld + channel] is added to the
    // convolution's value (after the bias, before the activation) - a residual block's Add and activation in
    // the convolution's own pass. Null = none.
    const float* res;
    int res_ld;
    int overlapped;           // this launch may start its set-up while the launch before it - the library's own - still runs
    uint32_t spin_limit;      // polls a role waits for its turn before it gives up (kSpinLimit by default)
};

// Polls of the role waits for the launches that follow (see ogle_cuda_set_wait_limit).
uint32_t role_wait_limit();

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase with the given parity. false = gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// Wait for a role's turn: gives up after `limit` polls, or once another role has.
__device__ __forceinline__ bool wait_turn(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t limit) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t spin = 0; spin < limit; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
        if ((spin & 255u) == 255u && *abort_flag) return false;
    }
    return false;
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// 128 pixels of an im2col map from input pixel (c1, c2, c3) on, each moved by the filter tap (ox, oy).
__device__ __forceinline__ void tma_load_im2col(uint32_t dst, const CUtensorMap* map, uint64_t* bar,
                                                int c0, int c1, int c2, int c3, int ox, int oy) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
        ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "h"((unsigned short)ox), "h"((unsigned short)oy)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}

// K-major operand tile, 128-byte rows, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);   // start address, bits [0,14)
    d |= (uint64_t)1 << 16;                              // leading byte offset (unused with swizzle), bits [16,30)
    d |= (uint64_t)(1024 >> 4) << 32;                    // stride byte offset, bits [32,46)
    d |= (uint64_t)1 << 46;                              // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                              // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// One reduction chunk (32 elements = four K=8 steps) issued from a single asm block.
// A lone thread issues every MMA of the block, and a warp can only issue an instruction
// every few cycles, so descriptor arithmetic per MMA is kept to one 64-bit add.
// Descriptors advance by 32 bytes (2 in encoded units) per K step inside the swizzle atom.
__device__ __forceinline__ void umma_tf32_chunk(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t idesc,
                                                uint32_t accumulate_first) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 q, 0, 0;\n\t"
        "add.s64 a1, %1, 2;\n\tadd.s64 b1, %2, 2;\n\t"
        "add.s64 a2, %1, 4;\n\tadd.s64 b2, %2, 4;\n\t"
        "add.s64 a3, %1, 6;\n\tadd.s64 b3, %2, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], a1, b1, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], a2, b2, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], a3, b3, %3, q;\n\t}"
        ::"r"(tmem_d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate_first) : "memory");
}

// A chunk of the BF16 pass of the split mode: operands are 128-byte rows of 64 bf16
// ([a_hi | a_lo] against [b_lo | b_hi]), K = 16 per instruction, so the same four
// 32-byte steps cover the chunk.
__device__ __forceinline__ void umma_bf16_chunk(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t idesc,
                                                uint32_t accumulate_first) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 q, 0, 0;\n\t"
        "add.s64 a1, %1, 2;\n\tadd.s64 b1, %2, 2;\n\t"
        "add.s64 a2, %1, 4;\n\tadd.s64 b2, %2, 4;\n\t"
        "add.s64 a3, %1, 6;\n\tadd.s64 b3, %2, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, q;\n\t}"
        ::"r"(tmem_d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate_first) : "memory");
}

// The same two chunks with the A operand in tensor memory: lane = row, one 32-bit column per TF32 value (32 columns a
// chunk, 8 per K step) or per pair of BF16 values (32 columns, 8 per K step).
__device__ __forceinline__ void umma_tf32_chunk_ta(uint32_t tmem_d, uint32_t ta, uint64_t bd, uint32_t idesc,
                                                   uint32_t accumulate_first) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 q, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.s64 b1, %2, 2;\n\t"
        "add.u32 a2, %1, 16;\n\tadd.s64 b2, %2, 4;\n\t"
        "add.u32 a3, %1, 24;\n\tadd.s64 b3, %2, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [a1], b1, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [a2], b2, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [a3], b3, %3, q;\n\t}"
        ::"r"(tmem_d), "r"(ta), "l"(bd), "r"(idesc), "r"(accumulate_first) : "memory");
}
__device__ __forceinline__ void umma_bf16_chunk_ta(uint32_t tmem_d, uint32_t ta, uint64_t bd, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "setp.eq.b32 q, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.s64 b1, %2, 2;\n\t"
        "add.u32 a2, %1, 16;\n\tadd.s64 b2, %2, 4;\n\t"
        "add.u32 a3, %1, 24;\n\tadd.s64 b3, %2, 6;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, q;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, q;\n\t}"
        ::"r"(tmem_d), "r"(ta), "l"(bd), "r"(idesc) : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// Operand split into tensor memory: 16 values of a row (half 0 or 1 of a chunk) become A operands of both passes in
// this thread's lane: columns 0..31 the TF32 values (low 13 mantissa bits cleared), 32..63 the BF16 pairs
// [bf16(a_hi) x 32 | bf16(a_lo) x 32]. Warp-collective; the caller waits for the stores (tcgen05.wait::st).
__device__ __forceinline__ void split_half_to_tmem(const float (&f)[16], int half, uint32_t taddr) {
    uint32_t hi[16], ph[8], pl[8];
#pragma unroll
    for (int l = 0; l < 16; ++l) hi[l] = __float_as_uint(f[l]) & 0xffffe000u;
#pragma unroll
    for (int l = 0; l < 16; l += 2) {
        const float h0 = __uint_as_float(hi[l]), h1 = __uint_as_float(hi[l + 1]);
        const __nv_bfloat162 a = __floats2bfloat162_rn(h0, h1), b = __floats2bfloat162_rn(f[l] - h0, f[l + 1] - h1);
        ph[l / 2] = *reinterpret_cast<const uint32_t*>(&a);
        pl[l / 2] = *reinterpret_cast<const uint32_t*>(&b);
    }
    tmem_st16(taddr + half * 16, hi);
    tmem_st8(taddr + 32 + half * 8, ph);
    tmem_st8(taddr + 48 + half * 8, pl);
}
// The BF16 part of it alone, in the 32 columns at taddr (the TF32 pass then reads the tile as it landed in shared memory).
__device__ __forceinline__ void cross_row_to_tmem(const float4* row, int r, uint32_t taddr) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t ph[8], pl[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 v = row[(half * 4 + q) ^ (r & 7)];
            const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int l = 0; l < 4; l += 2) {
                const float h0 = __uint_as_float(__float_as_uint(f[l]) & 0xffffe000u), h1 = __uint_as_float(__float_as_uint(f[l + 1]) & 0xffffe000u);
                const __nv_bfloat162 a = __floats2bfloat162_rn(h0, h1), b = __floats2bfloat162_rn(f[l] - h0, f[l + 1] - h1);
                ph[q * 2 + l / 2] = *reinterpret_cast<const uint32_t*>(&a);
                pl[q * 2 + l / 2] = *reinterpret_cast<const uint32_t*>(&b);
            }
        }
        tmem_st8(taddr + half * 8, ph);
        tmem_st8(taddr + 16 + half * 8, pl);
    }
}
// One row of an activation tile (128 bytes in the 128-byte swizzle at `row`, which is row r of its tile).
__device__ __forceinline__ void split_row_to_tmem(const float4* row, int r, uint32_t taddr) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float f[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 v = row[(half * 4 + q) ^ (r & 7)];
            f[q * 4] = v.x; f[q * 4 + 1] = v.y; f[q * 4 + 2] = v.z; f[q * 4 + 3] = v.w;
        }
        split_half_to_tmem(f, half, taddr);
    }
}
// Gather form, three input channels: chunk kChunkNo of the row whose first tap lies at `win` in the window of 16-byte
// pixels (iw4 floats a row) - value k is channel k % 3 of tap k / 3. A tap is one 16-byte load, and which of its values
// go where is known when this is compiled. (A value at a time through a table of offsets into an operand in shared
// memory, as other channel counts have it: ResNet-18 at 128 images 2624 us, 2546 this way.)
template <int kK, int kChunkNo>
__device__ __forceinline__ void gather_chunk_to_tmem(const float* win, int iw4, uint32_t taddr) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int k0 = kChunkNo * 32 + half * 16;
        float f[16];
#pragma unroll
        for (int l = 0; l < 16; ++l) f[l] = 0.f;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            const int tap = k0 / 3 + i;
            if (tap < kK * kK && tap * 3 < k0 + 16) {
                const float4 v = *reinterpret_cast<const float4*>(win + (tap / kK) * iw4 + (tap % kK) * 4);
                const float c[3] = {v.x, v.y, v.z};
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const int at = tap * 3 + l - k0;
                    if (at >= 0 && at < 16) f[at] = c[l];
                }
            }
        }
        split_half_to_tmem(f, half, taddr);
    }
}
template <int kK>
__device__ __forceinline__ void gather_row_to_tmem(const float* win, int iw4, int chunk, uint32_t taddr) {
    if (chunk == 0) gather_chunk_to_tmem<kK, 0>(win, iw4, taddr);
    if (kK >= 5 && chunk == 1) gather_chunk_to_tmem<kK, 1>(win, iw4, taddr);
    if (kK >= 5 && chunk == 2) gather_chunk_to_tmem<kK, 2>(win, iw4, taddr);
    if (kK >= 7 && chunk == 3) gather_chunk_to_tmem<kK, 3>(win, iw4, taddr);
    if (kK >= 7 && chunk == 4) gather_chunk_to_tmem<kK, 4>(win, iw4, taddr);
}

// Arrivals that complete a stage's operand in tensor memory: the threads of the split group that built it, and one per
// warp of the other group, which has seen the stage's copies land. Without the second the ring could refill the stage
// twice before a warp that was not scheduled looked at it; waits name a phase by its parity, and that warp would sleep on.
constexpr uint32_t kXfBuilders = 128;
constexpr uint32_t kXfPassers = 4;

// One lane of a converged warp, for the roles that a single thread plays. Chosen this way - not as lane 0 - the compiler
// knows that exactly one thread runs the role and keeps addresses and descriptors in uniform registers, which is where
// the tensor-core and copy instructions take them from: an MMA costs its issuer 10 cycles instead of 55.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Operand split: piece index (row * 8 + 16-byte piece) -> the piece a thread takes instead, with the rows of
// every group of eight permuted to 0,4,1,5,2,6,3,7 (a bijection on the pieces of a tile).
__device__ __forceinline__ int split_row_order(int i) {
    const int x = i >> 3;
    const int r = (x & ~7) | ((x & 1) << 2) | ((x >> 1) & 3);
    return (r << 3) | (i & 7);
}

// Records the first error seen by any block in the library's device status word.
__device__ __forceinline__ void record_error(int* flag, int code) { atomicCAS(flag, 0, code); }


}  // namespace tc
}  // namespace ogle
