// Persistent tcgen05 kernel for the dense contractions (conv2d general/pointwise
// as implicit GEMM, gemm; tile shapes and tensor maps come from conv_tc.cu):
// one block per SM walks a list of output tiles and every stage of the pipeline
// overlaps with the others ACROSS tiles:
//
//   warp 0, 18  TMA producers (activation tiles / filter tiles): keep a ring of operand
//               stages full, running ahead into the next tile while the current one is
//               still being multiplied; two issuing threads because one tensor copy
//               costs its issuer over a hundred cycles;
//   warp 1      MMA issuer: accumulates tile i into one of 2-4 tensor-memory buffers while
//               the epilogues drain earlier tiles from the others;
//   warps 2-9   two epilogue groups of four warps, taking alternate 32-column slabs of every tile (so that the last
//               tile, or the only one, is stored by both), or alternate tiles where that is the faster rhythm:
//               tcgen05.ld -> bias / activation -> shared-memory staging in the
//               128-byte swizzle -> TMA tensor store (fully coalesced, clipped at the
//               tensor edge by the hardware);
//   warps 10-17 two operand-split groups for the split (fp32-grade) mode: they build the
//               BF16 operand [a_hi | a_lo] of the cross-term pass (idle in one-pass mode).
//               Where the accumulators leave room (tiles of up to 192 columns) both A operands -
//               TF32 and BF16 - are written into tensor memory, one row per thread, and the
//               multiplies read them there; else the BF16 one goes next to the activation tile in
//               shared memory. Same products in the same order either way: the same bits.
//
// What a chunk costs (clock stamps of the roles, one block; 3x3 64 -> 64 at 56 x 56 x 128 images, split mode): the
// ring, the copies and the operand split all wait for the issuing thread, which spent 1230 cycles a chunk: 55 per
// multiply, because its descriptors went from ordinary to uniform registers each time, and 200-300 per barrier it
// looks at. Elected by elect.sync it issues in 10 (elect_one), with A in tensor memory it looks at one barrier
// instead of two, and shared memory carries 16 KB less per chunk: 309 us with both in the old form (217 in the
// channels-on-M form), 195 us now; 19x19x512->75 3x3, 256 images: 570 (399) -> 318; 512->512 pointwise on SM
// pairs, 256 images at 19x19: 184 -> 155 (316 of about 400 TFLOP/s that a library reaches with the two passes).
// The copy producers keep lane 0: elected, they start the copies of bandwidth-bound layers in tighter bursts and
// those lose 3-4 %.
// Each group's work item has a latency of about a microsecond (shared-memory round
// trip plus a proxy fence); two groups per role keep that off the critical path.
//
// HBM traffic per tile is the algorithmic minimum: the activation tile is read
// once, the output tile written once; filters come from L2.
// All mbarrier waits are bounded and abort the block cleanly: the role records a code in
// the status word and raises the block's abort flag, the other roles leave at their next
// wait, the teardown waits for the multiplies and the
// operand copies still in flight, and only then is tensor memory freed and the block retired.
// The threads of an epilogue group may disagree about whether an accumulator came in time, and one that left by itself would
// be missed at the group's barriers: it goes on to the end of the block's tiles with them - with the block's abort flag up no
// wait lasts -, and what the group stores is then no valid output. With a residual operand, whose copies it would have to
// wait for, the group votes and leaves as one. (That vote in every form: 256 x 150 x 150 x 32 -> 64 pointwise 389 -> 440 us;
// a flag in shared memory that all look at, 427; this way 399.)
// The number of polls of the role waits can be shortened at run time (ogle_cuda_set_wait_limit,
// for tests of this path); the waits of the abort path itself always use the full bound.
#include <cuda_bf16.h>

#include <cstdlib>

#include "tc_common.cuh"

namespace ogle {
namespace {

using namespace tc;

constexpr int kThreads2 = 608;
constexpr int kMaxStages = 8;
constexpr int kTcSmem = 224 * 1024;           // a block always takes the whole of it: it then has its SM to itself
constexpr int kStagingBytes = kTileM * 128;   // one 128-row x 32-column fp32 slab

// Bounded wait of a role for its turn; also gives up early when another role of the block has
// aborted. `limit` is the number of polls (kSpinLimit unless the host shortened it).
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t limit) {
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

__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// The same, and whether all 128 threads say so. (The lanes leave a polling loop one by one; bar.red wants the whole warp.)
__device__ __forceinline__ bool group_and(int id, bool mine) {
    uint32_t all;
    mine = __all_sync(0xffffffffu, mine);
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbar.red.and.pred q, %1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"(id), "r"((uint32_t)mine) : "memory");
    return all != 0;
}

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t (&r)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

struct TileCoord { int n_tile, n0, h0, w0; };

template <bool kBeside = false>
__device__ __forceinline__ TileCoord tile_coord(const TcArgs& a, int tile) {
    TileCoord c;
    c.n_tile = tile % a.n_tiles;
    const int m_tile = tile / a.n_tiles;
    c.n0 = 0; c.h0 = 0;
    if (a.flat) {
        c.w0 = m_tile * (kBeside ? kTapsPixels : kTileM);
    } else {
        const int tw_i = m_tile % a.tiles_w;
        const int t = m_tile / a.tiles_w;
        c.w0 = tw_i * a.tw;
        c.h0 = (t % a.tiles_h) * a.th;
        c.n0 = (t / a.tiles_h) * a.tn;
    }
    return c;
}

struct WorkItem { int tile, ks, c_begin, c_end; };

// Compile-time form of the kernel, so that the common, unsplit one carries nothing of the others.
enum TcForm {
    kWhole = 0,       // a work item is a tile
    kRanges = 1,      // a range of a tile's reduction, combined through scratch or by reduce-add stores
    kCluster = 2,     // a range of a tile's reduction; the blocks of a cluster hold one tile's ranges and add them up
    // A tile of a 3x3 convolution whose filter rows lie side by side: per filter row (ky) and 32 channels one multiply of
    // 128 input pixels by [kx = 0 | 1 | 2] x BN channels; output pixel p is the sum of the first set's row p - 1, the
    // second's row p and the third's row p + 1, which the epilogue brings together. A third of the activation copies and
    // operand splits, and 3 BN columns a multiply: 64 channels alone leave the tensor cores half idle. With 64 channels a
    // tile a split-mode chunk moves 144 KB through shared memory (copies 64, operand split 16, multiplies 64), at the
    // 117 bytes a clock seen here 0.6 us, which is what it takes; a tile's epilogue adds about 1 us to that.
    // Split mode, before and after: 128 x 56 x 56 x 64 -> 64 172 -> 110 us, 128 x 28 x 28 x 128 -> 128 107 -> 94,
    // 128 x 14 x 14 x 256 -> 256 101 -> 95, 128 x 7 x 7 x 512 -> 512 115 -> 92; one pass, the first: 131 -> 74.
    kTaps = 3,
    kTapsRes = 4,     // ... with a residual operand (checked for at run time it costs 7 us of 110 where there is none)
    kWholeRes = 5,    // a work item is a tile, with a residual operand
    // Gather form whose filters all fit beside two input windows: filters copied once a block, a tile's window once, and the
    // ring's stages are places in tensor memory alone. Copied per chunk they were 140 KB a tile of the shared-memory
    // traffic that bounds the form.
    kKept = 6
};

template <TcForm kForm>
__device__ __forceinline__ WorkItem work_item(const TcArgs& a, int w, int chunks) {
    WorkItem it;
    if (kForm != kRanges && kForm != kCluster) {
        it.tile = w; it.ks = 0; it.c_begin = 0; it.c_end = chunks;
    } else {
        it.tile = w / a.split_k;
        it.ks = w - it.tile * a.split_k;
        it.c_begin = it.ks * a.chunks_per_split;
        it.c_end = it.c_begin + a.chunks_per_split < chunks ? it.c_begin + a.chunks_per_split : chunks;
    }
    return it;
}

__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// A float4 of another block's shared memory (addr: the same variable's address in this block).
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

// Cluster form: this block's band of the tile's rows, summed over the partial tiles of the cluster in rank order (the
// order the slices of the scratch form are added in: the same bits), then bias, residual operand and activation, and
// plain coalesced stores. The band's columns are dealt out as float4s, a row's neighbours to neighbouring threads.
// s_bias: the tile's columns' (with beta), staged while the accumulator was being computed.
__device__ __forceinline__ void cluster_reduce(const TcArgs& a, uint32_t partial, const float* s_bias, const float* __restrict__ bias) {
    const int ranks = a.split_k, tile = (int)blockIdx.x / ranks, rank = (int)blockIdx.x - tile * ranks;
    const TileCoord tc_ = tile_coord(a, tile);
    const int nbase = tc_.n_tile * a.BN;
    const int rows = a.flat ? kTileM : a.tn * a.th * a.tw;
    const int r0 = rows * rank / ranks, r1 = rows * (rank + 1) / ranks;
    const int quads = (a.Kp - nbase < a.BN ? a.Kp - nbase : a.BN) >> 2;
    for (int i = threadIdx.x; i < (r1 - r0) * quads; i += kThreads2) {
        const int row = r0 + i / quads, q = i % quads;
        long pixel;
        if (a.flat) {
            pixel = (long)tc_.w0 + row;
            if (pixel >= a.Wo) continue;
        } else {
            const int rw = row % a.tw, t2 = row / a.tw;
            const int n = tc_.n0 + t2 / a.th, h = tc_.h0 + t2 % a.th, w = tc_.w0 + rw;
            if (n >= a.N || h >= a.Ho || w >= a.Wo) continue;
            pixel = ((long)n * a.Ho + h) * a.Wo + w;
        }
        const int col = nbase + q * 4;                     // stacked column
        const bool second = a.split_col > 0 && col >= a.split_col;
        const int lcol = second ? col - a.split_col : col;
        const int real = second ? a.K - a.split_col : (a.split_col > 0 ? a.K1 : a.K);
        if (lcol >= real) continue;                        // between the two outputs
        const uint32_t at = partial + (uint32_t)((q >> 3) * kStagingBytes + row * 128 + (((q & 7) ^ (row & 7)) << 4));
        float4 res = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.res) res = __ldg(reinterpret_cast<const float4*>(a.res + pixel * a.res_ld + lcol));
        float4 part[8];
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < ranks) part[p] = load_cluster(at, (uint32_t)p);
        float v[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
        for (int p = 1; p < 8; ++p)
            if (p < ranks) { v[0] += part[p].x; v[1] += part[p].y; v[2] += part[p].z; v[3] += part[p].w; }
        const float rr[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (lcol + l < real) {
                if (a.bias_mode == 1) v[l] = fmaf(a.beta, __ldg(bias + pixel * a.ldc + lcol + l), a.alpha * v[l]);
                else v[l] = fmaf(a.alpha, v[l], s_bias[q * 4 + l]);
                if (a.res) v[l] += rr[l];
                v[l] = apply_act(v[l], a.act, a.lo, a.hi);
            } else {
                v[l] = 0.f;                                // padded lanes stay zero
            }
        }
        float* y = second ? a.y2 + pixel * a.y2_ld : a.y + pixel * a.y_ld;
        *reinterpret_cast<float4*>(y + lcol) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

template <TcForm kForm>
__global__ void __launch_bounds__(kThreads2, 1)
conv_tc2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBhi,
                const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmY,
                const __grid_constant__ CUtensorMap tmY2, const float* __restrict__ bias, const TcArgs a, int* err_flag) {
    // 1024-byte alignment (the 128-byte swizzle atom) comes from the declaration, so that
    // every byte of the 224 KB request is usable
    constexpr bool kSplit = kForm == kRanges || kForm == kCluster;
    constexpr bool kBeside = kForm == kTaps || kForm == kTapsRes;
    constexpr int kSets = kBeside ? 3 : 1;       // of BN accumulator columns
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kMaxStages], bar_xf[kMaxStages], bar_empty[kMaxStages];
    __shared__ __align__(8) uint64_t bar_acc_full[4], bar_acc_empty[4];
    __shared__ __align__(8) uint64_t bar_drain;     // abort path: the MMAs issued so far have finished
    __shared__ __align__(8) uint64_t bar_res[2];    // a group's slab of the residual operand has landed
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    __shared__ int s_issued[2];                     // operand copies issued by the two producers (abort path)
    __shared__ __align__(16) float s_bias[2][kBeside ? 64 : 256];
    __shared__ __align__(8) short s_goff[kBeside ? 4 : kMaxGatherK];   // gather form: window offset of each reduction index
    // taps side by side: the rows that the neighbouring warps of a group need, [group][warp][last or first row][column]
    __shared__ __align__(16) float s_edge[kBeside ? 2 * 4 * 2 * 32 : 4];

    grid_dependency_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool split = a.passes == 3;
    const uint32_t b_bytes = (uint32_t)(a.BN * kSets) * 128u;
    // activation part of a stage (none where the gather form builds its operand in tensor memory)
    const uint32_t a_bytes = a.gather && a.ta ? 0u : (split && !a.ta ? 2u : 1u) * kABytes;
    const int chunks = (kBeside ? 1 : a.kernel) * a.kernel * a.chunks_per_tap;
    const uint32_t stage_bytes = kForm == kKept ? 0u : a_bytes + (split ? 2u : 1u) * b_bytes + (a.gather ? (uint32_t)a.g_bytes : 0u);
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    // ring of operand stages (A | A cross (bf16 hi|lo), unless it lives in tensor memory | B_hi | B cross (bf16 lo|hi)),
    // then the output staging slabs
    auto sA = [&](int s) { return base + (uint32_t)s * stage_bytes; };
    auto sBhi = [&](int s) { return sA(s) + a_bytes; };
    auto sWin = [&](int s) { return sA(s) + a_bytes + (split ? 2u : 1u) * b_bytes; };   // gather form: input window
    const uint32_t kept_filters = (uint32_t)chunks * 2u * b_bytes;           // (kKept) then the two windows
    const uint32_t staging_off = kForm == kKept ? kept_filters + 2u * (uint32_t)a.g_bytes : (uint32_t)a.stages * stage_bytes;
    {
        // the layout must fit what the launch reserved (it does when the base is 1024-aligned as
        // declared); checked, not assumed, because an overrun would write past the block's window
        uint32_t dyn;
        asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        const uint32_t need = (base - smem_u32(smem_raw)) + staging_off +
                              (uint32_t)(a.epi_groups * a.epi_slabs) * (uint32_t)kStagingBytes;
        if (need > dyn) {
            if (threadIdx.x == 0) record_error(err_flag, 9);
            return;
        }
    }

    const int acc_cols = a.BN * kSets;     // tensor-memory columns of one accumulator
    const int rows_in_tile = a.flat ? kTileM : a.tn * a.th * a.tw;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 32 * 18) {
        // the copy descriptors are fetched while the barriers and tensor memory are being set up
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmBhi)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmBlo)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmY)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmY2)) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&bar_full[s], 2);     // one arrive.expect_tx from each producer
            mbar_init(&bar_xf[s], a.ta ? kXfBuilders + kXfPassers : (uint32_t)(a.xf_groups * 128));
            mbar_init(&bar_empty[s], 1);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(&bar_acc_full[i], 1);
            mbar_init(&bar_acc_empty[i], (uint32_t)(128 * a.epi_groups));
        }
        mbar_init(&bar_drain, 1);
        if (kForm == kTapsRes || kForm == kWholeRes) {
            mbar_init(&bar_res[0], 1);
            mbar_init(&bar_res[1], 1);
        }
        s_abort = 0;
        s_issued[0] = 0; s_issued[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (!kBeside && a.gather) {
        // reduction index k = (ky * kernel + kx) * C + c -> float offset of that value in the
        // [g_ih][g_iw][4] input window relative to the output pixel's first tap; -1 = padding column
        const int kred = a.g_k * a.g_k * a.g_C;
        for (int k = threadIdx.x; k < a.chunks_per_tap * kChunk && k < kMaxGatherK; k += blockDim.x) {
            int off = -1;
            if (k < kred) {
                const int tap = k / a.g_C, c = k - tap * a.g_C;
                const int ky = tap / a.g_k, kx = tap - ky * a.g_k;
                off = (ky * a.g_iw + kx) * 4 + c;
            }
            s_goff[k] = (short)off;
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)a.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = tmem_slot;
    const uint32_t tmem_a = tmem_d + (uint32_t)(a.n_acc * acc_cols);      // A operands in tensor memory: 64 (32) columns per stage
    // barriers, tensor memory and tables are set up; what follows reads and writes global memory
    grid_dependency_wait();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            const uint32_t tx = (uint32_t)rows_in_tile * 128u;
            // ring position kept incrementally (no divisions in this loop: one thread feeds
            // the whole pipeline and every cycle here is on the critical path)
            int s = 0;                 // stage of the next chunk
            uint32_t wrap = 0;         // how many times the ring has wrapped
            int issued = 0;            // chunks in flight bookkeeping for the abort path
            bool ok = true;
            int window = 0;
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x, window ^= 1) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                const TileCoord tc_ = tile_coord<kBeside>(a, wi.tile);
                int ax, ay, an;
                if constexpr (kBeside) {
                    // from the pixel before the first output pixel on
                    const int p = tc_.w0 > 0 ? tc_.w0 - 1 : 0, line = p / a.oW;
                    an = line / a.oH;
                    ax = p - line * a.oW;
                    ay = line - an * a.oH - 1;
                } else {
                    ax = a.flat ? tc_.w0 : tc_.w0 * a.stride - a.pad;
                    ay = a.flat ? 0 : tc_.h0 * a.stride - a.pad;
                    an = tc_.n0;
                }
                // gather form: the tile's input window
                auto load_window = [&](uint32_t to, uint64_t* bar) {
                    if (a.g_iw > 128) tma_load_4d(to, &tmA, bar, 0, ax, ay, an);
                    else tma_load_4d(to, &tmA, bar, 2 * ax, ay, an, 0);
                };
                // position of the first chunk: filter row, filter column, channel offset
                int ky = 0, kx = 0, c0 = 0;
                if (kSplit && wi.c_begin != 0) {      // only the later ranges of a split reduction pay the divisions
                    const int tap0 = wi.c_begin / a.chunks_per_tap;
                    ky = tap0 / a.kernel;
                    kx = tap0 - ky * a.kernel;
                    c0 = (wi.c_begin - tap0 * a.chunks_per_tap) * kChunk;
                }
                for (int it = wi.c_begin; it < wi.c_end; ++it) {
                    if (wrap > 0) ok = wait_or_abort(&bar_empty[s], (wrap - 1) & 1u, abort_flag, a.spin_limit);
                    if (!ok) { record_error(err_flag, 1); break; }
                    if (kForm == kKept) {
                        // (the ring is at most a stage longer than a tile's reduction: the window before the last has been read)
                        if (it == 0) {
                            mbar_expect_tx(&bar_full[s], (uint32_t)(a.g_iw * a.g_ih * 16));
                            load_window(base + kept_filters + (uint32_t)(window * a.g_bytes), &bar_full[s]);
                        } else {
                            mbar_arrive(&bar_full[s]);
                        }
                    } else if (a.gather) {
                        mbar_expect_tx(&bar_full[s], (uint32_t)(a.g_iw * a.g_ih * 16));
                        load_window(sWin(s), &bar_full[s]);
                    } else {
                        mbar_expect_tx(&bar_full[s], tx);
                        if constexpr (kBeside) tma_load_im2col(sA(s), &tmA, &bar_full[s], c0, ax, ay, an, 0, ky);
                        else tma_load_4d(sA(s), &tmA, &bar_full[s], c0, ax + kx * a.dil, ay + ky * a.dil, an);
                    }
                    ++issued;
                    if (++s == a.stages) { s = 0; ++wrap; }
                    // next chunk: channels fastest, then filter column, then filter row
                    c0 += kChunk;
                    if (c0 == a.Cp32) { c0 = 0; if (kBeside || ++kx == a.kernel) { kx = 0; ++ky; } }
                }
            }
            if (!ok) s_abort = 1;
            s_issued[0] = issued;      // the teardown waits for these copies if the block aborts
        }
    } else if (warp == 18) {
        // ------------------------------------------------ TMA producer, filter tiles
        if (lane == 0) {
            const uint32_t tx = (split ? 2u : 1u) * b_bytes;
            int s = 0;
            uint32_t wrap = 0;
            int issued = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                const int bcol = (wi.tile % a.n_tiles) * a.BN;
                int brow = wi.c_begin * kChunk, ky = 0;      // (taps side by side: channel and filter row)
                for (int it = wi.c_begin; it < wi.c_end; ++it) {
                    if (wrap > 0) ok = wait_or_abort(&bar_empty[s], (wrap - 1) & 1u, abort_flag, a.spin_limit);
                    if (!ok) { record_error(err_flag, 7); break; }
                    if (kForm == kKept) {
                        if (w == (int)blockIdx.x) {
                            const uint32_t to = base + (uint32_t)it * 2u * b_bytes;
                            mbar_expect_tx(&bar_full[s], tx);
                            tma_load_2d(to, &tmBhi, &bar_full[s], brow, bcol);
                            tma_load_2d(to + b_bytes, &tmBlo, &bar_full[s], brow, bcol);
                        } else {
                            mbar_arrive(&bar_full[s]);
                        }
                        ++issued;
                        if (++s == a.stages) { s = 0; ++wrap; }
                        brow += kChunk;
                        continue;
                    }
                    mbar_expect_tx(&bar_full[s], tx);
                    if constexpr (kBeside) {
                        // the filter row's three taps, one below the other in shared memory (with a copy for each its
                        // issuer falls behind: one pass, 7 x 7 x 512, 128 images, 67.6 us, 61.3 with one for all)
                        tma_load_3d(sBhi(s), &tmBhi, &bar_full[s], brow, bcol, ky * 3);
                        if (split) tma_load_3d(sBhi(s) + b_bytes, &tmBlo, &bar_full[s], brow, bcol, ky * 3);
                    } else {
                        tma_load_2d(sBhi(s), &tmBhi, &bar_full[s], brow, bcol);
                        if (split) tma_load_2d(sBhi(s) + b_bytes, &tmBlo, &bar_full[s], brow, bcol);   // the BF16 cross operand
                    }
                    ++issued;
                    if (++s == a.stages) { s = 0; ++wrap; }
                    brow += kChunk;       // packed filter rows follow the chunk order
                    if (kBeside && brow == a.Cp32) { brow = 0; ++ky; }
                }
            }
            if (!ok) s_abort = 1;
            s_issued[1] = issued;
        }
    } else if (warp == 1) {
        // -------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(acc_cols >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
            // kind::f16 with BF16 operands (format code 1), fp32 accumulation
            const uint32_t idesc_bf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(acc_cols >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
            int s = 0;
            uint32_t ph = 0;           // parity of the ring pass
            bool ok = true;
            int ti = 0;
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x, ++ti) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                const int as = a.n_acc == 4 ? (ti & 3) : (ti & 1), use = a.n_acc == 4 ? (ti >> 2) : (ti >> 1);
                if (use > 0) ok = wait_or_abort(&bar_acc_empty[as], (uint32_t)((use - 1) & 1), abort_flag, a.spin_limit);
                if (!ok) { record_error(err_flag, 5); s_abort = 1; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem_d + (uint32_t)(as * acc_cols);
                for (int it = wi.c_begin; it < wi.c_end; ++it) {
                    // gather form, A in tensor memory: the operand exists only once the split warps have built it (they
                    // arrive after the stage's copies have landed)
                    ok = wait_or_abort(a.gather || a.ta == 1 ? &bar_xf[s] : &bar_full[s], ph, abort_flag, a.spin_limit);
                    if (!ok) { record_error(err_flag, 2); s_abort = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = umma_desc(sA(s)), bd = umma_desc(kForm == kKept ? base + (uint32_t)it * 2u * b_bytes : sBhi(s));
                    const uint32_t acc_flag = it > (kSplit ? wi.c_begin : 0) ? 1u : 0u;     // the first chunk overwrites
                    if (a.ta == 1) {
                        const uint32_t ta = tmem_a + (uint32_t)s * 64u;
                        umma_tf32_chunk_ta(d, ta, bd, idesc, acc_flag);
                        umma_bf16_chunk_ta(d, ta + 32u, bd + (b_bytes >> 4), idesc_bf16);
                        umma_commit(&bar_empty[s]);
                        if (++s == a.stages) { s = 0; ph ^= 1u; }
                        continue;
                    }
                    umma_tf32_chunk(d, ad, bd, idesc, acc_flag);            // a x b_hi (a is read as its high part)
                    if (split) {
                        // cross terms [a_hi | a_lo] x [b_lo | b_hi] in BF16, once the split role has
                        // written the activation parts
                        if (!a.gather) {
                            ok = wait_or_abort(&bar_xf[s], ph, abort_flag, a.spin_limit);
                            if (!ok) { record_error(err_flag, 2); s_abort = 1; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        if (kBeside && a.ta == 2) umma_bf16_chunk_ta(d, tmem_a + (uint32_t)s * 32u, bd + (b_bytes >> 4), idesc_bf16);
                        else umma_bf16_chunk(d, ad + (kABytes >> 4), bd + (b_bytes >> 4), idesc_bf16, 1u);
                    }
                    umma_commit(&bar_empty[s]);
                    if (++s == a.stages) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit(&bar_acc_full[as]);
            }
        }
    } else if (warp >= 10) {
        // --------------------------------------------------- operand split (split mode)
        // Builds the BF16 operand of the cross-term pass next to the activation tile:
        // row r = [bf16(a_hi) x 32 | bf16(a_lo) x 32] (128 bytes, same 128-byte swizzle), with
        // a_hi = the value with its low 13 mantissa bits cleared (what the TF32 pass reads)
        // and a_lo = a - a_hi. The fp32 tile itself is left as TMA delivered it. One or two
        // warp groups work on EVERY chunk together.
        const int xg = (warp - 10) >> 2;           // group 0 or 1
        if (a.ta) {
            // A operands in tensor memory: a thread takes one row, the two groups take alternate chunks
            const int r = (warp & 3) * 32 + lane;
            const uint32_t lanes = tmem_a + ((uint32_t)((warp & 3) * 32) << 16);
            // gather form: this row's first tap in the input window
            const int g_row = a.gather ? ((r / a.tw * a.stride) * a.g_iw + r % a.tw * a.stride) * 4 : 0;
            int s = 0, turn = 0;
            uint32_t ph = 0;
            bool ok = true;
            int window = 0;
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x, window ^= 1) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                for (int it = wi.c_begin; it < wi.c_end; ++it) {
                    // Every stage is waited for in turn, also those of the other group's chunks: copies land out of
                    // order, and a group that only looked at every second chunk could, in a ring of three or five
                    // stages, meet a barrier two phases behind and take its parity for the coming one. And the multiply
                    // waits for both groups, so that the ring cannot pass the one that has nothing to build.
                    // The stage is refilled only after the multiplies that read it - shared and tensor memory - are done.
                    // (The lanes leave the polling loop one by one; the tensor-memory stores want the whole warp.)
                    ok = wait_or_abort(&bar_full[s], ph, abort_flag, a.spin_limit);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { record_error(err_flag, 3); s_abort = 1; break; }
                    if (turn == xg) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const unsigned char* stage = base_ptr + (size_t)s * stage_bytes;
                        const uint32_t to = lanes + (uint32_t)s * (kBeside && a.ta == 2 ? 32u : 64u);
                        if (kBeside && a.ta == 2) {
                            cross_row_to_tmem(reinterpret_cast<const float4*>(stage + (size_t)r * 128), r, to);
                        } else if (kBeside || !a.gather) {
                            split_row_to_tmem(reinterpret_cast<const float4*>(stage + (size_t)r * 128), r, to);
                        } else {
                            const float* win = reinterpret_cast<const float*>(kForm == kKept ? base_ptr + kept_filters + (size_t)(window * a.g_bytes)
                                                                                             : stage + 2u * b_bytes) + g_row;
                            if (a.g_k == 7) gather_row_to_tmem<7>(win, a.g_iw * 4, it, to);
                            else if (a.g_k == 5) gather_row_to_tmem<5>(win, a.g_iw * 4, it, to);
                            else gather_row_to_tmem<3>(win, a.g_iw * 4, it, to);
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&bar_xf[s]);
                    } else if (lane == 0) {
                        mbar_arrive(&bar_xf[s]);
                    }
                    turn ^= 1;
                    if (++s == a.stages) { s = 0; ph ^= 1u; }
                }
            }
        } else if ((split || a.gather) && xg < a.xf_groups) {
            const int nthr = a.xf_groups * 128;
            const int t = threadIdx.x - 320;       // 0 .. nthr-1
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            // gather form: a thread always builds the same 16-byte piece (t & 7) of the same rows, so the
            // rows' offsets into the input window are computed once: g_row[q] for row (t >> 3) + q * nthr / 8.
            // The four reduction indices of the piece change with the chunk and come from s_goff.
            int g_row[4] = {0, 0, 0, 0};
            if (a.gather) {
                for (int q = 0; q < 4; ++q) {
                    const int r = (t >> 3) + q * (nthr >> 3);
                    const int ry = r / a.tw, rx = r - ry * a.tw;          // tn == 1, tw * th == 128 in this form
                    g_row[q] = ((ry * a.stride) * a.g_iw + rx * a.stride) * 4;
                }
            }
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                for (int it = wi.c_begin; it < wi.c_end; ++it) {
                    ok = wait_or_abort(&bar_full[s], ph, abort_flag, a.spin_limit);
                    if (!ok) { record_error(err_flag, 3); s_abort = 1; break; }
                    float4* pa = reinterpret_cast<float4*>(base_ptr + (size_t)s * stage_bytes);
                    float4* pl = pa + kABytes / 16;
                    uint2* p2 = reinterpret_cast<uint2*>(pl);                 // 8-byte pieces of the BF16 tile
                    if (a.gather) {
                        // build the operand from the input window: one 16-byte piece (4 values) per step;
                        // which values and which rows this thread handles never changes (see g_off / g_row)
                        const float* win = reinterpret_cast<const float*>(base_ptr + (size_t)s * stage_bytes +
                                                                          (split ? 2u : 1u) * (kABytes + b_bytes));
                        const int j = t & 7;
                        const short4 go = *reinterpret_cast<const short4*>(&s_goff[it * kChunk + j * 4]);
                        const int g_off[4] = {go.x, go.y, go.z, go.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if (q * nthr >= kABytes / 16) break;
                            const int r = (t >> 3) + q * (nthr >> 3);
                            const float* w0 = win + g_row[q];
                            float v[4];
#pragma unroll
                            for (int l = 0; l < 4; ++l) v[l] = g_off[l] >= 0 ? w0[g_off[l]] : 0.f;
                            pa[(r << 3) + (j ^ (r & 7))] = make_float4(v[0], v[1], v[2], v[3]);
                            if (split) {
                                float h[4];
#pragma unroll
                                for (int l = 0; l < 4; ++l) h[l] = __uint_as_float(__float_as_uint(v[l]) & 0xffffe000u);
                                const __nv_bfloat162 h01 = __floats2bfloat162_rn(h[0], h[1]), h23 = __floats2bfloat162_rn(h[2], h[3]);
                                const __nv_bfloat162 l01 = __floats2bfloat162_rn(v[0] - h[0], v[1] - h[1]),
                                                     l23 = __floats2bfloat162_rn(v[2] - h[2], v[3] - h[3]);
                                uint2 hv, lv;
                                hv.x = *reinterpret_cast<const uint32_t*>(&h01); hv.y = *reinterpret_cast<const uint32_t*>(&h23);
                                lv.x = *reinterpret_cast<const uint32_t*>(&l01); lv.y = *reinterpret_cast<const uint32_t*>(&l23);
                                const int ch = (j >> 1) ^ (r & 7), cl = (4 + (j >> 1)) ^ (r & 7);
                                p2[r * 16 + ch * 2 + (j & 1)] = hv;
                                p2[r * 16 + cl * 2 + (j & 1)] = lv;
                            }
                        }
                    } else
                    for (int i0 = t; i0 < kABytes / 16; i0 += nthr) {
                        // rows of a group of eight are taken in the order 0,4,1,5,2,6,3,7: the four rows a warp
                        // handles at once then put their BF16 halves into both halves of the banks (rows r and
                        // r + 4 swizzle to different 64-byte halves), two wavefronts per store instead of four
                        const int i = split_row_order(i0);
                        const float4 v = pa[i];
                        const int r = i >> 3, j = (i & 7) ^ (r & 7);          // row; logical 16-byte chunk = channels 4j..4j+3
                        float4 h;
                        h.x = __uint_as_float(__float_as_uint(v.x) & 0xffffe000u);
                        h.y = __uint_as_float(__float_as_uint(v.y) & 0xffffe000u);
                        h.z = __uint_as_float(__float_as_uint(v.z) & 0xffffe000u);
                        h.w = __uint_as_float(__float_as_uint(v.w) & 0xffffe000u);
                        const __nv_bfloat162 h01 = __floats2bfloat162_rn(h.x, h.y), h23 = __floats2bfloat162_rn(h.z, h.w);
                        const __nv_bfloat162 l01 = __floats2bfloat162_rn(v.x - h.x, v.y - h.y), l23 = __floats2bfloat162_rn(v.z - h.z, v.w - h.w);
                        uint2 hv, lv;
                        hv.x = *reinterpret_cast<const uint32_t*>(&h01); hv.y = *reinterpret_cast<const uint32_t*>(&h23);
                        lv.x = *reinterpret_cast<const uint32_t*>(&l01); lv.y = *reinterpret_cast<const uint32_t*>(&l23);
                        // bf16 column 4j (hi) / 32 + 4j (lo): 16-byte chunk j/2 resp. 4 + j/2, half j & 1
                        const int ch = (j >> 1) ^ (r & 7), cl = (4 + (j >> 1)) ^ (r & 7);
                        p2[r * 16 + ch * 2 + (j & 1)] = hv;
                        p2[r * 16 + cl * 2 + (j & 1)] = lv;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive(&bar_xf[s]);
                    if (++s == a.stages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if constexpr (kBeside) {
        // -------------------------------------------- epilogue, taps side by side
        // The groups take alternate 32-channel slabs. A thread's value is the sum of its own row of the second set, the
        // row before it of the first and the row behind it of the third - a neighbouring lane's, or, at a warp's ends,
        // left in shared memory by the neighbouring warp - where those pixels lie in the same row of the image.
        const int eg = (warp - 2) >> 2, t = (threadIdx.x - 64) & 127, q = warp & 3, row = q * 32 + lane, bar_id = 1 + eg;
        if (eg < a.epi_groups) {
            const uint32_t my_staging = staging_off + (uint32_t)(eg * a.epi_slabs) * (uint32_t)kStagingBytes;
            unsigned char* staging = base_ptr + my_staging;
            float* edge = s_edge + eg * 256;
            // (the tile's first and last rows have none: nothing of them is kept, or they are an image row's ends)
            const bool at_end = (lane == 0 && q > 0) || (lane == 31 && q < 3);
            const float* my_edge = lane == 0 ? edge + (q - 1) * 64 : edge + (q + 1) * 64 + 32;
            float* my_bias = s_bias[eg];
            bool ok = true, came = true;        // (came: looked at with a residual operand only)
            int ti = 0, staged_nbase = -1, round_no = 0;
            int res_copies = 0;        // of the residual operand, asked for by this thread
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x, ++ti) {
                const TileCoord tc_ = tile_coord<kBeside>(a, w);
                const int as = a.n_acc == 4 ? (ti & 3) : (ti & 1), use = a.n_acc == 4 ? (ti >> 2) : (ti >> 1);
                const int nbase = tc_.n_tile * a.BN;
                int groups = (a.Kp - nbase + 31) / 32;
                if (groups > a.BN / 32) groups = a.BN / 32;
                const int step = a.epi_groups;
                const int first = a.epi_groups == 1 || ((eg + ti) & 1) == 0 ? 0 : 1;
                if (nbase != staged_nbase) {
                    for (int i = t; i < a.BN; i += 128) my_bias[i] = a.bias_mode == 2 && nbase + i < a.K ? a.beta * bias[nbase + i] : 0.f;
                    staged_nbase = nbase;
                }
                // this thread's pixel, its place in the image row and in the staging slab
                const int shift = tc_.w0 > 0 ? 1 : 0, out_row = row - shift, pixel = tc_.w0 + out_row;
                const int x = (pixel < 0 ? 0 : pixel) % a.oW;
                const bool left = x > 0, right = x + 1 < a.oW, mine = out_row >= 0 && out_row < kTapsPixels;
                // A slab is free once the store from it has been read; the residual operand's values are then copied to it
                // - a thread that loads its own row of them holds up the tile: 56 x 56 x 64, 128 images, 145 us -,
                // and each thread adds its row and leaves the sum in their place.
                auto free_slab = [&](int slab, int lcol) {
                    if (a.epi_slabs == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    if constexpr (kForm == kTapsRes) {
                        ++res_copies;
                        mbar_expect_tx(&bar_res[eg], (uint32_t)kTapsPixels * 128u);
                        tma_load_4d(base + my_staging + (uint32_t)slab * (uint32_t)kStagingBytes, &tmY2, &bar_res[eg], lcol, tc_.w0, 0, 0);
                    }
                };
                if (t == 0 && first < groups) free_slab(round_no % a.epi_slabs, nbase + first * 32);
                if (!__all_sync(0xffffffffu, wait_or_abort(&bar_acc_full[as], (uint32_t)(use & 1), abort_flag, a.spin_limit))) {
                    record_error(err_flag, 4);
                    s_abort = 1;
                    came = false;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (first >= groups) {                  // none of them this time
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(&bar_acc_empty[as]);
                }
                for (int g0 = first; g0 < groups; g0 += step) {
                    const int sb = round_no % a.epi_slabs;
                    ++round_no;
                    const int col = g0 * 32;
                    const uint32_t taddr = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * acc_cols + col);
                    if (t == 0 && g0 != first) free_slab(sb, nbase + col);
#pragma unroll
                    for (int side = 0; side < 2; ++side) {
                        uint32_t r[32];
                        tmem_ld32(r, taddr + (uint32_t)(side * 2 * a.BN));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (lane == (side ? 0 : 31)) {
                            uint4* e = reinterpret_cast<uint4*>(edge + (q * 2 + side) * 32);
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) e[c4] = make_uint4(r[c4 * 4], r[c4 * 4 + 1], r[c4 * 4 + 2], r[c4 * 4 + 3]);
                        }
                    }
                    if constexpr (kForm == kTapsRes) {
                        ok = group_and(bar_id, came && wait_or_abort(&bar_res[eg], (uint32_t)((round_no - 1) & 1), abort_flag, a.spin_limit));
                        if (!ok) { record_error(err_flag, 4); s_abort = 1; break; }
                    } else {
                        group_sync(bar_id);
                    }
                    float4* dst = reinterpret_cast<float4*>(staging + (size_t)sb * kStagingBytes + (size_t)(mine ? out_row : 0) * 128);
                    // which output this slab belongs to, and its first column there
                    const bool second = a.split_col > 0 && nbase + col >= a.split_col;
                    const int lcol = second ? nbase + col - a.split_col : nbase + col;
                    const int kout = second ? a.K - a.split_col : (a.split_col > 0 ? a.K1 : a.K);
                    const bool fast = lcol + 32 <= kout;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t r0[16], r1[16], r2[16];
                        tmem_ld16(r0, taddr + (uint32_t)(half * 16));
                        tmem_ld16(r1, taddr + (uint32_t)(a.BN + half * 16));
                        tmem_ld16(r2, taddr + (uint32_t)(2 * a.BN + half * 16));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (half == 1 && g0 + step >= groups) {
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            mbar_arrive(&bar_acc_empty[as]);
                        }
#pragma unroll
                        for (int c4 = 0; c4 < 4; ++c4) {
                            float4 over = make_float4(0.f, 0.f, 0.f, 0.f);          // the neighbouring warp's row
                            if (at_end) over = *reinterpret_cast<const float4*>(my_edge + half * 16 + c4 * 4);
                            const float ov[4] = {over.x, over.y, over.z, over.w};
                            const float4 bb = *reinterpret_cast<const float4*>(my_bias + col + half * 16 + c4 * 4);
                            const float bv[4] = {bb.x, bb.y, bb.z, bb.w};
                            float4 res = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (kForm == kTapsRes && mine) res = dst[(half * 4 + c4) ^ (out_row & 7)];
                            const float rv[4] = {res.x, res.y, res.z, res.w};
                            float v[4];
#pragma unroll
                            for (int l = 0; l < 4; ++l) {
                                float l0 = __uint_as_float(__shfl_up_sync(0xffffffffu, r0[c4 * 4 + l], 1));
                                float l2 = __uint_as_float(__shfl_down_sync(0xffffffffu, r2[c4 * 4 + l], 1));
                                if (lane == 0) l0 = ov[l];
                                if (lane == 31) l2 = ov[l];
                                float sum = (left ? l0 : 0.f) + __uint_as_float(r1[c4 * 4 + l]);
                                if (right) sum += l2;
                                v[l] = fmaf(a.alpha, sum, bv[l]);
                                if (kForm == kTapsRes) v[l] += rv[l];
                            }
                            if (a.act == OGLE_ACT_RELU) {
#pragma unroll
                                for (int l = 0; l < 4; ++l) v[l] = fmaxf(v[l], 0.f);
                            } else if (a.act == OGLE_ACT_CLIP) {
#pragma unroll
                                for (int l = 0; l < 4; ++l) v[l] = fminf(fmaxf(v[l], a.lo), a.hi);
                            }
                            if (!fast) {
#pragma unroll
                                for (int l = 0; l < 4; ++l)
                                    if (lcol + half * 16 + c4 * 4 + l >= kout) v[l] = 0.f;             // padded lanes stay zero
                            }
                            if (mine) dst[(half * 4 + c4) ^ (out_row & 7)] = make_float4(v[0], v[1], v[2], v[3]);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    group_sync(bar_id);
                    if (t == 0) {
                        tma_store_4d(second ? &tmY2 : &tmY, base + my_staging + (uint32_t)sb * (uint32_t)kStagingBytes, lcol, tc_.w0, 0, 0);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            }
            // (an aborting block waits for the copy it has asked for)
            if (!ok && res_copies > 0) mbar_wait(&bar_res[eg], (uint32_t)((res_copies - 1) & 1));
            if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
    } else if constexpr (kForm == kCluster) {
        // ------------------------------------------------------------ partial tile
        // One work item per block: its raw sums go to the operand ring, which the last multiply has left, slab by slab
        // in the swizzle of the staging slabs; both groups take part.
        const int row = (warp & 3) * 32 + lane;
        if (warp < 6) {
            const int nbase = tile_coord(a, (int)blockIdx.x / a.split_k).n_tile * a.BN;
            for (int i = threadIdx.x - 64; i < a.BN; i += 128)
                s_bias[0][i] = a.bias_mode == 2 && nbase + i < a.K ? a.beta * __ldg(bias + nbase + i) : 0.f;
        }
        bool ok = wait_or_abort(&bar_acc_full[0], 0u, abort_flag, a.spin_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { record_error(err_flag, 4); s_abort = 1; }
        else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int g = (warp - 2) >> 2; g < a.BN / 32; g += 2) {
                uint32_t r[32];
                tmem_ld32(r, tmem_d + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * 32));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                uint4* dst = reinterpret_cast<uint4*>(base_ptr + (size_t)g * kStagingBytes + (size_t)row * 128);
#pragma unroll
                for (int c4 = 0; c4 < 8; ++c4) dst[c4 ^ (row & 7)] = make_uint4(r[c4 * 4], r[c4 * 4 + 1], r[c4 * 4 + 2], r[c4 * 4 + 3]);
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int eg = (warp - 2) >> 2;               // group 0 or 1
        if (eg < a.epi_groups) {
            const int t = (threadIdx.x - 64) & 127;
            const int q = warp & 3;                   // TMEM lane quarter this warp may read
            const int row = q * 32 + lane;
            const int bar_id = 1 + eg;
            float* my_bias = s_bias[eg];
            // each group owns one or two staging slabs and fills them in rounds
            const uint32_t my_staging = staging_off + (uint32_t)(eg * a.epi_slabs) * (uint32_t)kStagingBytes;
            unsigned char* staging = base_ptr + my_staging;
            bool ok = true, came = true;
            int ti = 0;
            int staged_nbase = -1;
            int round_no = 0;          // rounds of this group so far (selects the staging slab)
            int res_copies = 0;        // of the residual operand, asked for by this thread
            for (int w = blockIdx.x; w < a.total_work && ok; w += gridDim.x, ++ti) {
                const WorkItem wi = work_item<kForm>(a, w, chunks);
                const TileCoord tc_ = tile_coord<kBeside>(a, wi.tile);
                const int as = a.n_acc == 4 ? (ti & 3) : (ti & 1), use = a.n_acc == 4 ? (ti >> 2) : (ti >> 1);
                const int nbase = tc_.n_tile * a.BN;
                int groups = (a.Kp - nbase + 31) / 32;
                if (groups > a.BN / 32) groups = a.BN / 32;
                // this group's slabs: first, first + step, ...
                const int step = a.epi_share ? a.epi_groups : 1;
                const int first = a.epi_groups == 1 || ((eg + ti) & 1) == 0 ? 0 : (a.epi_share ? 1 : groups);
                long pix = 0;
                if (a.bias_mode == 1) {
                    pix = (long)tc_.w0 + row;
                    if (pix >= a.Wo) pix = a.Wo - 1;  // clipped rows are dropped by the store; keep reads in range
                }
                // bias of this tile's columns (pre-multiplied by beta), staged while the accumulator
                // is still being produced; skipped when the previous tile had the same columns.
                // Safe to overwrite here: every thread of the group passed the sync that follows the
                // last read of the previous tile's values.
                // (with a split reduction only the first work item of a tile adds the bias)
                const int bias_key = kSplit ? nbase * 2 + (wi.ks == 0 ? 1 : 0) : nbase;
                if (bias_key != staged_nbase) {
                    for (int i = t; i < a.BN; i += 128)
                        my_bias[i] = (a.bias_mode == 2 && (!kSplit || (wi.ks == 0 && !a.ws_mode)) && nbase + i < a.K) ? a.beta * bias[nbase + i] : 0.f;
                    staged_nbase = bias_key;
                }
                // A slab is free once the store from it has been read. A residual operand's values are then copied to it, and
                // each thread adds its row and leaves the sum in their place.
                auto free_slab = [&](int slab, int lcol) {
                    if (a.epi_slabs == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    if constexpr (kForm == kWholeRes) {
                        ++res_copies;
                        mbar_expect_tx(&bar_res[eg], (uint32_t)rows_in_tile * 128u);
                        tma_load_4d(base + my_staging + (uint32_t)slab * (uint32_t)kStagingBytes, &tmY2, &bar_res[eg], lcol, tc_.w0, tc_.h0, tc_.n0);
                    }
                };
                if (kForm == kWholeRes && t == 0 && first < groups) free_slab(round_no % a.epi_slabs, nbase + first * 32);
                if (!wait_or_abort(&bar_acc_full[as], (uint32_t)(use & 1), abort_flag, a.spin_limit)) {
                    record_error(err_flag, 4);
                    s_abort = 1;
                    came = false;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (first >= groups) {                  // none of them this time
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(&bar_acc_empty[as]);
                }
                // one 32-column slab per round through a ring of one or two staging slabs: a slab
                // is reused once the store issued from it (one or two rounds ago) has read it, so
                // with two slabs a round never waits for the store of the round just before
                for (int g0 = first; g0 < groups; g0 += step) {
                    const int sb = round_no % a.epi_slabs;
                    ++round_no;
                    if (t == 0 && (kForm != kWholeRes || g0 != first)) free_slab(sb, nbase + g0 * 32);
                    if constexpr (kForm == kWholeRes) {
                        ok = group_and(bar_id, came && wait_or_abort(&bar_res[eg], (uint32_t)((round_no - 1) & 1), abort_flag, a.spin_limit));
                        if (!ok) { record_error(err_flag, 4); s_abort = 1; break; }
                    } else {
                        group_sync(bar_id);
                    }
                    {
                        const int col = g0 * 32;
                        uint32_t r[32];
                        const uint32_t taddr = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * acc_cols + col);
                        tmem_ld32(r, taddr);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (g0 + step >= groups) {
                            // this thread's part of the accumulator is in registers: hand the buffer back
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            mbar_arrive(&bar_acc_empty[as]);
                        }
                        float4* dst = reinterpret_cast<float4*>(staging + (size_t)sb * kStagingBytes + (size_t)row * 128);
                        // which output this slab belongs to, and its first column there
                        // (a partial tile bound for the workspace keeps the stacked column order of the accumulator)
                        const bool to_ws = kSplit && a.ws_mode;
                        const bool second = !to_ws && a.split_col > 0 && nbase + col >= a.split_col;
                        const int lcol = second ? nbase + col - a.split_col : nbase + col;
                        const int kout = to_ws ? a.ws_cols : (second ? a.K - a.split_col : (a.split_col > 0 ? a.K1 : a.K));
                        const bool fast = a.bias_mode != 1 && lcol + 32 <= kout;
                        if (fast) {
                            // every column is a real channel and the bias is per column:
                            // two instructions per value, bias read as 128-bit vectors;
                            // all values first, then the eight 128-bit stores back to back
                            // (measured faster than storing as they come)
                            const float4* bv = reinterpret_cast<const float4*>(my_bias + col);
                            float4 o[8];
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) {
                                const float4 bb = bv[c4];
                                float4 v;
                                v.x = fmaf(a.alpha, __uint_as_float(r[c4 * 4 + 0]), bb.x);
                                v.y = fmaf(a.alpha, __uint_as_float(r[c4 * 4 + 1]), bb.y);
                                v.z = fmaf(a.alpha, __uint_as_float(r[c4 * 4 + 2]), bb.z);
                                v.w = fmaf(a.alpha, __uint_as_float(r[c4 * 4 + 3]), bb.w);
                                if constexpr (kForm == kWholeRes) {
                                    const float4 rr = dst[c4 ^ (row & 7)];
                                    v.x += rr.x; v.y += rr.y; v.z += rr.z; v.w += rr.w;
                                }
                                if (a.act == OGLE_ACT_RELU) {
                                    v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
                                } else if (a.act == OGLE_ACT_CLIP) {
                                    v.x = fminf(fmaxf(v.x, a.lo), a.hi); v.y = fminf(fmaxf(v.y, a.lo), a.hi);
                                    v.z = fminf(fmaxf(v.z, a.lo), a.hi); v.w = fminf(fmaxf(v.w, a.lo), a.hi);
                                }
                                o[c4] = v;
                            }
                            // 128-byte swizzle: 16-byte chunk index XOR (row mod 8)
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) dst[c4 ^ (row & 7)] = o[c4];
                        } else {
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) {
                                float v[4];
                                float rr[4] = {0.f, 0.f, 0.f, 0.f};
                                if constexpr (kForm == kWholeRes) {
                                    const float4 q4 = dst[c4 ^ (row & 7)];
                                    rr[0] = q4.x; rr[1] = q4.y; rr[2] = q4.z; rr[3] = q4.w;
                                }
#pragma unroll
                                for (int l = 0; l < 4; ++l) {
                                    const int n = lcol + c4 * 4 + l;
                                    float acc = a.alpha * __uint_as_float(r[c4 * 4 + l]);
                                    if (n < kout) {
                                        if (a.bias_mode == 2) acc += my_bias[col + c4 * 4 + l];
                                        else if (a.bias_mode == 1) acc = fmaf(a.beta, bias[pix * a.ldc + n], acc);
                                        if (kForm == kWholeRes) acc += rr[l];
                                        acc = apply_act(acc, a.act, a.lo, a.hi);
                                    } else {
                                        acc = 0.f;         // padded lanes stay zero
                                    }
                                    v[l] = acc;
                                }
                                dst[c4 ^ (row & 7)] = make_float4(v[0], v[1], v[2], v[3]);
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    group_sync(bar_id);
                    if (t == 0) {
                        {
                            const uint32_t src = base + my_staging + (uint32_t)sb * (uint32_t)kStagingBytes;
                            int col = nbase + g0 * 32;
                            const CUtensorMap* my = &tmY;
                            const bool to_ws = kSplit && a.ws_mode;
                            if (!to_ws && a.split_col > 0 && col >= a.split_col) { col -= a.split_col; my = &tmY2; }
                            if (to_ws) {
                                // slice ks of the scratch tensor; the reduce kernel adds the slices
                                if (a.flat) tma_store_4d(&tmY, src, col, tc_.w0 + wi.ks * a.ws_slice, 0, 0);
                                else tma_store_4d(&tmY, src, col, tc_.w0, tc_.h0, tc_.n0 + wi.ks * a.ws_slice);
                            } else if (kSplit) {
                                if (a.flat) tma_reduce_add_4d(my, src, col, tc_.w0, 0, 0);
                                else tma_reduce_add_4d(my, src, col, tc_.w0, tc_.h0, tc_.n0);
                            } else if (a.flat) {
                                tma_store_4d(my, src, col, tc_.w0, 0, 0);
                            } else {
                                tma_store_4d(my, src, col, tc_.w0, tc_.h0, tc_.n0);
                            }
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            }
            // (an aborting block waits for the copy it has asked for)
            if (!ok && res_copies > 0) mbar_wait(&bar_res[eg], (uint32_t)((res_copies - 1) & 1));
            // the staging slabs must outlive the stores that read them (their writes to global memory are
            // complete, like every write of the grid, when the grid is)
            if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
    }

    // ------------------------------------------------------------------ teardown
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_abort) {
        // Some role gave up. Every role has left its loop (a role that was not waiting finished
        // what it had issued), but multiplies and operand copies may still be in flight - also where the
        // issuer itself came to its end and only an epilogue gave up -, and tensor memory may not be freed
        // nor the block retire before they are done. The thread that issued the multiplies (the one that is
        // elected each time) waits for them. A ring stage's
        // barrier completes when BOTH producers have announced their copy and the bytes are in;
        // the producers may have stopped up to a ring apart, so first supply the announcement
        // the other one never made, then wait (full bound) for the last ring of stages.
        if (warp == 1 && elect_one()) {
            umma_commit(&bar_drain);
            mbar_wait(&bar_drain, 0u);
        }
        if (threadIdx.x == 0) {
            const int na = s_issued[0], nb = s_issued[1];
            const int lo = na < nb ? na : nb, hi = na < nb ? nb : na;
            for (int i = lo; i < hi; ++i) mbar_arrive(&bar_full[i % a.stages]);
            for (int i = (hi > a.stages ? hi - a.stages : 0); i < hi; ++i)
                mbar_wait(&bar_full[i % a.stages], (uint32_t)((i / a.stages) & 1));
        }
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"((uint32_t)a.tmem_cols));
    }
    if constexpr (kForm == kCluster) {
        // Every block of the cluster gets here, also one that gave up (its sums are then meaningless, and the status
        // word says so); none leaves while another may still read its partial tile.
        __syncwarp();
        cluster_sync();
        cluster_reduce(a, base, s_bias[0], bias);
        // (what was read has been used, and nobody reads what was written: no order to be kept, and no wait for the stores)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
}

int num_sms() {
    static thread_local int sms = 0, sms_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (sms_device != dev) {
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return kNumSMs;
        sms = prop.multiProcessorCount;
        sms_device = dev;
    }
    return sms;
}

}  // namespace

// [k]: how many clusters of k blocks can be resident at once (a block has its SM to itself): the GPU's own answer,
// asked once per thread and device. 0 = such clusters cannot run.
const int* tc_cluster_capacity() {
    static thread_local int device = -1, known[9];
    static const int none[9] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return none;
    if (device != dev) {
        if (cudaFuncSetAttribute(conv_tc2_kernel<kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess) {
            (void)cudaGetLastError();
            return none;
        }
        for (int b = 2; b <= 8; ++b) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)b);
            cfg.blockDim = dim3(kThreads2);
            cfg.dynamicSmemBytes = kTcSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)b; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&known[b], conv_tc2_kernel<kCluster>, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                known[b] = 0;
            }
        }
        device = dev;
    }
    return known;
}

int launch_tc_v2(TcArgs& t, const CUtensorMap& mA, const CUtensorMap& mBhi, const CUtensorMap& mBlo,
                 const CUtensorMap& mY, const CUtensorMap& mY2, long m_tiles, const float* bias, int* err_flag,
                 cudaStream_t s) {
    if (t.BN % 32 || t.BN > 256) return OGLE_ERR_UNSUPPORTED;
    // accumulators: two, or four when they fit (half of) the 512 columns of tensor memory - the multiplies
    // of a tile can then start while the epilogues of the two tiles before it still drain theirs
    const int b_rows = t.BN * (t.taps ? 3 : 1), acc_cols = b_rows;
    // Split mode: the A operands of both passes go through tensor memory where two stages or more of them fit beside
    // the accumulators (tiles of up to 192 columns).
    // (In the gather form too, for three input channels.)
    const bool ta_form = t.passes == 3 && (!t.gather || t.g_C == 3);
    t.n_acc = 4 * acc_cols <= (ta_form ? 256 : 512) ? 4 : 2;
    static const bool ta_off = [] { const char* e = getenv("OGLE_TC_TA"); return e && e[0] == '0'; }();
    // Taps side by side, 64 channels a tile: with both in tensor memory the ring would have two stages; the BF16 one alone
    // leaves room for four, and shared memory for three.
    const int ta_cols = t.taps && t.n_acc * acc_cols > 256 ? 32 : 64;
    const int ta_stages = (512 - t.n_acc * acc_cols) / ta_cols;
    t.ta = ta_form && !ta_off && ta_stages >= 2 ? (ta_cols == 32 ? 2 : 1) : 0;
    if (!t.ta) t.n_acc = 4 * acc_cols <= 512 ? 4 : 2;
    size_t stage = (size_t)(t.ta && t.gather ? 0 : (t.passes == 3 && !t.ta ? 2 : 1)) * kABytes + (size_t)(t.passes == 3 ? 2 : 1) * b_rows * 128 +
                         (t.gather ? (size_t)t.g_bytes : 0);
    // Shared memory is split between the operand ring and the epilogue's staging slabs
    // (128 rows x 32 columns each). Preference: two epilogue groups with two slabs each;
    // give slabs back to the ring while that buys another stage and the ring is shallow.
    const size_t kBudget = kTcSmem;
    const int chunks = (t.taps ? 1 : t.kernel) * t.kernel * t.chunks_per_tap;
    t.xf_groups = (t.passes == 3 || t.gather) ? 2 : 1;   // both operand-split groups work on each chunk
    t.epi_groups = 2;
    t.epi_slabs = 2;
    if (t.passes == 3 && chunks >= 8) {
        // long reductions: the epilogue is rare, the ring needs the room. What it leaves over (where tensor memory bounds
        // it, or the last stage does not fit) goes to the epilogue: a tile of 128 columns and eight chunks takes as
        // long to store by one group as to multiply
        t.epi_groups = 1;
        t.epi_slabs = 1;
        int ring = (int)((kBudget - kStagingBytes) / stage);
        if (ring > kMaxStages) ring = kMaxStages;
        if (t.ta && ring > ta_stages) ring = ta_stages;
        const size_t over = kBudget - (size_t)ring * stage;
        if (over >= 2 * (size_t)kStagingBytes) t.epi_groups = 2;
        if (over >= 4 * (size_t)kStagingBytes) t.epi_slabs = 2;
    } else {
        auto stages_with = [&](int groups, int slabs) { return (int)((kBudget - (size_t)groups * slabs * kStagingBytes) / stage); };
        // (measured: the bandwidth-bound pointwise layers want the second slab more than a
        // fourth stage; reductions of 16+ chunks want the stage)
        const int shallow = chunks >= 16 ? 4 : 3;
        if (stages_with(2, 2) < shallow && stages_with(2, 1) > stages_with(2, 2)) t.epi_slabs = 1;
        if (stages_with(t.epi_groups, t.epi_slabs) < 2) { t.epi_groups = 1; t.epi_slabs = 1; }
    }
    static const char* env_xf = getenv("OGLE_TC_XF_GROUPS");
    static const char* env_groups = getenv("OGLE_TC_EPI_GROUPS");
    static const char* env_slabs = getenv("OGLE_TC_EPI_SLABS");
    if (const char* e = env_xf) t.xf_groups = ((t.passes == 3 || t.gather) && e[0] == '2') ? 2 : 1;
    if (t.gather) t.xf_groups = 2;        // the gather code is laid out for 256 threads
    if (const char* e = env_groups) t.epi_groups = e[0] == '1' ? 1 : 2;
    if (const char* e = env_slabs) t.epi_slabs = e[0] == '1' ? 1 : 2;
    if (t.cluster) t.epi_slabs = 0;       // partial tiles go where the operand ring was
    size_t staging = (size_t)t.epi_groups * t.epi_slabs * kStagingBytes;
    const size_t budget = kBudget - staging;
    int stages = (int)(budget / stage);
    if (stages > kMaxStages) stages = kMaxStages;
    if (t.ta && stages > ta_stages) stages = ta_stages;
    // Filters and windows kept where they fit; two windows are enough while the ring is at most a stage longer than a tile's
    // reduction, and one filter tile serves all.
    const size_t kept = (size_t)chunks * 2 * b_rows * 128 + 2 * (size_t)t.g_bytes;
    const int kept_stages = ta_stages < chunks + 1 ? ta_stages : chunks + 1;
    const bool keep = t.gather && t.ta && !t.res && t.n_tiles == 1 && t.split_k <= 1 && chunks >= 2 && kept_stages >= 2 &&
                      kept + 4 * (size_t)kStagingBytes <= kBudget;
    if (keep) {
        t.epi_groups = 2;
        t.epi_slabs = 2;
        staging = 4 * (size_t)kStagingBytes + kept;
        stage = 0;
        stages = kept_stages < kMaxStages ? kept_stages : kMaxStages;
    }
    if (stages < 2) return OGLE_ERR_UNSUPPORTED;
    t.stages = stages;
    int cols = 32;
    while (cols < t.n_acc * acc_cols + (t.ta ? t.stages * ta_cols : 0)) cols <<= 1;
    t.tmem_cols = cols;
    const long total = m_tiles * t.n_tiles;
    if (total <= 0 || total > 0x7fffffffL) return OGLE_ERR_UNSUPPORTED;
    t.total_tiles = (int)total;
    t.spin_limit = role_wait_limit();
    if (t.split_k < 1) t.split_k = 1;
    if (total * t.split_k > 0x7fffffffL) return OGLE_ERR_UNSUPPORTED;
    t.total_work = (int)(total * t.split_k);
    t.chunks_per_split = (chunks + t.split_k - 1) / t.split_k;
    if (t.cluster && (t.split_k < 2 || t.split_k > 8 || (size_t)t.BN * 512 > kBudget)) return OGLE_ERR_UNSUPPORTED;
    // Always the whole budget, also when the layout needs less: a block then has its SM to
    // itself whatever else is running, so its tensor-memory allocation can never wait for
    // another resident block's columns.
    const size_t smem = kBudget;
    if (stage * stages + staging > smem) return OGLE_ERR_UNSUPPORTED;
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        cudaError_t e = cudaFuncSetAttribute(conv_tc2_kernel<kWhole>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kRanges>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kKept>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kWholeRes>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kTapsRes>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_tc2_kernel<kTaps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    const int sms = num_sms();
    // A tile of 128 x 256 takes one group 8 us after the last multiply, which launches of a round or two feel; and a wide
    // tile's buffer is handed back sooner by two. Many rounds of one or two chunks are bound by HBM and keep a better
    // rhythm with whole tiles per group: 5.76 M pixels 32 -> 64, split mode 443 against 454 us, one pass 414 against 436;
    // 1.44 M 64 -> 128: 195 against 201, 184 against 188. At four chunks 128 -> 256 (0.37 M) it is 182-189 against 166.
    t.epi_share = t.total_work <= 4 * sms || chunks > 2 ? 1 : 0;
    const unsigned grid = (unsigned)(t.total_work < sms ? t.total_work : sms);
    const bool overlapped = overlapped_launches_enabled(t.overlapped);
    note_contraction(t.cluster ? 3 : (t.split_k > 1 ? 2 : (t.taps ? 6 : (keep ? 7 : 1))), t.split_k, t.BN, overlapped);
    if (t.cluster) {
        // every block one work item; the blocks of a tile are consecutive, and a cluster
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)t.total_work);
        cfg.blockDim = dim3(kThreads2);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = overlapped ? 1 : 0;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = (unsigned)t.split_k; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        cudaError_t e = cudaLaunchKernelEx(&cfg, conv_tc2_kernel<kCluster>, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
        if (e != cudaSuccess) { set_last_error(e); (void)cudaGetLastError(); return OGLE_ERR_CUDA; }
        return finish_launch();
    }
    if (t.split_k > 1)
        launch_overlapped_if(overlapped, conv_tc2_kernel<kRanges>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    else if (keep)
        launch_overlapped_if(overlapped, conv_tc2_kernel<kKept>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    else if (t.taps && t.res)
        launch_overlapped_if(overlapped, conv_tc2_kernel<kTapsRes>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    else if (t.taps)
        launch_overlapped_if(overlapped, conv_tc2_kernel<kTaps>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    else if (t.res)
        launch_overlapped_if(overlapped, conv_tc2_kernel<kWholeRes>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    else
        launch_overlapped_if(overlapped, conv_tc2_kernel<kWhole>, dim3(grid), dim3(kThreads2), smem, s, mA, mBhi, mBlo, mY, mY2, bias, t, err_flag);
    return finish_launch();
}

}  // namespace ogle
