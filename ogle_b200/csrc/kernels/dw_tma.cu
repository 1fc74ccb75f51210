// Depthwise 3x3 and 5x5 convolution (stride 1 or 2, any channel count) as a
// persistent, TMA-fed, HBM-bound kernel.
//
// One block per SM slot walks a list of tiles. A tile is th x tw output pixels of
// one image for a slab of 32 channels (16 where 32 would leave much of the last slab
// empty; channels past the tensor arrive as zeros and are not stored), chosen by an estimate
// (choose_shape). Its input window, halo included, is ONE TMA box
// [IH rows][IW cols][channels of the slab]; pixels outside the image arrive as zeros,
// which is the convolution's padding. A ring of two to four shared-memory stages: while
// the block computes tile i from one stage, the TMA engine fills the others with the next tiles, so
// the only HBM traffic is the input read once (halo rows come from L2) and the
// output written once, both as 128-byte runs.
// A thread owns 4 channels (one float4) of one output column and slides the window
// down RPG output rows of it; 8 lanes cover one pixel's 128 bytes, so
// shared-memory reads are conflict-free (slabs of 16 at stride 2 are not: two wavefronts).
// The 32 pixel slots of a block (64 with slabs of 16) are split into row groups of tw.
// Widths that are no multiple of 32 channels, and 5x5 windows, ran on kernels that fetch every
// tap through L1: 16 x 75 x 75 x 144 channels took 39 us there and 23.5 us here (16 us floor).
#include <cmath>
#include <cstdlib>

#include "tc_common.cuh"
#include "tma_host.h"

namespace ogle {
namespace {

using namespace tc;

constexpr int kDwSmemMax = 110 * 1024;   // two blocks per SM
constexpr int kDwMaxStages = 4;

struct DwTiles {
    int tiles_x, tiles_y, cblocks;   // tile grid per image, 32-channel slabs
    int tw, th, row_groups;          // tile shape: th = RPG * row_groups
    int iw, ih;                      // input window of a tile, halo included
    int stages;                      // tiles in flight per block (2..4)
    long total;
};

// KS: window size. CB: float4s of a channel slab (8 = 32 channels, 4 = 16). A 5x5 window keeps its 25 taps
// in registers too (100 of them), which leaves one block per SM: eight warps with 4-row accumulators are
// enough to keep the copies ahead of the multiplies. RAGGED: the last slab reaches past the channels; widths that
// fill their slabs carry none of its checks (stride 1: 17.6 us, 19.2 with them, at 6 x 64 x 70 x 384).
template <int KS, int S, int RPG, int CB, bool RAGGED>
__global__ void __launch_bounds__(256, KS == 3 ? 2 : 1)
dw_tma_kernel(const __grid_constant__ CUtensorMap tmX, const float4* __restrict__ w, const float* __restrict__ bias,
                 float4* __restrict__ y, const ConvArgs a, const DwTiles tl, int* err_flag) {
    constexpr int ROWS_IN = (RPG - 1) * S + KS;
    const int TW = tl.tw, TH = tl.th, IW = tl.iw;
    const uint32_t kTileBytes = (uint32_t)(tl.ih * tl.iw * CB * 16);
    const uint32_t pitch = (kTileBytes + 127u) & ~127u;      // TMA destinations are 128-byte aligned
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kDwMaxStages];

    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
    const float4* stage0 = reinterpret_cast<const float4*>(smem_raw + (base - smem_u32(smem_raw)));

    const int out_q = a.Ks >> 2, off_q = a.koff >> 2;
    const int c = threadIdx.x % CB;
    const int slot = threadIdx.x / CB;
    const int col = slot % TW, rg = slot / TW;
    const bool active = rg < tl.row_groups;        // slots past tw * row_groups idle

    grid_dependency_trigger();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kDwMaxStages; ++i) mbar_init(&bar_full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    grid_dependency_wait();         // nothing from global memory before this point
    __syncthreads();

    // tile id -> (channel slab fastest, then x, y, image): neighbouring blocks share halo rows in L2
    // (tile counts fit 32 bits: the launch refuses more)
    auto issue = [&](long tile, int stage) {
        unsigned t = (unsigned)tile;
        const int cb = (int)(t % (unsigned)tl.cblocks); t /= (unsigned)tl.cblocks;
        const int tx = (int)(t % (unsigned)tl.tiles_x); t /= (unsigned)tl.tiles_x;
        const int ty = (int)(t % (unsigned)tl.tiles_y); t /= (unsigned)tl.tiles_y;
        const int n = (int)t;
        mbar_expect_tx(&bar_full[stage], kTileBytes);
        tma_load_4d(base + (uint32_t)stage * pitch, &tmX, &bar_full[stage], cb * CB * 4, tx * TW * S - a.pad,
                    ty * TH * S - a.pad, n);
    };

    // prologue: fill all but one stage; each iteration then tops the ring up before computing
    const int nst = tl.stages;
    long issued = 0;                               // tiles whose copy was started (thread 0 only)
    if (threadIdx.x == 0)
        for (int k = 0; k < nst - 1; ++k)
            if ((long)blockIdx.x + (long)k * gridDim.x < tl.total) { issue((long)blockIdx.x + (long)k * gridDim.x, k); ++issued; }
    long it = 0;
    int stage = 0;
    uint32_t phase = 0;
    float4 wk[KS * KS];
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
    int loaded_cb = -1;
    for (long tile = blockIdx.x; tile < tl.total; tile += gridDim.x, ++it) {
        // the stage refilled here was last read by tile it-1, which every thread finished
        // before the __syncthreads at the bottom of the previous iteration
        if (threadIdx.x == 0) {
            const long ahead = tile + (long)(nst - 1) * gridDim.x;
            if (ahead < tl.total) { issue(ahead, stage == 0 ? nst - 1 : stage - 1); ++issued; }
        }
        unsigned t = (unsigned)tile;
        const int cb = (int)(t % (unsigned)tl.cblocks); t /= (unsigned)tl.cblocks;
        const int tx = (int)(t % (unsigned)tl.tiles_x); t /= (unsigned)tl.tiles_x;
        const int ty = (int)(t % (unsigned)tl.tiles_y); t /= (unsigned)tl.tiles_y;
        const int n = (int)t;
        const int cq = cb * CB + c;
        // filter taps and bias of this channel slab: when the grid is a multiple of the slab
        // count every tile of a block has the same slab, and they are loaded once
        if (cb != loaded_cb) {
#pragma unroll
            for (int k = 0; k < KS * KS; ++k) wk[k] = !RAGGED || cq < (a.Kp >> 2) ? w[k * (a.Kp >> 2) + cq] : make_float4(0.f, 0.f, 0.f, 0.f);
            bv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!RAGGED) {
                if (a.has_bias) bv = make_float4(bias[cq * 4], bias[cq * 4 + 1], bias[cq * 4 + 2], bias[cq * 4 + 3]);
            } else if (a.has_bias) {                   // bias holds exactly K floats
                if (cq * 4 + 0 < a.K) bv.x = bias[cq * 4 + 0];
                if (cq * 4 + 1 < a.K) bv.y = bias[cq * 4 + 1];
                if (cq * 4 + 2 < a.K) bv.z = bias[cq * 4 + 2];
                if (cq * 4 + 3 < a.K) bv.w = bias[cq * 4 + 3];
            }
            loaded_cb = cb;
        }

        if (!mbar_wait(&bar_full[stage], phase)) {
            if (threadIdx.x == 0) {
                record_error(err_flag, 6);
                // let the later copies already in flight land (bounded) before the block retires
                for (long j = it + 1; j < issued; ++j) mbar_wait(&bar_full[j % nst], (uint32_t)((j / nst) & 1));
            }
            break;   // uniform: every thread waits on the same barrier with the same bound
        }
        const float4* tile_s = stage0 + (size_t)stage * (pitch / 16);
        if (active) {
        float4 acc[RPG];
#pragma unroll
        for (int r = 0; r < RPG; ++r) acc[r] = bv;
        const int row0 = rg * RPG * S;
#pragma unroll
        for (int r = 0; r < ROWS_IN; ++r) {
            float4 v[KS];
#pragma unroll
            for (int kx = 0; kx < KS; ++kx) v[kx] = tile_s[((row0 + r) * IW + col * S + kx) * CB + c];
#pragma unroll
            for (int o = 0; o < RPG; ++o) {
                const int ky = r - o * S;
                if (ky < 0 || ky >= KS) continue;
#pragma unroll
                for (int kx = 0; kx < KS; ++kx) {
                    const float4 f = wk[ky * KS + kx];
                    acc[o].x = fmaf(f.x, v[kx].x, acc[o].x);
                    acc[o].y = fmaf(f.y, v[kx].y, acc[o].y);
                    acc[o].z = fmaf(f.z, v[kx].z, acc[o].z);
                    acc[o].w = fmaf(f.w, v[kx].w, acc[o].w);
                }
            }
        }
        const int ox = tx * TW + col;
        if (ox < a.Wo && (!RAGGED || cq < (a.Kp >> 2))) {
#pragma unroll
            for (int o = 0; o < RPG; ++o) {
                const int oy = ty * TH + rg * RPG + o;
                if (oy >= a.Ho) continue;
                float4 r = apply_act4(acc[o], a.act, a.lo, a.hi);
                if (RAGGED && cq * 4 + 4 > a.K) {                // lanes past K stay zero
                    if (cq * 4 + 1 >= a.K) r.y = 0.f;
                    if (cq * 4 + 2 >= a.K) r.z = 0.f;
                    r.w = 0.f;
                }
                y[(((long)n * a.Ho + oy) * a.Wo + ox) * out_q + off_q + cq] = r;
            }
        }
        }
        __syncthreads();
        if (++stage == nst) { stage = 0; phase ^= 1u; }
    }
}

template <int KS, int S, int RPG, int CB, bool RAGGED>
int launch_kernel(const ConvArgs& a, const DwTiles& shape, const float* x, const float* w, const float* bias, float* y, cudaStream_t s) {
    CUtensorMap mX;
    const cuuint64_t dims[4] = {(cuuint64_t)a.Kp, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.N};
    const cuuint64_t str[3] = {(cuuint64_t)a.Cs * 4, (cuuint64_t)a.Cs * 4 * a.W, (cuuint64_t)a.Cs * 4 * a.W * a.H};
    const cuuint32_t box[4] = {CB * 4, (cuuint32_t)shape.iw, (cuuint32_t)shape.ih, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    if (!make_map_sw(CU_TENSOR_MAP_SWIZZLE_NONE, &mX, x, 4, dims, str, box, es)) return OGLE_ERR_CUDA;
    DwTiles tl = shape;
    tl.tiles_x = (a.Wo + tl.tw - 1) / tl.tw;
    tl.tiles_y = (a.Ho + tl.th - 1) / tl.th;
    tl.cblocks = (a.Kp + CB * 4 - 1) / (CB * 4);
    tl.total = (long)tl.tiles_x * tl.tiles_y * tl.cblocks * a.N;
    const size_t smem = (size_t)tl.stages * (((size_t)tl.ih * tl.iw * CB * 16 + 127) / 128 * 128) + 128;
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {
        cudaError_t e = cudaFuncSetAttribute(dw_tma_kernel<KS, S, RPG, CB, RAGGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDwSmemMax);
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        attr_device = dev;
    }
    if (tl.total > 0x7fffffffL) return OGLE_ERR_UNSUPPORTED;
    long blocks = (long)kNumSMs * (KS == 3 ? 2 : 1);
    // a multiple of the channel-slab count: block b then always works on slab b % cblocks
    if (tl.cblocks <= blocks) blocks -= blocks % tl.cblocks;
    if (blocks > tl.total) blocks = tl.total;
    launch_overlapped(dw_tma_kernel<KS, S, RPG, CB, RAGGED>, dim3((unsigned)blocks), dim3(256), smem, s, mX, reinterpret_cast<const float4*>(w),
                      bias, reinterpret_cast<float4*>(y), a, tl, error_flag_ptr());
    return finish_launch();
}

template <int KS, int S, int RPG, int CB>
int launch(const ConvArgs& a, const DwTiles& shape, const float* x, const float* w, const float* bias, float* y, cudaStream_t s) {
    return a.K % (CB * 4) ? launch_kernel<KS, S, RPG, CB, true>(a, shape, x, w, bias, y, s)
                          : launch_kernel<KS, S, RPG, CB, false>(a, shape, x, w, bias, y, s);
}

// Float4s of a channel slab: 32 channels, or 16 where slabs of 32 would compute over a sixth more channels than
// slabs of 16 do (a slab's empty lanes cost shared memory and issue slots, not traffic). At stride 2 it is the copies that
// set the pace, by the pixel and not by the byte, and only layers of one slab are better off with a narrow one
// (52 x 132 x 116 x 72: 61 us, 50 with slabs of 32).
int slab_quads(const ConvArgs& a) {
    if (a.stride == 2) return a.Kp <= 16 ? 4 : 8;
    const int full = (a.Kp + 31) / 32 * 32, half = (a.Kp + 15) / 16 * 16;
    return 6 * full <= 7 * half ? 8 : 4;
}

// Whether tiles of th x tw pixels leave room for two stages; t's shape and stages.
bool fit_tile(const ConvArgs& a, int quads, int tw, int rpg, DwTiles* t) {
    const int S = a.stride, KS = a.kernel, groups = 256 / quads / tw, th = rpg * groups;
    const int iw = (tw - 1) * S + KS, ih = (th - 1) * S + KS;
    if (iw > 256 || ih > 256) return false;
    const size_t tile = ((size_t)ih * iw * quads * 16 + 127) / 128 * 128;
    if (2 * tile + 128 > (size_t)kDwSmemMax) return false;
    t->tw = tw; t->th = th; t->row_groups = groups; t->iw = iw; t->ih = ih;
    // as many tiles in flight as fit: HBM latency x bandwidth needs ~90 KB per SM
    const int st = (int)((size_t)(kDwSmemMax - 128) / tile);
    t->stages = st > kDwMaxStages ? kDwMaxStages : st;
    return true;
}

// Output pixels of all tiles of a map, those past its edges included.
double covered(const ConvArgs& a, const DwTiles& t) {
    return (double)((a.Wo + t.tw - 1) / t.tw) * t.tw * ((a.Ho + t.th - 1) / t.th) * t.th;
}

// Estimate of a launch's time (us) at stride 1: rounds of tiles over the resident blocks, of which each takes a fixed
// time, its rows' multiply-adds and its copies, partly beside one another; or the time at the HBM rate, which rings of fewer
// than four stages do not reach.
double stride1_us(const ConvArgs& a, int quads, const DwTiles& t, int rows) {
    const int slab = quads * 4, cblocks = (a.Kp + slab - 1) / slab;
    int resident = kNumSMs * (a.kernel == 3 ? 2 : 1);
    if (cblocks <= resident) resident -= resident % cblocks;
    const double hbm = 8.0 * a.N * a.Ho * a.Wo * a.Kp / 6.0e6;
    const double tiles = (double)((a.Wo + t.tw - 1) / t.tw) * ((a.Ho + t.th - 1) / t.th) * cblocks * a.N;
    const double rounds = ceil(tiles / resident);
    const double compute = 1.47 + 0.088 * rows * (a.kernel == 3 ? 1.0 : 3.8), copy = 0.0023 * t.ih * t.iw * quads / 8;
    const double work = rounds * (compute > copy ? compute + 0.37 * copy : copy + 0.37 * compute);
    const double memory = t.stages < 4 ? 1.24 * hbm : hbm;
    return work > memory ? work + 0.33 * memory : memory + 0.33 * work;
}

// Tile shape at stride 1: equal parts of the map's width, or one of a few widths that fill a block's pixel slots, and the
// rows a thread computes, by the estimate. Fitted to 60 layers, 4 us to 170, with every width and row count timed: 5 % faster
// on average than choose_shape_by_rows, 3 % off the best; 16 x 75 x 75 x 144 25.2 -> 23.5 us (tiles of 15 keep 30 of 32
// slots busy where 32, 32 and 11 kept 25), 64 x 75 x 75 x 128 64 -> 59, 22 x 83 x 99 x 345 101 -> 86.
int choose_shape_stride1(const ConvArgs& a, int quads, DwTiles* t) {
    static const int kRows3[] = {10, 8, 7, 5, 4, 2}, kRows5[] = {4, 2};
    const int* rows = a.kernel == 5 ? kRows5 : kRows3;
    const int nrows = a.kernel == 5 ? 2 : 6;
    const char* env_tw = getenv("OGLE_DW_TW");
    const char* env_rows = getenv("OGLE_DW_RPG");
    const int force_rows = env_rows ? atoi(env_rows) : 0;
    int best = 0;
    double best_us = 0.0;
    auto consider = [&](int tw) {
        for (int i = 0; i < nrows; ++i) {
            DwTiles s;
            if ((force_rows && rows[i] != force_rows) || !fit_tile(a, quads, tw, rows[i], &s)) continue;
            const double us = stride1_us(a, quads, s, rows[i]);
            if (!best || us < best_us) { best = rows[i]; best_us = us; *t = s; }
        }
    };
    if (env_tw && atoi(env_tw) >= 1 && atoi(env_tw) <= 32) {
        consider(atoi(env_tw) < a.Wo ? atoi(env_tw) : a.Wo);
        return best;
    }
    for (int tw = a.Wo < 32 ? a.Wo : 32; tw >= 5; --tw) {
        const int parts = (a.Wo + tw - 1) / tw;
        if ((a.Wo + parts - 1) / parts == tw || tw == 8 || tw == 10 || tw == 16 || tw == 32) consider(tw);
    }
    return best;
}

// Tile shape at stride 2, and of large tensors: full-width tiles when the map is at most 16 wide, equal parts up to 48, else
// 32 or, at stride 2, 16 pixels; the rows per thread (one of the compiled RPG values) that leaves the fewest idle output rows.
// Returns the chosen RPG, or 0 when no shape fits two stages in kDwSmemMax.
int choose_shape_by_rows(const ConvArgs& a, int quads, DwTiles* t) {
    const int S = a.stride, KS = a.kernel;
    int tw = a.Wo <= 32 ? a.Wo : (S == 1 ? 32 : 16);
    // Widths that would leave many of the 32 pixel slots of a block idle are cut into equal parts
    // (measured at batch 256: 19 -> 2 x 10 is 6 % faster, 38 -> 3 x 13 is 18 % faster than 32 + 6)
    if (a.Wo >= 17 && a.Wo <= 32) tw = (a.Wo + 1) / 2;
    else if (a.Wo > 32 && a.Wo <= 48) tw = (a.Wo + 2) / 3;
    if (const char* e = getenv("OGLE_DW_TW")) { const int v = atoi(e); if (v >= 1 && v <= 32) tw = v < a.Wo ? v : a.Wo; }
    const int force_rpg = getenv("OGLE_DW_RPG") ? atoi(getenv("OGLE_DW_RPG")) : 0;
    static const int kRpg1[] = {10, 8, 7, 5, 4, 2}, kRpg2[] = {7, 5, 4, 2}, kRpg5[] = {4, 2};
    const int* cand = KS == 5 ? kRpg5 : (S == 1 ? kRpg1 : kRpg2);
    const int ncand = KS == 5 ? 2 : (S == 1 ? 6 : 4);
    int best = 0;
    long best_cost = -1;
    for (int i = 0; i < ncand; ++i) {
        const int rpg = cand[i];
        DwTiles s;
        if ((force_rpg && rpg != force_rpg) || !fit_tile(a, quads, tw, rpg, &s)) continue;
        const long tiles_y = (a.Ho + s.th - 1) / s.th;
        // rows computed (idle ones included) plus a charge per tile for its halo rows
        long cost = tiles_y * (s.th * S + KS - 1);
        // a single channel slab: neighbouring blocks then work on neighbouring
        // tiles of the same rows, and a ring of three shallower tiles measured 20 % faster
        // than two deep ones on the 150x150 map
        if (a.Kp <= quads * 4 && s.stages < 3) cost *= 2;
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = rpg; *t = s; }
    }
    return best;
}

// The shape for a layer, and the rows a thread computes (0: none fits). Those of the last layers are kept, by their sizes:
// to weigh some eighty shapes takes the host 0.45 us. There is room for a few networks' layers: a network runs its layers in
// turn, and fewer places than it has (eight, of MobileNet's nine) would all have changed hands when they come round again.
// A layer lies in one of four places.
int choose_shape(const ConvArgs& a, DwTiles* t) {
    struct Known { int N, H, W, Kp, K, kernel, stride, pad, rows; DwTiles t; };
    constexpr int kKnown = 64, kPlaces = 4;
    static thread_local Known known[kKnown];
    static thread_local unsigned next = 0;
    const bool forced = getenv("OGLE_DW_TW") || getenv("OGLE_DW_RPG");
    unsigned at = 0;
    for (int v : {a.N, a.H, a.W, a.K, a.kernel, a.stride, a.pad}) at = (at ^ (unsigned)v) * 2654435761u;
    at >>= 26;                       // (the upper six bits)
    for (unsigned i = 0; !forced && i < kPlaces; ++i) {
        const Known& k = known[(at + i) % kKnown];
        if (k.kernel == a.kernel && k.stride == a.stride && k.pad == a.pad && k.N == a.N && k.H == a.H && k.W == a.W && k.Kp == a.Kp && k.K == a.K) {
            *t = k.t;
            return k.rows;
        }
    }
    const int quads = slab_quads(a);
    // Tensors that do not stay in L2 are bound by HBM, by what the estimate does not see (256 x 38 x 38 x 256: 127 us in
    // parts of 13, 146 in what it takes), unless tiles of 32 hang far over the map's edge (27 x 127 x 70 x 160 56 -> 52).
    int rows = choose_shape_by_rows(a, quads, t);
    const bool large = 8.0 * a.N * a.Ho * a.Wo * a.Kp > 160e6;
    if (a.stride == 1 && !(rows && large && (double)a.Wo * a.Ho >= 0.72 * covered(a, *t))) {
        // Where the two are estimated alike, and this one neither hangs less over the map's edge nor keeps as many of a block's
        // pixel slots busy, it is not the better one (12 x 9 x 45 x 832 in parts of 15 8.3 us, of 23, estimated 1 % better, 9.5;
        // 10 x 41 x 27 x 807 of 14 15.4, of 27 17.5). Of 360 layers ten are 5 to 13 % slower than by the other rule, the
        // geometric mean of all is 0.91.
        DwTiles other;
        const int other_rows = choose_shape_stride1(a, quads, &other);
        if (!rows || (other_rows && (covered(a, other) <= 0.97 * covered(a, *t) || other.tw * other.row_groups >= t->tw * t->row_groups ||
                                     stride1_us(a, quads, other, other_rows) < 0.984 * stride1_us(a, quads, *t, rows)))) {
            rows = other_rows;
            *t = other;
        }
    }
    if (forced) return rows;
    unsigned place = at + next++ % kPlaces;
    for (unsigned i = 0; i < kPlaces; ++i)
        if (!known[(at + i) % kKnown].kernel) { place = at + i; break; }          // (a free one)
    known[place % kKnown] = {a.N, a.H, a.W, a.Kp, a.K, a.kernel, a.stride, a.pad, rows, *t};
    return rows;
}

}  // namespace

bool dw_tma_supported(const ConvArgs& a) {
    if (!((a.kernel == 3 || a.kernel == 5) && a.dil == 1 && a.pad <= a.kernel / 2 && (a.stride == 1 || a.stride == 2) &&
          a.C == a.K && a.Wo >= 8 && a.Ho >= 4 && encode_fn() != nullptr))
        return false;
    DwTiles t;
    if (!choose_shape(a, &t)) return false;
    // Widths of whole slabs always. Others at stride 2, where a tile's copies bring two to four times the pixels that it
    // stores: 60 k pixels of halo, padding and slab per us against the register kernel's 1 us and 7 GB/ms of input and
    // output, while those stay in L2 (45 x 71 x 119 x 12: 11.6 us by copies, 6.5; 59 x 20 x 41 x 230 13.6 against 11.5;
    // 44 x 29 x 105 x 228 29.6 against 36).
    const double bytes = 4.0 * a.N * a.Kp * ((double)a.H * a.W + (double)a.Ho * a.Wo);
    if (a.kernel == 5 || a.stride == 1 || a.K % 32 == 0 || bytes > 100e6) return true;
    const int slab = slab_quads(a) * 4;
    const double tiles = (double)((a.Wo + t.tw - 1) / t.tw) * ((a.Ho + t.th - 1) / t.th) * ((a.Kp + slab - 1) / slab) * a.N;
    const double copies_us = tiles * t.iw * t.ih / 60e3, registers_us = 1.0 + bytes / 7e6;
    return copies_us <= (registers_us > 2.7 ? registers_us : 2.7);
}

template <int CB>
static int launch_slab(const ConvArgs& a, const float* x, const float* w, const float* bias, float* y, cudaStream_t s) {
    DwTiles t = {};
    const int rpg = choose_shape(a, &t);
    if (a.kernel == 5) {
        if (a.stride == 1) return rpg == 4 ? launch<5, 1, 4, CB>(a, t, x, w, bias, y, s) : launch<5, 1, 2, CB>(a, t, x, w, bias, y, s);
        return rpg == 4 ? launch<5, 2, 4, CB>(a, t, x, w, bias, y, s) : launch<5, 2, 2, CB>(a, t, x, w, bias, y, s);
    }
    if (a.stride == 1) {
        switch (rpg) {
            case 10: return launch<3, 1, 10, CB>(a, t, x, w, bias, y, s);
            case 8: return launch<3, 1, 8, CB>(a, t, x, w, bias, y, s);
            case 7: return launch<3, 1, 7, CB>(a, t, x, w, bias, y, s);
            case 5: return launch<3, 1, 5, CB>(a, t, x, w, bias, y, s);
            case 4: return launch<3, 1, 4, CB>(a, t, x, w, bias, y, s);
            case 2: return launch<3, 1, 2, CB>(a, t, x, w, bias, y, s);
        }
    } else {
        switch (rpg) {
            case 7: return launch<3, 2, 7, CB>(a, t, x, w, bias, y, s);
            case 5: return launch<3, 2, 5, CB>(a, t, x, w, bias, y, s);
            case 4: return launch<3, 2, 4, CB>(a, t, x, w, bias, y, s);
            case 2: return launch<3, 2, 2, CB>(a, t, x, w, bias, y, s);
        }
    }
    return OGLE_ERR_UNSUPPORTED;
}

int launch_dw_tma(const ConvArgs& a, const float* x, const float* w, const float* bias, float* y, cudaStream_t s) {
    return slab_quads(a) == 8 ? launch_slab<8>(a, x, w, bias, y, s) : launch_slab<4>(a, x, w, bias, y, s);
}

}  // namespace ogle
