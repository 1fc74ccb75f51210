// Host side of the tcgen05 tensor-core path for the dense contractions: conv2d (general
// and pointwise, as implicit GEMM) and gemm. Builds the TMA tensor maps, chooses tile
// shapes and launches the persistent kernel of conv_tc2.cu.
//
//   D[128 x BN] (fp32, in TMEM)  +=  A[128 x 32] * B[BN x 32]^T   per 32-wide reduction chunk
//
// A = activations, fetched by TMA straight from the NHWC4 tensor: one 4-D box per
//     filter tap, [tn images][th rows][tw cols][32 channels], zero-filled outside
//     the image (that is the convolution's padding), traversal stride = conv stride.
// B = filter, pre-packed K-major [out channel][tap][channel] (see FilterLayout).
// Both land in shared memory in the 128-byte swizzle that the UMMA shared-memory
// descriptors name.
//
// Math modes: OGLE_MATH_TF32 issues one tensor-core pass (operands carry 10 mantissa
// bits). OGLE_MATH_TF32X3 recovers fp32-grade accuracy from three products,
// hi*hi + hi*lo + lo*hi (the dropped lo*lo term is 2^-22 relative): hi*hi as a TF32
// pass, the two cross terms as one BF16 pass over K-concatenated operands
// [a_hi | a_lo] x [b_lo | b_hi] (eight mantissa bits are ample for terms that are
// themselves 2^-11 of the result). The filter parts are made when it is packed; the
// activation parts in shared memory while the pipeline runs.
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "few_rows.cuh"
#include "tc_common.cuh"
#include "tma_host.h"

namespace ogle {

int launch_tc_v2(tc::TcArgs& t, const CUtensorMap& mA, const CUtensorMap& mBhi, const CUtensorMap& mBlo,
                 const CUtensorMap& mY, const CUtensorMap& mY2, long m_tiles, const float* bias, int* err_flag,
                 cudaStream_t s);
int launch_tc_t(tc::TcArgs& t, const CUtensorMap& mA, const CUtensorMap& mBhi, const CUtensorMap& mBlo,
                const CUtensorMap& mY, const CUtensorMap& mY2, long m_tiles, const float* bias, int* err_flag,
                cudaStream_t s);
int launch_tc_pair(tc::TcArgs& t, const CUtensorMap& mA, const CUtensorMap& mBhi, const CUtensorMap& mBlo,
                   const CUtensorMap& mY, const CUtensorMap& mY2, long m_tiles, const float* bias, int* err_flag,
                   cudaStream_t s);

int launch_conv_window(const ConvArgs& a, int passes, bool row_tiles, const float* x, const float* w, const float* bias, float* y,
                       const float* residual, int res_ld, cudaStream_t s);

const int* tc_cluster_capacity();      // [k], 2 <= k <= 8: clusters of k blocks that can be resident at once

__device__ int g_tc_error = 0;   // first error seen by any block (0 = none)

int* error_flag_ptr() {
    // per-device address of the status word
    static thread_local int* ptr = nullptr;
    static thread_local int ptr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (ptr_device != dev) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_tc_error) != cudaSuccess) return nullptr;
        ptr = static_cast<int*>(p);
        ptr_device = dev;
    }
    return ptr;
}

namespace {

using namespace tc;

// N tiling of the persistent kernel: multiples of 32 columns (one staging slab each).
// Picks the width that minimises (rounds of one tile per SM) x (time of a tile), with a
// tile's time modelled by its tensor-core instructions: one instruction costs about 100
// cycles up to ~180 columns (bound by the shared-memory fetch of its 128-row A operand)
// and 0.55 cycles per column beyond.
// wide_ties: among widths of equal cost take the wider one even when everything fits in one round - for
// layers whose reduction can be split through scratch, which fills the SMs better than narrow tiles do (a
// narrow tile pays the same instruction floor as a wide one).
void choose_n_tiling_v2(int Kp, long m_tiles, TcArgs* t, int requested = 0, bool wide_ties = false) {
    const int kmax = (Kp + 31) / 32 * 32;
    auto mma = [](int n) { const double c = 0.55 * n; return c < 100.0 ? 100.0 : c; };
    int best_bn = 32;
    double best_cost = -1.0;
    for (int bn = 32; bn <= 256 && bn <= kmax; bn += 32) {
        const int n_tiles = (Kp + bn - 1) / bn;
        // the last tile of an uneven split is narrower; even splits are what the candidates give
        const long tiles = m_tiles * n_tiles;
        const long rounds = (tiles + kNumSMs - 1) / kNumSMs;
        double per_tile;
        per_tile = (t->passes == 3 ? 2.0 : 1.0) * mma(bn);     // split mode: a TF32 and a BF16 instruction per step
        const double cost = (double)rounds * per_tile;
        // equal cost: the wider tile when there are several rounds (fewer passes over A), the
        // narrower one when everything fits in one round (more SMs busy, shorter epilogues)
        if (best_cost < 0 || cost < best_cost || (cost == best_cost && (rounds > 1 || wide_ties))) { best_cost = cost; best_bn = bn; }
    }
    if (requested >= 32 && requested <= 256 && requested % 32 == 0 && requested <= kmax) best_bn = requested;
    t->BN = best_bn;
    t->n_tiles = (Kp + best_bn - 1) / best_bn;
}

// Tile width that the environment forces on layers it fits, 0 = none (experiments).
int forced_width(int Kp) {
    static const int v = [] { const char* e = getenv("OGLE_TC_BN"); return e ? atoi(e) : 0; }();
    return v >= 32 && v <= 256 && v % 32 == 0 && v <= (Kp + 31) / 32 * 32 ? v : 0;
}

// Two-SM form (conv_tc2_pair.cu): 0 = the built-in rule, 1 = never, 2 = wherever it can run.
int pair_mode_override() {
    static const int v = [] { const char* e = getenv("OGLE_TC_PAIR"); return e ? (e[0] == '0' ? 1 : (e[0] == '1' ? 2 : 0)) : 0; }();
    return v;
}

bool split_k_enabled() {
    static const bool v = [] { const char* e = getenv("OGLE_TC_SPLIT_K"); return !(e && e[0] == '0'); }();
    return v;
}

// Time of one reduction chunk (us) of an unsplit split-mode tile of 32, 64, ... columns on operands that come from L2:
// up to 160 columns the activation operands go through tensor memory, wider tiles build them in shared memory.
// On SM pairs: a chunk of both blocks' tiles. (148 tiles of one kind, 3x3, 18 and 36 chunks.)
constexpr double kChunkUs[8] = {0.355, 0.355, 0.355, 0.386, 0.48, 0.725, 0.81, 0.84};
constexpr double kPairChunkUs[4] = {0.65, 0.675, 0.70, 0.71};
// ... and of an epilogue, per column: in the shadow of the next tile's multiplies (two groups), and at the end.
constexpr double kEpilogueUs = 0.018, kTailUs = 0.035;

// Modelled time (us) of an unsplit launch in tiles of bn columns, and on SM pairs (split mode): rounds of tiles times the
// measured time of a tile; pointwise layers, whose tiles are read once, wait more for L2.
double whole_tiles_us(const TcArgs& t, int bn, int Kp, long m_tiles, int chunks) {
    const long tiles = m_tiles * ((Kp + bn - 1) / bn);
    // (one pass: 0.28 us up to 160 columns, bound by the copies, then by the multiplies)
    const double chunk = t.passes == 3 ? kChunkUs[bn / 32 - 1] : (0.0016 * bn + 0.01 > 0.28 ? 0.0016 * bn + 0.01 : 0.28);
    const double mul = chunks * chunk * (t.flat ? 1.25 : 1.0), epi = kEpilogueUs * bn;
    return (double)((tiles + kNumSMs - 1) / kNumSMs) * (mul > epi ? mul : epi) + 4.5 + (t.passes == 3 ? kTailUs : 0.02) * bn;
}
double pair_tiles_us(const TcArgs& t, int bn, int Kp, long m_tiles, int chunks) {
    const long work = (m_tiles + 1) / 2 * ((Kp + bn - 1) / bn);
    const double mul = chunks * kPairChunkUs[bn / 64 - 1] * (t.flat ? 1.1 : 1.0), epi = kEpilogueUs * bn;
    return (double)((work + kNumSMs / 2 - 1) / (kNumSMs / 2)) * (mul > epi ? mul : epi) + 5.5 + kTailUs * bn;
}

// Tiles of a launch whose taps lie side by side, bn channels each.
long tile_taps(const ConvArgs& a, int bn, TcArgs* t) {
    t->taps = 1;
    t->oH = a.Ho; t->oW = a.Wo;
    t->flat = 1; t->N = 1; t->Ho = 1; t->Wo = (int)a.M;
    t->tn = 1; t->th = 1; t->tw = kTapsPixels;
    t->BN = bn;
    t->n_tiles = (a.Kp + bn - 1) / bn;
    return (a.M + kTapsPixels - 1) / kTapsPixels;
}

// Width and form of an unsplit split-mode launch (the sums of an output value are the same in all of them): rounds of
// tiles times the measured time of a tile; pointwise layers, whose tiles are read once, wait more for L2. true: on SM
// pairs. 250 columns, 1350 elements, 14335 pixels: one tile of 256 columns 53.9 us, pairs 44.1, two tiles of 128 45.5;
// 512 -> 1024 pointwise, 25600 pixels: 118, 88, 95.
bool refine_width(TcArgs* t, int Kp, long m_tiles, int chunks, bool may_pair) {
    if (t->passes != 3 || t->gather || chunks < 8) return false;      // (short reductions are bound by HBM and the epilogue)
    const int kmax = (Kp + 31) / 32 * 32;
    auto one = [&](int bn) { return whole_tiles_us(*t, bn, Kp, m_tiles, chunks); };
    auto pair = [&](int bn) { return pair_tiles_us(*t, bn, Kp, m_tiles, chunks); };
    double best = 0.97 * one(t->BN);
    int best_bn = t->BN;
    bool best_pair = false;
    for (int bn = 32; bn <= 256 && bn <= kmax; bn += 32) {
        if (one(bn) < best) { best = one(bn); best_bn = bn; best_pair = false; }
        if (may_pair && m_tiles >= 2 && bn % 64 == 0 && pair(bn) < best) { best = pair(bn); best_bn = bn; best_pair = true; }
    }
    t->BN = best_bn;
    t->n_tiles = (Kp + best_bn - 1) / best_bn;
    return best_pair;
}

// Tiles of a k x k layer in whole rows of the map (pieces of one where it is wider than a tile); returns their number.
// may_split: the reduction may be split in two where that fills the SMs.
long whole_row_tiles(const ConvArgs& a, bool may_split, TcArgs* t) {
    if (a.Wo >= kTileM) {
        const int parts = (a.Wo + kTileM - 1) / kTileM;
        t->tw = (a.Wo + parts - 1) / parts; t->th = 1; t->tn = 1;
    } else {
        // full-width tiles of th rows from tn consecutive images (th * tn * Wo <= 128):
        // take the shape that needs the fewest rounds of one tile per SM; among equals the
        // tallest, whose filter taps overlap most in L2
        t->tw = a.Wo;
        long best = -1;
        for (int th = 1; th <= a.Ho && th * a.Wo <= kTileM; ++th) {
            int tn = kTileM / (th * a.Wo);
            if (tn > a.N) tn = a.N;
            if ((th - 1) * a.stride + 1 > 256) continue;          // TMA box limit
            const long tiles = (long)((a.Ho + th - 1) / th) * ((a.N + tn - 1) / tn);
            // in half-rounds; a reduction split in two can fill a ragged last round
            long rounds = 2 * ((tiles + kNumSMs - 1) / kNumSMs);
            if (may_split && (2 * tiles + kNumSMs - 1) / kNumSMs < rounds) rounds = (2 * tiles + kNumSMs - 1) / kNumSMs;
            if (best < 0 || rounds <= best) { best = rounds; t->th = th; t->tn = tn; }
        }
    }
    t->tiles_w = (a.Wo + t->tw - 1) / t->tw;
    t->tiles_h = (a.Ho + t->th - 1) / t->th;
    return (long)t->tiles_w * t->tiles_h * ((a.N + t->tn - 1) / t->tn);
}

// Tiles of a k x k layer cut along the width too: a map 75 pixels wide fills 75 of a tile's 128 rows in whole rows, and
// 114 in pieces of 38 x 3. Replaces the tile in t where that saves rounds (or, below one round, tiles); the sums of an
// output value do not change. 4 x 75 x 75 x 128 -> 256, 3x3: 103 -> 74 us (51 with tiles of 128 columns). cols: tiles
// along the output channels.
void cut_tiles(const ConvArgs& a, long cols, TcArgs* t, long* m_tiles) {
    auto cost = [&](long tiles) {
        tiles *= cols;
        return tiles > kNumSMs ? (double)((tiles + kNumSMs - 1) / kNumSMs) : 0.6 + 0.4 * tiles / kNumSMs;
    };
    double best = 0.92 * cost(*m_tiles);
    int best_parts = 0;
    for (int parts = (a.Wo + kTileM - 1) / kTileM; parts <= 16; ++parts) {
        const int tw = (a.Wo + parts - 1) / parts;
        if (tw < 8) break;
        if ((tw - 1) * a.stride + 1 > 256) continue;               // TMA box limit
        for (int th = 1; th <= a.Ho && th * tw <= kTileM && (th - 1) * a.stride + 1 <= 256; ++th) {
            int tn = kTileM / (th * tw);
            if (tn > a.N) tn = a.N;
            const long tiles_w = (a.Wo + tw - 1) / tw, tiles_h = (a.Ho + th - 1) / th;
            const long tiles = tiles_w * tiles_h * ((a.N + tn - 1) / tn);
            const double c = cost(tiles);
            if (c < (best_parts && parts != best_parts ? 0.97 * best : best) || (parts == best_parts && c == best)) {
                best = c; best_parts = parts;                     // (among equals of a width the tallest)
                t->tw = tw; t->th = th; t->tn = tn;
                t->tiles_w = (int)tiles_w; t->tiles_h = (int)tiles_h;
                *m_tiles = tiles;
            }
        }
    }
}

// Channels of a tile whose taps lie side by side (kTaps form), 0 = the launch does not take it: 3x3, stride 1, padding 1,
// where rounds of its tiles - 32 or 64 channels, a chunk and filter row at the measured time, and a longer epilogue - are
// modelled to take less than whole tiles in their better form. OGLE_TC_TAPS: 0 never, 1 wherever it can run.
// The sums are others than those of whole tiles, so that the layer's shape alone decides: the whole tiles compared with are
// those of a launch with an activation and without scratch, whatever this one has.
int taps_width(const ConvArgs& a, const TcArgs& own, int chunks) {
    static const int mode = [] { const char* e = getenv("OGLE_TC_TAPS"); return e ? (e[0] == '0' ? 1 : (e[0] == '1' ? 2 : 0)) : 0; }();
    if (mode == 1 || a.kernel != 3 || a.stride != 1 || a.pad != 1 || a.dil != 1 || a.M > 0x7fffff00L || !encode_im2col_fn()) return 0;
    if (mode == 0 && (forced_width(a.Kp) || pair_mode_override() == 2)) return 0;        // (those switches come first)
    double best = 1e30;
    int width = 0;
    long rounds = 0;
    for (int bn = 32; bn <= 64; bn += 32) {
        const long tiles = (a.M + kTapsPixels - 1) / kTapsPixels * ((a.Kp + bn - 1) / bn);
        // (a single round is mostly start, fill and drain; stacked siblings are padded to 32 channels each and seldom fill
        // tiles of 64: in few rounds the model cannot tell which form is the better one)
        if (mode == 0 && tiles <= (own.split_col ? 4 : 1) * kNumSMs) continue;
        const double chunk = own.passes == 3 ? (bn == 64 ? 0.57 : 0.45) : (bn == 64 ? 0.33 : 0.28);
        const double least = own.passes == 3 ? (bn == 64 ? 3.7 : 2.5) : (bn == 64 ? 3.1 : 2.2), tile = chunks / 3 * chunk + 1.0;
        const double us = (double)((tiles + kNumSMs - 1) / kNumSMs) * (tile > least ? tile : least) + 7.0;
        if (us < best) { best = us; width = bn; rounds = (tiles + kNumSMs - 1) / kNumSMs; }
    }
    if (!width || mode == 2) return width;
    TcArgs t = own;
    long m_tiles = whole_row_tiles(a, false, &t);
    choose_n_tiling_v2(a.Kp, m_tiles, &t);
    cut_tiles(a, (a.Kp + 127) / 128, &t, &m_tiles);
    double other = 1e30;
    for (int bn = 32; bn <= 256 && bn <= (a.Kp + 31) / 32 * 32; bn += 32) {
        if (t.passes != 3 && bn != t.BN) continue;
        const double one = whole_tiles_us(t, bn, a.Kp, m_tiles, chunks);
        const double two = t.passes == 3 && m_tiles >= 2 && bn % 64 == 0 ? pair_tiles_us(t, bn, a.Kp, m_tiles, chunks) : one;
        other = one < other ? one : other;
        other = two < other ? two : other;
    }
    // (split mode, tensors that come from HBM: whole tiles take 1.08 of the model and 3 us more, 20-170 us measured)
    if (t.passes == 3) other = 1.08 * other + 3.0;
    // (in two rounds start and drain are most of the time, and the models further off: 4 x 8 x 64 x 16 -> 577 11.3 us, 11.9)
    return best < (rounds <= 2 ? 0.88 : 0.97) * other ? width : 0;
}

// Tile width and number of ranges of a reduction split inside a cluster, for launches whose tiles leave SMs idle. All
// clusters have to fit the GPU at once (a block takes a whole SM; the GPU is asked how many clusters of a size fit), and
// the model has to see a tenth less time than in one piece: rounds of chunks, a block's start, fill and drain, and the
// cluster's barriers and exchange of partial tiles.
// split: the caller's choice (0 = any). otherwise: the ranges that the launch would have in its other forms.
// Where the caller leaves the number open, there are never fewer ranges than otherwise: sums in tensor memory are truncated,
// so that a range's error grows with its length (6e-9 of the result's norm per element in split mode), and results are to
// be as exact as in the launch's other forms. Nor do they move by more than 8e-6 of their norm against those: k and
// `otherwise` ranges of a reduction over R elements differ by 6e-9 * R * |1/k - 1/otherwise| (R = 512: 2.4e-6, R = 1500: 6.0e-6).
// 1000 x 1500 x 700 gemm: 32.8 -> 28.8 us with its packing pass (24.6 with that pass as it is now); MobileNet-SSD, one frame: 374 -> 335 us.
bool choose_cluster(TcArgs* t, int Kp, long m_tiles, int chunks, int split, int otherwise) {
    if (!split_k_enabled() || t->gather || split == 1 || split > 8 || m_tiles > kNumSMs / 2) return false;
    const int* capacity = tc_cluster_capacity();
    const int kmax = (Kp + 31) / 32 * 32;
    auto chunk = [&](int bn) { return t->passes == 3 ? kChunkUs[bn / 32 - 1] : 0.26 + 0.0002 * bn; };
    const long tiles0 = m_tiles * t->n_tiles;
    double best = otherwise > 1 || split ? 1e30 : 0.9 * ((tiles0 + kNumSMs - 1) / kNumSMs * (chunks * chunk(t->BN)) + 4.5 + kTailUs * t->BN);
    int best_bn = 0, best_k = 0;
    for (int bn = 32; bn <= 256 && bn <= kmax; bn += 32) {
        const long tiles = m_tiles * ((Kp + bn - 1) / bn);
        for (int k = split ? split : 2; k <= (split ? split : 8); ++k) {
            const int cps = (chunks + k - 1) / k;
            if ((k - 1) * cps >= chunks || tiles > capacity[k]) continue;
            if (!split && k < otherwise) continue;
            if (!split && t->passes == 3 && chunks * kChunk * fabs(1.0 / k - 1.0 / otherwise) > 1330.0) continue;
            const double cost = cps * chunk(bn) + 5.7 + (kTailUs + 0.004) * bn;
            if (cost < best) { best = cost; best_bn = bn; best_k = k; }
        }
    }
    if (!best_k) return false;
    t->BN = best_bn;
    t->n_tiles = (Kp + best_bn - 1) / best_bn;
    t->split_k = best_k;
    t->ws_mode = 0;
    t->cluster = 1;
    return true;
}

// Whether an unsplit launch can take the channels-on-M form (conv_tc2_t.cu): at most 128 (stacked) output channels, no
// gather, at least two 128-pixel tiles.
bool fits_channels_on_m(const TcArgs& t, int Kp_total, long m_tiles) {
    return !t.gather && t.bias_mode != 1 && Kp_total <= 128 && m_tiles >= 2;
}
// Whether a launch takes it: it can, its reduction is unsplit, and the caller asked for it (2) or the environment forces it
// for experiments.
bool want_channels_on_m(const TcArgs& t, int Kp_total, long m_tiles, int requested, bool through_scratch = false) {
    static const int mode = [] { const char* e = getenv("OGLE_TC_T"); return e ? (e[0] == '0' ? 1 : (e[0] == '1' ? 2 : 0)) : 0; }();
    if (!fits_channels_on_m(t, Kp_total, m_tiles)) return false;
    // a split reduction only in the form that goes through scratch
    if (through_scratch ? !(t.ws_mode && t.split_k > 1) : (t.split_k > 1 || t.ws_mode)) return false;
    if (mode == 1 || requested == 1) return false;
    return mode == 2 || requested == 2;
}

// Whether a launch takes the two-SM form because the caller or the environment asked for it: it can (no gather, no split
// reduction, a tile width that halves into multiples of 32 columns, at least one pair of tiles). Where neither asks,
// refine_width decides.
bool want_pair(const TcArgs& t, long m_tiles, int requested) {
    if (t.gather || t.split_k > 1 || t.ws_mode || t.BN % 64 || m_tiles < 2) return false;
    const int mode = pair_mode_override();
    if (mode == 1 || requested == 1) return false;
    if (mode == 2 || requested == 2) return true;
    return false;
}

}  // namespace

bool conv_tc_supported(const ConvArgs& a, int variant) {
    if (variant != CONV_GENERAL && variant != CONV_POINTWISE) return false;
    if (a.group != 1) return false;
    if (a.Cp < 16 || a.kernel * a.kernel * a.Cp < 32) return false;   // too few channels per tap: the RGB stem stays on CUDA cores
    if (a.kernel > 7) return false;
    if (!encode_fn()) return false;
    if (variant == CONV_GENERAL) {
        const int tw = a.Wo < 128 ? a.Wo : 128;
        if ((tw - 1) * a.stride + 1 > 256) return false;     // TMA box limit
    }
    return true;
}

// y2 != null: two-output form. a.K counts the stacked filters (first conv's K1 channels,
// zero rows up to split_col, then the second conv's); y receives [0, K1), y2 the rest.
// The gather form of the kernel: 3x3, at most three input channels stored as 16-byte pixels
// (the RGB stem), whole reduction (9 x C <= 27 values) in one chunk.
// Tile of the gather form: tw x th output pixels of one image, tw * th = 128; the shape that
// wastes the fewest rows among those whose input window (halo included) is at most 1024
// pixels = 16 KB of shared memory per stage. Windows of up to 128 pixels a row have their map of row-long extents, which
// is the faster copy; wider ones, up to 256 (a TMA box limit), are taken where they waste a good deal less, on maps one to
// five rows high mostly: one pass, 512 images of 1 x 1024 5x5 64 us, 111 in the best narrow tile, 5 x 128 44 and 48;
// at 7 % fewer rows (13 x 128) 97 and 99, split mode 95 and 91. Split-mode tiles of 256 channels leave no room for two
// stages with wider windows. wide = 0: narrow ones only.
static bool gather_tile(const ConvArgs& a, bool wide, int* tw_out, int* th_out) {
    double best = -1;
    for (int tw = 128; tw >= 16; tw >>= 1) {
        const int th = kTileM / tw;
        const int iw = (tw - 1) * a.stride + a.kernel, ih = (th - 1) * a.stride + a.kernel;
        if (iw > (wide ? 256 : 128) || iw * ih > 1024) continue;
        const double covered = (double)((a.Wo + tw - 1) / tw) * tw * ((a.Ho + th - 1) / th) * th * (iw > 128 ? 1.08 : 1.0);
        if (best < 0 || covered < best) { best = covered; *tw_out = tw; *th_out = th; }
    }
    return best >= 0;
}

bool conv_tc_gather_supported(const ConvArgs& a, int variant) {
    // 3x3 layers have the direct small-channel kernel, which is as fast on the networks measured: the
    // gather form is opt-in for them and the default for the larger filters, which have no such kernel
    static const bool enabled3 = [] { const char* e = getenv("OGLE_TC_GATHER"); return e && e[0] == '1'; }();
    static const bool disabled = [] { const char* e = getenv("OGLE_TC_GATHER"); return e && e[0] == '0'; }();
    if (disabled || (a.kernel == 3 && !enabled3)) return false;
    int tw, th;
    return variant == CONV_GENERAL && filter_compact(a.C / a.group, a.kernel, a.group) && a.dil == 1 &&
           filter_compact_cols(a.C, a.kernel) <= kMaxGatherK &&
           (a.stride == 1 || a.stride == 2) && a.Cp == 4 && a.Cs == 4 && a.Wo >= 16 && a.K <= 256 && gather_tile(a, false, &tw, &th) &&
           encode_fn() != nullptr;
}

// Adds the slices of a split reduction in slice order, then bias and activation, and writes the
// output tensor(s). One thread per four channels of a pixel. ws: [slices][rows_stride rows][ws_cols];
// y: stride Ks, first channel koff, K real channels (lanes K..up4(K)-1 written as zero); with y2 the
// columns from split_col on go to the second tensor (dense, K2 channels).
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float4* __restrict__ ws, int slices, long slice_q, int ws_cols_q, long rows,
                     const float* __restrict__ bias, int act, float lo, float hi,
                     float4* __restrict__ y, int Ks_q, int koff_q, int K, int out_q,
                     float4* __restrict__ y2, int split_col, int K2, int out2_q) {
    grid_dependency_trigger();
    grid_dependency_wait();
    const int per_row = out_q + out2_q;
    const long total = rows * per_row;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long m = i / per_row;
        int c = int(i - m * per_row);
        const bool second = c >= out_q;
        if (second) c -= out_q;
        const int col = (second ? split_col : 0) + c * 4;          // column in the stacked accumulator order
        const int real = second ? K2 : K;
        const float4* src = ws + m * ws_cols_q + (col >> 2);
        float4 acc = src[0];
        for (int s = 1; s < slices; ++s) {
            const float4 v = src[(long)s * slice_q];
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        float r[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const int n = c * 4 + l;
            if (n < real) {
                if (bias) r[l] += bias[col + l];
                r[l] = apply_act(r[l], act, lo, hi);
            } else {
                r[l] = 0.f;                                         // padded lanes stay zero
            }
        }
        const float4 o = make_float4(r[0], r[1], r[2], r[3]);
        if (second) y2[m * out2_q + c] = o;
        else y[m * Ks_q + koff_q + c] = o;
    }
}

// ws / ws_bytes: scratch for a split reduction of more than two ranges (or of a layer with an
// activation), may be null. ws_needed != null: plan only - no tensor maps, no launch - and report the
// scratch size this layer would like.
// Whether a convolution has so few pixels that the CUDA cores are quicker (few_rows.cu), and the caller leaves the ranges of
// the reduction open (a tile width, pairs of SMs or channels on M say how tiles are laid out, and there are none):
// a fixed 3 us instead of 6 to 8, but by the multiply-add (in graphs: 9 pixels, 256 -> 128 pointwise 6.4 -> 3.8 us, 4 pixels
// of 3x3 256 -> 150 9.3 -> 4.6, 8 of them 9.5 -> 5.8; 16 pixels of 3x3 69 -> 271, 2.7 M products, 7.9 -> 8.5).
// Not where a reduction is short for its columns: blocks that the GPU does not hold at once (three to an SM) take one and a half
// to five us more, and 64 elements take the tensor cores 5.0 (6.2 with more than 512 columns). 24 pixels 64 -> 700, 528 blocks,
// 6.4 -> 5.8, 32 of 64 -> 512 4.9 -> 5.8, of 33 -> 1366 6.4 -> 11.2; two steps a warp 6 of 164 -> 2342 7.3 -> 8.1; 128 elements
// 7 of 2785 columns 7.1 -> 6.4, and longer ones have no more columns than that.
static bool few_rows(const ConvArgs& a) {
    if (a.split || filter_compact(a.C, a.kernel, 1)) return false;
    const double products = (double)a.M * a.K * a.kernel * a.kernel * a.C;
    if (!((a.M <= 32 && products <= 1.5e6) || (a.M <= 8 && products <= 3e6))) return false;
    const int total = a.kernel * a.kernel * ((a.C + 31) / 32 * 32), rows = few_rows_rows(a.M);
    const int per_block = 8 / few_rows_warps(a.K, total) * few_rows_cols(a.K);
    const long blocks = (long)div_up(up4(a.K), per_block) * div_up(a.M, rows);
    if (rows < 4 || blocks <= 3 * kNumSMs) return true;
    if (total <= 64) return a.K > 512 && blocks <= 560;
    return total <= 128 || total >= 256;
}

// Whether a stem of 5 x 5 or 7 x 7 filters takes its windows as they are (conv_window.cu): one tile of channels, and maps that
// its tiles of 8 x 16 pixels (or, at stride 1, 128 x 1) cover about as well as the gather form's best shape. In graphs, 7 x 7 / 2, 3 -> 64 channels, one
// pass: 1 image of 224 x 224 8.2 us gathered, 7.2 so, 8 24.1 and 14.5, 128 279 and 135; split mode 32 images 69.3 and 62.1,
// 128 257 and 226. With 49 channels and more and three values to gather it is no better up to eight rounds of tiles (1 image
// 7.7 and 8.6, 8 20.9 and 21.0, 16 34.1 and 33.6), with fewer channels from the first on (3 x 200 x 120 -> 48 20.9 and 14.6).
// One input channel is a quarter of what the window's pixels carry, and 25 or 49 values a row are soon gathered: where whole
// slabs of outputs leave the gather form without ragged ends it is the better one in split mode (7x7, 3 images of 112 x 70 -> 64
// 7.3 and 8.6, 5 of 241 x 143 at stride 1 26.3 and 29.4; 5x5 between 0.90 and 1.07 of it), in one pass up to a round of 7x7 tiles
// (86 x 193 -> 64 7.0 and 7.8; 20 images of 38 x 114 15.9 and 14.6).
static double window_tiles(const ConvArgs& a, bool* row_tiles) {
    const double tall = (double)((a.Wo + 7) / 8) * ((a.Ho + 15) / 16), flat = (double)((a.Wo + 127) / 128) * a.Ho;
    *row_tiles = a.stride == 1 && flat < tall;
    return *row_tiles ? flat : tall;
}
static bool window_form(const ConvArgs& a, int variant, bool split_mode) {
    int tw, th;
    bool row_tiles;
    if (a.kernel == 3 || a.K > 64 || !conv_tc_gather_supported(a, variant) || !gather_tile(a, true, &tw, &th)) return false;
    const double gathered = (double)((a.Wo + tw - 1) / tw) * ((a.Ho + th - 1) / th), windows = window_tiles(a, &row_tiles);
    if (split_mode && a.kernel == 7 && a.C == 3 && a.K > 48 && windows * a.N <= 8.0 * kNumSMs) return false;
    if (a.C == 1 && a.K % 32 == 0 && a.kernel == 7 && (split_mode || (windows < gathered ? windows : gathered) * a.N <= kNumSMs)) return false;
    return windows <= 1.3 * gathered && windows * a.N < 0x7fffffff - 2 * kNumSMs;
}

// The kernel that launch_conv_tc runs for a layer (the tensor-core forms by one name); with two outputs none has a window.
const char* conv_tc_name(const ConvArgs& a, int variant, int math_mode) {
    if (few_rows(a)) return "few_rows_kernel";
    return window_form(a, variant, math_mode == OGLE_MATH_TF32X3) ? "conv_window_kernel" : "conv_tc2_kernel";
}

int launch_conv_tc(const ConvArgs& a, int variant, int math_mode, const float* x, const float* w_hi,
                   const float* w_lo, const float* bias, float* y, cudaStream_t s, float* y2, int K1,
                   int split_col, void* ws, size_t ws_bytes, size_t* ws_needed, const float* residual, int res_ld) {
    const bool plan_only = ws_needed != nullptr;
    if (residual && (y2 || res_ld < a.Kp || (res_ld & 3))) return OGLE_ERR_UNSUPPORTED;
    if (plan_only) *ws_needed = 0;
    TcArgs t = {};
    if (y2) {
        if (split_col <= 0 || (split_col & 31) || K1 <= 0 || K1 > split_col || split_col >= a.K ||
            a.koff != 0)
            return OGLE_ERR_UNSUPPORTED;
        t.split_col = split_col;
        t.K1 = K1;
    }
    if (!plan_only && few_rows(a)) {
        FewRowsArgs r = {};
        r.x = x; r.hi = w_hi; r.lo = math_mode == OGLE_MATH_TF32X3 ? w_lo : nullptr; r.bias = bias; r.res = residual;
        r.y = y + a.koff; r.y2 = y2;
        r.M = (int)a.M; r.N = a.K; r.C = a.C; r.Cp32 = (a.C + 31) / 32 * 32; r.kernel = a.kernel;
        r.H = a.H; r.W = a.W; r.Ho = a.Ho; r.Wo = a.Wo; r.stride = a.stride; r.pad = a.pad; r.dil = a.dil;
        r.ldx = a.Cs; r.ldy = y2 ? up4(K1) : a.Ks; r.ldy2 = y2 ? up4(a.K - split_col) : 0; r.res_ld = res_ld;
        r.split_col = y2 ? split_col : 0; r.N1 = K1;
        r.alpha = 1.f; r.beta = 1.f; r.bias_mode = a.has_bias ? 2 : 0;
        r.act = a.act; r.lo_clip = a.lo; r.hi_clip = a.hi;
        return launch_few_rows(r, s);
    }
    if (!plan_only && !y2 && window_form(a, variant, math_mode == OGLE_MATH_TF32X3)) {
        // (the tap-major section of the packed filter lies in front of the one that w_hi points to)
        const float* taps_first = w_hi - filter_layout(a.K, a.C, a.kernel, 1, a.Cp).off_hi / sizeof(float);
        bool row_tiles;
        window_tiles(a, &row_tiles);
        return launch_conv_window(a, math_mode == OGLE_MATH_TF32X3 ? 3 : 1, row_tiles, x, taps_first, bias, y, residual, res_ld, s);
    }
    // channel extents and row strides of the output tensor(s)
    const int kp_a = y2 ? up4(K1) : a.Kp, ks_a = y2 ? up4(K1) : a.Ks;
    const int kp_b = y2 ? up4(a.K - split_col) : a.Kp;
    const int taps = a.kernel * a.kernel;
    t.Cp32 = (a.C + 31) / 32 * 32;
    t.chunks_per_tap = t.Cp32 / kChunk;
    t.kernel = a.kernel; t.stride = a.stride; t.pad = a.pad; t.dil = a.dil;
    t.K = a.K; t.Kp = a.Kp; t.Ks = a.Ks; t.koff = a.koff;
    t.act = a.act; t.lo = a.lo; t.hi = a.hi;
    t.alpha = 1.f; t.beta = 1.f; t.bias_mode = a.has_bias ? 2 : 0; t.ldc = 0;
    t.passes = math_mode == OGLE_MATH_TF32X3 ? 3 : 1;
    const bool v2 = true;

    CUtensorMap mA, mBhi, mBlo, mY, mY2;
    long m_tiles;
    // planning needs the tile geometry only
    auto make_map = [&](CUtensorMap* m, const void* p, int rank, const cuuint64_t* d, const cuuint64_t* st, const cuuint32_t* b,
                        const cuuint32_t* e) { return plan_only ? true : ogle::make_map(m, p, rank, d, st, b, e); };
    if (variant == CONV_POINTWISE) {
        t.flat = 1;
        t.N = 1; t.Ho = 1; t.Wo = (int)a.M;
        t.tn = 1; t.th = 1; t.tw = kTileM;
        m_tiles = (a.M + kTileM - 1) / kTileM;
        const cuuint64_t dims[4] = {(cuuint64_t)a.Cp, (cuuint64_t)a.M, 1, 1};
        const cuuint64_t str[3] = {(cuuint64_t)a.Cs * 4, (cuuint64_t)a.Cs * 4 * (cuuint64_t)a.M, (cuuint64_t)a.Cs * 4 * (cuuint64_t)a.M};
        const cuuint32_t box[4] = {kChunk, kTileM, 1, 1};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        if (!make_map(&mA, x, 4, dims, str, box, es)) return OGLE_ERR_CUDA;
        if (v2) {
            const cuuint64_t yd[4] = {(cuuint64_t)kp_a, (cuuint64_t)a.M, 1, 1};
            const cuuint64_t ys[3] = {(cuuint64_t)ks_a * 4, (cuuint64_t)ks_a * 4 * (cuuint64_t)a.M, (cuuint64_t)ks_a * 4 * (cuuint64_t)a.M};
            if (!make_map(&mY, y + a.koff, 4, yd, ys, box, es)) return OGLE_ERR_CUDA;
            if (residual) {
                const cuuint64_t rs[3] = {(cuuint64_t)res_ld * 4, (cuuint64_t)res_ld * 4 * (cuuint64_t)a.M, (cuuint64_t)res_ld * 4 * (cuuint64_t)a.M};
                if (!make_map(&mY2, residual, 4, yd, rs, box, es)) return OGLE_ERR_CUDA;
            }
            if (y2) {
                const cuuint64_t yd2[4] = {(cuuint64_t)kp_b, (cuuint64_t)a.M, 1, 1};
                const cuuint64_t ys2[3] = {(cuuint64_t)kp_b * 4, (cuuint64_t)kp_b * 4 * (cuuint64_t)a.M, (cuuint64_t)kp_b * 4 * (cuuint64_t)a.M};
                if (!make_map(&mY2, y2, 4, yd2, ys2, box, es)) return OGLE_ERR_CUDA;
            }
        }
    } else if (conv_tc_gather_supported(a, variant) && !y2) {
        t.flat = 0;
        t.N = a.N; t.Ho = a.Ho; t.Wo = a.Wo;
        t.gather = 1; t.g_C = a.C; t.g_k = a.kernel;
        t.kernel = 1;                                            // the reduction is a run of gathered chunks
        t.Cp32 = filter_compact_cols(a.C, a.kernel); t.chunks_per_tap = t.Cp32 / kChunk;
        if (!gather_tile(a, t.passes == 1 || a.Kp <= 224, &t.tw, &t.th)) return OGLE_ERR_UNSUPPORTED;
        t.tn = 1;
        t.tiles_w = (a.Wo + t.tw - 1) / t.tw;
        t.tiles_h = (a.Ho + t.th - 1) / t.th;
        m_tiles = (long)t.tiles_w * t.tiles_h * a.N;
        t.g_iw = (t.tw - 1) * a.stride + a.kernel;
        t.g_ih = (t.th - 1) * a.stride + a.kernel;
        t.g_bytes = (t.g_iw * t.g_ih * 16 + 1023) / 1024 * 1024;
        const cuuint32_t es[4] = {1, 1, 1, 1};
        if (t.g_iw > 128) {
            const cuuint64_t dims[4] = {4, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.N};
            const cuuint64_t str[3] = {16, (cuuint64_t)a.W * 16, (cuuint64_t)a.W * 16 * a.H};
            const cuuint32_t box[4] = {4, (cuuint32_t)t.g_iw, (cuuint32_t)t.g_ih, 1};
            if (!plan_only && !make_map_sw(CU_TENSOR_MAP_SWIZZLE_NONE, &mA, x, 4, dims, str, box, es)) return OGLE_ERR_CUDA;
        } else if (!plan_only && !make_map_pixels(&mA, x, a.W, a.H, a.N, t.g_iw, t.g_ih)) {
            return OGLE_ERR_CUDA;
        }
        const cuuint64_t yd[4] = {(cuuint64_t)kp_a, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)a.N};
        const cuuint64_t ys[3] = {(cuuint64_t)ks_a * 4, (cuuint64_t)ks_a * 4 * a.Wo, (cuuint64_t)ks_a * 4 * a.Wo * a.Ho};
        const cuuint32_t yb[4] = {kChunk, (cuuint32_t)t.tw, (cuuint32_t)t.th, 1};
        if (!make_map(&mY, y + a.koff, 4, yd, ys, yb, es)) return OGLE_ERR_CUDA;
        if (residual) {
            const cuuint64_t rs[3] = {(cuuint64_t)res_ld * 4, (cuuint64_t)res_ld * 4 * a.Wo, (cuuint64_t)res_ld * 4 * a.Wo * a.Ho};
            if (!make_map(&mY2, residual, 4, yd, rs, yb, es)) return OGLE_ERR_CUDA;
        }
    } else {
        t.flat = 0;
        t.N = a.N; t.Ho = a.Ho; t.Wo = a.Wo;
        m_tiles = whole_row_tiles(a, v2 && a.act == OGLE_ACT_NONE && split_k_enabled() && taps * t.chunks_per_tap >= 16, &t);
    }
    // How many ranges the reduction has is settled at the library's own tile width, whatever width or form the caller
    // asks for: those change how a launch is laid out, not the order in which a value's products are added.
    const bool wide_ties = (plan_only || (ws != nullptr && aligned16(ws))) && !t.gather && split_k_enabled() &&
                           taps * t.chunks_per_tap >= 16;
    choose_n_tiling_v2(a.Kp, m_tiles, &t, 0, wide_ties);
    // Split the reduction when whole tiles would leave SMs idle (few tiles) or a last round
    // mostly empty. Two forms, for reductions that do not fit clusters (below):
    //  - through scratch memory (the caller lent some): any number of ranges and any activation;
    //    each range stores its partial tile into its own slice and a small second kernel adds the
    //    slices in slice order, then bias and activation - bit-reproducible whatever the order in
    //    which blocks finish;
    //  - in place, two ranges, no activation: the output (a dense tensor, or this convolution's
    //    channel slice of a wider one) is zeroed first and the two partial tiles are added to it by
    //    TMA reduce stores; a sum of two addends onto zero does not depend on their order either.
    t.split_k = 1;
    const int chunks = t.kernel * t.kernel * t.chunks_per_tap;
    const double tiles = (double)m_tiles * t.n_tiles;
    // rows (flat form) or images between consecutive slices: whole tiles, so that a tile that
    // hangs over the end of its slice writes padding, not the next slice
    const long slice_units = t.flat ? m_tiles * kTileM : (long)((a.N + t.tn - 1) / t.tn) * t.tn;
    const size_t slice_rows = (size_t)(t.flat ? slice_units : slice_units * a.Ho * a.Wo);
    size_t slice_bytes = slice_rows * (t.n_tiles * t.BN) * sizeof(float);
    if (split_k_enabled() && chunks >= 8 && !residual) {      // (a residual operand is added by whole tiles only)
        // cost of the layer in units of one reduction chunk of one tile: rounds of one work item per SM,
        // each item paying its chunks plus a fixed fill / drain of about four chunks
        auto cost_of = [&](int k) {
            const int cps = (chunks + k - 1) / k;
            return ceil(tiles * k / kNumSMs) * (cps + 4.0);
        };
        double best = cost_of(1);
        int best_k = 1;
        bool best_ws = false;
        if (a.act == OGLE_ACT_NONE && chunks / 2 >= 8 && cost_of(2) + 2.0 < 0.9 * best) { best = cost_of(2) + 2.0; best_k = 2; }
        const bool ws_usable = plan_only || (ws != nullptr && aligned16(ws));
        if (ws_usable && !t.gather) {
            static const int cand[] = {2, 3, 4, 6, 8, 12, 16};
            for (int k : cand) {
                if (chunks / k < 4) break;
                if (!plan_only && slice_bytes * k > ws_bytes) break;
                if (slice_bytes * k > ((size_t)192 << 20)) break;
                // + the second kernel: a launch and a pass over k slices
                const double c = cost_of(k) + 10.0 + 0.5 * k;
                if (c < 0.85 * best) { best = c; best_k = k; best_ws = true; }
            }
        }
        if (a.split >= 1) {
            // the caller's choice, as far as it can be served: the in-place form for two ranges without an
            // activation, else the scratch form when scratch of the right size was lent
            int k = a.split;
            while (k > 1 && chunks / k < 1) --k;
            const bool fits = ws_usable && !t.gather && (plan_only || slice_bytes * k <= ws_bytes) &&
                              slice_bytes * k <= ((size_t)192 << 20);
            if (k == 1) { best_k = 1; best_ws = false; }
            else if (k == 2 && a.act == OGLE_ACT_NONE && !fits) { best_k = 2; best_ws = false; }
            else if (fits) { best_k = k; best_ws = true; }
        }
        t.split_k = best_k;
        t.ws_mode = best_ws ? 1 : 0;
        const int cps = (chunks + t.split_k - 1) / t.split_k;
        while (t.split_k > 1 && (t.split_k - 1) * cps >= chunks) --t.split_k;     // no empty ranges
        if (t.split_k == 1) t.ws_mode = 0;
    }
    const TcArgs own = t;
    // (a wider tile than the layer is no wish)
    const int wish = a.n_tile >= 32 && a.n_tile <= (a.Kp + 31) / 32 * 32 ? a.n_tile : forced_width(a.Kp);
    if (wish) {
        choose_n_tiling_v2(a.Kp, m_tiles, &t, wish, wide_ties);
        const size_t wished = slice_rows * (t.n_tiles * t.BN) * sizeof(float), most = (size_t)192 << 20;
        if (t.ws_mode && wished * t.split_k > (plan_only || ws_bytes > most ? most : ws_bytes)) t = own;
        else slice_bytes = wished;
    }
    const int ws_cols = t.n_tiles * t.BN;
    const bool on_m = want_channels_on_m(t, a.Kp, m_tiles, a.on_m);
    const bool tiled = variant != CONV_POINTWISE && !t.gather;       // tiles of image pieces
    bool on_pairs = false;
    // (the scratch a layer asks for does not depend on whether the launch then splits inside clusters instead)
    // The ranges are settled on whole-row tiles; an unsplit launch is then free to cut its tiles and choose their width
    // and form, and so is one that splits inside clusters.
    if (!plan_only) {
        TcArgs c = own;
        long cut = m_tiles;
        if (tiled) cut_tiles(a, (a.Kp + 127) / 128, &c, &cut);
        // (the environment's SM pairs, "wherever they can run", come before the cluster form)
        const bool forced_pairs = !residual && pair_mode_override() == 2 && want_pair(t, m_tiles, a.pair);
        bool cluster = !(a.on_m == 2 && t.ws_mode) && !on_m && !forced_pairs && choose_cluster(&c, a.Kp, cut, chunks, a.split, own.split_k);
        if (cluster && wish) {
            c.BN = t.BN;
            c.n_tiles = t.n_tiles;
            // as many ranges, in more clusters than fit at once: through scratch where that is lent (the same bits)
            if (t.ws_mode && t.split_k == c.split_k && cut * c.n_tiles > tc_cluster_capacity()[c.split_k]) cluster = false;
        } else if (!cluster) {
            c.BN = t.BN;
            c.n_tiles = t.n_tiles;
        }
        if (cluster || t.split_k <= 1) { t = c; m_tiles = cut; }
        if (!cluster) {
            on_pairs = want_pair(t, m_tiles, a.pair);
            // (whether taps lie side by side is settled without a look at n_tile and sm_pair: it does touch the bits. Not
            // where channels lie on M, by the caller's wish or the environment's; and a caller who says 1 or 2 to that, of a
            // layer it fits, gets the same bits for both)
            const bool on_m_form = on_m || (a.on_m && fits_channels_on_m(t, a.Kp, m_tiles));
            const int beside = t.split_k <= 1 && !on_m_form && tiled ? taps_width(a, own, chunks) : 0;
            if (beside) {
                m_tiles = tile_taps(a, beside, &t);
                on_pairs = false;
            } else if (t.split_k <= 1 && !wish && !a.pair && !on_m && !forced_pairs)
                on_pairs = refine_width(&t, a.Kp, m_tiles, chunks, !residual && pair_mode_override() != 1);
        }
    }
    auto make_tile_maps = [&] {
        const cuuint64_t dims[4] = {(cuuint64_t)a.Cp, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.N};
        const cuuint64_t str[3] = {(cuuint64_t)a.Cs * 4, (cuuint64_t)a.Cs * 4 * a.W, (cuuint64_t)a.Cs * 4 * a.W * a.H};
        if (t.taps) {
            // rows from the one above the image on; of its columns every one, whose neighbours meet in the accumulator
            const int lower[2] = {0, -1}, upper[2] = {0, -1};
            const cuuint32_t yb[4] = {kChunk, kTapsPixels, 1, 1}, ye[4] = {1, 1, 1, 1};
            auto rows = [&](CUtensorMap* m, const float* p, int columns, int stride) {
                const cuuint64_t d[4] = {(cuuint64_t)columns, (cuuint64_t)a.M, 1, 1};
                const cuuint64_t st[3] = {(cuuint64_t)stride * 4, (cuuint64_t)stride * 4 * (cuuint64_t)a.M, (cuuint64_t)stride * 4 * (cuuint64_t)a.M};
                return make_map(m, p, 4, d, st, yb, ye);
            };
            return make_map_im2col(&mA, x, dims, str, lower, upper, kChunk, kTileM) && rows(&mY, y + a.koff, kp_a, ks_a) &&
                   (!y2 || rows(&mY2, y2, kp_b, kp_b)) && (!residual || rows(&mY2, residual, a.Kp, res_ld));
        }
        // the box spans the traversed input extent; one element in `stride` is taken
        const cuuint32_t box[4] = {kChunk, (cuuint32_t)((t.tw - 1) * a.stride + 1), (cuuint32_t)((t.th - 1) * a.stride + 1),
                                   (cuuint32_t)t.tn};
        const cuuint32_t es[4] = {1, (cuuint32_t)a.stride, (cuuint32_t)a.stride, 1};
        if (!make_map(&mA, x, 4, dims, str, box, es)) return false;
        if (v2) {
            const cuuint64_t yd[4] = {(cuuint64_t)kp_a, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)a.N};
            const cuuint64_t ys[3] = {(cuuint64_t)ks_a * 4, (cuuint64_t)ks_a * 4 * a.Wo, (cuuint64_t)ks_a * 4 * a.Wo * a.Ho};
            const cuuint32_t yb[4] = {kChunk, (cuuint32_t)t.tw, (cuuint32_t)t.th, (cuuint32_t)t.tn};
            const cuuint32_t ye[4] = {1, 1, 1, 1};
            if (!make_map(&mY, y + a.koff, 4, yd, ys, yb, ye)) return false;
            if (residual) {
                const cuuint64_t rs[3] = {(cuuint64_t)res_ld * 4, (cuuint64_t)res_ld * 4 * a.Wo, (cuuint64_t)res_ld * 4 * a.Wo * a.Ho};
                if (!make_map(&mY2, residual, 4, yd, rs, yb, ye)) return false;
            }
            if (y2) {
                const cuuint64_t yd2[4] = {(cuuint64_t)kp_b, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)a.N};
                const cuuint64_t ys2[3] = {(cuuint64_t)kp_b * 4, (cuuint64_t)kp_b * 4 * a.Wo, (cuuint64_t)kp_b * 4 * a.Wo * a.Ho};
                if (!make_map(&mY2, y2, 4, yd2, ys2, yb, ye)) return false;
            }
        }
        return true;
    };
    if (tiled && !plan_only && !make_tile_maps()) return OGLE_ERR_CUDA;
    const int Kp128 = (a.K + 127) / 128 * 128;
    const cuuint64_t bcols = t.gather ? (cuuint64_t)t.Cp32 : (cuuint64_t)taps * t.Cp32;
    const cuuint64_t bdims[2] = {bcols, (cuuint64_t)Kp128};
    const cuuint64_t bstr[1] = {bcols * 4};
    const cuuint32_t bbox[2] = {kChunk, (cuuint32_t)t.BN};
    const cuuint32_t bes[2] = {1, 1};
    if (t.taps) {
        // [channel][filter][tap]: a box takes the taps of a filter row one after the other
        const cuuint64_t d[3] = {(cuuint64_t)t.Cp32, (cuuint64_t)Kp128, (cuuint64_t)taps};
        const cuuint64_t st[2] = {bcols * 4, (cuuint64_t)t.Cp32 * 4};
        const cuuint32_t b[3] = {kChunk, (cuuint32_t)t.BN, 3}, e[3] = {1, 1, 1};
        if (!make_map(&mBhi, w_hi, 3, d, st, b, e) || !make_map(&mBlo, w_lo, 3, d, st, b, e)) return OGLE_ERR_CUDA;
    } else {
        if (!make_map(&mBhi, w_hi, 2, bdims, bstr, bbox, bes)) return OGLE_ERR_CUDA;
        if (!make_map(&mBlo, w_lo, 2, bdims, bstr, bbox, bes)) return OGLE_ERR_CUDA;
    }
    if (t.cluster) {
        t.res = residual;
        t.res_ld = res_ld;
        t.y = y + a.koff; t.y_ld = ks_a;
        t.y2 = y2; t.y2_ld = kp_b;
        return launch_tc_v2(t, mA, mBhi, mBlo, mY, y2 ? mY2 : mY, m_tiles, bias, error_flag_ptr(), s);
    }
    if (v2) {
        if (plan_only) {
            *ws_needed = t.ws_mode ? slice_bytes * t.split_k : 0;
            return OGLE_OK;
        }
        if (t.ws_mode) {
            // channels-on-M form: the scratch tensor is as wide as the filter tile (never wider than planned)
            const bool on_m = want_channels_on_m(t, a.Kp, m_tiles, a.on_m, true);
            const int wcols = on_m ? (a.Kp + 31) / 32 * 32 : ws_cols;
            const size_t wslice_bytes = (size_t)(t.flat ? slice_units : slice_units * a.Ho * a.Wo) * wcols * sizeof(float);
            t.ws_cols = wcols;
            t.ws_slice = (int)slice_units;
            const int act = t.act;
            const float lo = t.lo, hi = t.hi;
            t.act = OGLE_ACT_NONE;                 // the raw sums go to the scratch tensor
            const cuuint32_t es[4] = {1, 1, 1, 1};
            if (t.flat) {
                const cuuint64_t wd[4] = {(cuuint64_t)wcols, (cuuint64_t)slice_units * t.split_k, 1, 1};
                const cuuint64_t wst[3] = {(cuuint64_t)wcols * 4, (cuuint64_t)wcols * 4 * wd[1], (cuuint64_t)wcols * 4 * wd[1]};
                const cuuint32_t wb[4] = {kChunk, kTileM, 1, 1};
                if (!ogle::make_map(&mY, ws, 4, wd, wst, wb, es)) return OGLE_ERR_CUDA;
            } else {
                const cuuint64_t wd[4] = {(cuuint64_t)wcols, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)slice_units * t.split_k};
                const cuuint64_t wst[3] = {(cuuint64_t)wcols * 4, (cuuint64_t)wcols * 4 * a.Wo, (cuuint64_t)wcols * 4 * a.Wo * a.Ho};
                const cuuint32_t wb[4] = {kChunk, (cuuint32_t)t.tw, (cuuint32_t)t.th, (cuuint32_t)t.tn};
                if (!ogle::make_map(&mY, ws, 4, wd, wst, wb, es)) return OGLE_ERR_CUDA;
            }
            int rc;
            if (on_m) {
                t.BN = wcols;
                t.n_tiles = 1;
                const cuuint32_t fbox[2] = {kChunk, (cuuint32_t)t.BN};
                if (!ogle::make_map(&mBhi, w_hi, 2, bdims, bstr, fbox, bes)) return OGLE_ERR_CUDA;
                if (!ogle::make_map(&mBlo, w_lo, 2, bdims, bstr, fbox, bes)) return OGLE_ERR_CUDA;
                rc = launch_tc_t(t, mA, mBhi, mBlo, mY, mY, m_tiles, nullptr, error_flag_ptr(), s);
            } else {
                rc = launch_tc_v2(t, mA, mBhi, mBlo, mY, mY, m_tiles, nullptr, error_flag_ptr(), s);
            }
            if (rc != OGLE_OK) return rc;
            const long rows = a.M;
            const long slice_q = (long)(wslice_bytes / 16);
            const int out_q = kp_a / 4, out2_q = y2 ? kp_b / 4 : 0;
            const long items = rows * (out_q + out2_q);
            launch_overlapped(splitk_reduce_kernel, dim3(grid_for(items, 256)), dim3(256), 0, s,
                              reinterpret_cast<const float4*>(ws), t.split_k, slice_q, wcols / 4, rows,
                              a.has_bias ? bias : (const float*)nullptr, act, lo, hi, reinterpret_cast<float4*>(y), ks_a / 4,
                              a.koff / 4, y2 ? K1 : a.K, out_q, reinterpret_cast<float4*>(y2), split_col,
                              y2 ? a.K - split_col : 0, out2_q);
            return finish_launch();
        }
        if (t.split_k > 1) {
            const size_t rows = (size_t)a.M;
            if (ks_a == kp_a) {
                if (cudaMemsetAsync(y + a.koff, 0, rows * (size_t)ks_a * sizeof(float), s) != cudaSuccess) return OGLE_ERR_CUDA;
            } else if (cudaMemset2DAsync(y + a.koff, (size_t)ks_a * sizeof(float), 0, (size_t)kp_a * sizeof(float), rows, s) !=
                       cudaSuccess) {
                return OGLE_ERR_CUDA;
            }
            if (y2 && cudaMemsetAsync(y2, 0, rows * (size_t)kp_b * sizeof(float), s) != cudaSuccess) return OGLE_ERR_CUDA;
        }
        t.res = residual;
        t.res_ld = res_ld;
        if (on_m) {
            // the filter tile is the M-side operand: all (stacked) channels in one tile of FR rows
            t.BN = (a.Kp + 31) / 32 * 32;
            t.n_tiles = 1;
            const cuuint32_t fbox[2] = {kChunk, (cuuint32_t)t.BN};
            if (!ogle::make_map(&mBhi, w_hi, 2, bdims, bstr, fbox, bes)) return OGLE_ERR_CUDA;
            if (!ogle::make_map(&mBlo, w_lo, 2, bdims, bstr, fbox, bes)) return OGLE_ERR_CUDA;
            return launch_tc_t(t, mA, mBhi, mBlo, mY, y2 ? mY2 : mY, m_tiles, bias, error_flag_ptr(), s);
        }
        if (!residual && on_pairs) {
            // each block of a pair loads half of the filter tile's rows
            const cuuint32_t hbox[2] = {kChunk, (cuuint32_t)(t.BN / 2)};
            if (!ogle::make_map(&mBhi, w_hi, 2, bdims, bstr, hbox, bes)) return OGLE_ERR_CUDA;
            if (!ogle::make_map(&mBlo, w_lo, 2, bdims, bstr, hbox, bes)) return OGLE_ERR_CUDA;
            return launch_tc_pair(t, mA, mBhi, mBlo, mY, y2 ? mY2 : mY, m_tiles, bias, error_flag_ptr(), s);
        }
        return launch_tc_v2(t, mA, mBhi, mBlo, mY, y2 || residual ? mY2 : mY, m_tiles, bias, error_flag_ptr(), s);
    }
    return OGLE_ERR_UNSUPPORTED;
}

// gemm through the same kernel. B must be K-major: either the caller's B when
// transB == 1 (one-pass mode only) or a packed hi/lo copy made by gemm_pack_b.
bool gemm_tc_supported(const OgleGemmParams& p, const float* A, const float* B) {
    if (p.K < 64 || !encode_fn()) return false;
    if (p.math_mode == OGLE_MATH_TF32 && p.transB == 1 && aligned16(B)) return true;
    return false;
}

static int launch_gemm_common(const OgleGemmParams& p, const float* A, const float* Bhi, const float* Blo,
                              long b_row_stride, long b_rows, const float* C, float* Y, cudaStream_t s, int passes,
                              bool overlapped = false) {
    TcArgs t = {};
    t.overlapped = overlapped;
    t.flat = 1; t.N = 1; t.Ho = 1; t.Wo = p.M; t.tn = 1; t.th = 1; t.tw = kTileM;
    t.kernel = 1; t.stride = 1; t.pad = 0; t.dil = 1;
    t.Cp32 = (p.K + 31) / 32 * 32;
    t.chunks_per_tap = t.Cp32 / kChunk;
    t.K = p.N; t.Kp = up4(p.N); t.Ks = p.ldy; t.koff = 0;
    t.act = OGLE_ACT_NONE;
    t.alpha = p.alpha; t.beta = p.beta; t.bias_mode = p.bias_mode; t.ldc = p.ldc;
    t.passes = passes;
    const bool v2 = true;
    const long m_tiles = (p.M + kTileM - 1) / kTileM;
    choose_n_tiling_v2(t.Kp, m_tiles, &t);
    const int forced = forced_width(t.Kp);
    if (forced) choose_n_tiling_v2(t.Kp, m_tiles, &t, forced);
    bool on_pairs = pair_mode_override() == 2 && want_pair(t, m_tiles, 0);
    if (!on_pairs) {
        TcArgs c = t;
        if (choose_cluster(&c, t.Kp, m_tiles, t.chunks_per_tap, 0, 1)) {
            if (forced) { c.BN = t.BN; c.n_tiles = t.n_tiles; }
            t = c;
        } else if (!forced) {
            on_pairs = refine_width(&t, t.Kp, m_tiles, t.chunks_per_tap, pair_mode_override() != 1);
        }
    }
    t.y = Y; t.y_ld = p.ldy;
    CUtensorMap mA, mBhi, mBlo, mY;
    const cuuint64_t dims[4] = {(cuuint64_t)p.K, (cuuint64_t)p.M, 1, 1};
    const cuuint64_t str[3] = {(cuuint64_t)p.lda * 4, (cuuint64_t)p.lda * 4 * (cuuint64_t)p.M, (cuuint64_t)p.lda * 4 * (cuuint64_t)p.M};
    const cuuint32_t box[4] = {kChunk, kTileM, 1, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    if (!make_map(&mA, A, 4, dims, str, box, es)) return OGLE_ERR_CUDA;
    const cuuint64_t bdims[2] = {(cuuint64_t)(Blo ? t.Cp32 : p.K), (cuuint64_t)b_rows};
    const cuuint64_t bstr[1] = {(cuuint64_t)b_row_stride * 4};
    const cuuint32_t bbox[2] = {kChunk, (cuuint32_t)(on_pairs ? t.BN / 2 : t.BN)};      // each block of a pair loads half
    const cuuint32_t bes[2] = {1, 1};
    if (!make_map(&mBhi, Bhi, 2, bdims, bstr, bbox, bes)) return OGLE_ERR_CUDA;
    if (!make_map(&mBlo, Blo ? Blo : Bhi, 2, bdims, bstr, bbox, bes)) return OGLE_ERR_CUDA;
    if (v2) {
        const cuuint64_t yd[4] = {(cuuint64_t)t.Kp, (cuuint64_t)p.M, 1, 1};
        const cuuint64_t ys[3] = {(cuuint64_t)p.ldy * 4, (cuuint64_t)p.ldy * 4 * (cuuint64_t)p.M, (cuuint64_t)p.ldy * 4 * (cuuint64_t)p.M};
        if (!make_map(&mY, Y, 4, yd, ys, box, es)) return OGLE_ERR_CUDA;
        if (on_pairs) return launch_tc_pair(t, mA, mBhi, mBlo, mY, mY, m_tiles, C, error_flag_ptr(), s);
        return launch_tc_v2(t, mA, mBhi, mBlo, mY, mY, m_tiles, C, error_flag_ptr(), s);
    }
    return OGLE_ERR_UNSUPPORTED;
}

int launch_gemm_tc(const OgleGemmParams& p, const float* A, const float* B, const float* C, float* Y, cudaStream_t s) {
    return launch_gemm_common(p, A, B, nullptr, p.ldb, p.N, C, Y, s, 1);
}

int launch_gemm_tc_packed(const OgleGemmParams& p, const float* A, const float* Bhi, const float* Blo,
                          const float* C, float* Y, cudaStream_t s, bool overlapped) {
    const long Cp32 = (p.K + 31) / 32 * 32;
    const long rows = (p.N + 127) / 128 * 128;
    return launch_gemm_common(p, A, Bhi, Blo, Cp32, rows, C, Y, s, p.math_mode == OGLE_MATH_TF32X3 ? 3 : 1, overlapped);
}

namespace {
std::atomic<uint32_t> g_role_wait_limit{tc::kSpinLimit};
}
uint32_t tc::role_wait_limit() { return g_role_wait_limit.load(std::memory_order_relaxed); }
void set_role_wait_limit(long polls) {
    g_role_wait_limit.store(polls < 0 ? tc::kSpinLimit : (polls > long(tc::kSpinLimit) ? tc::kSpinLimit : uint32_t(polls)),
                            std::memory_order_relaxed);
}

int read_tc_error() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
int clear_tc_error() {
    const int z = 0;
    return cudaMemcpyToSymbol(g_tc_error, &z, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace ogle
