// SSD box decoder and detection post-process.
//
// decode: one thread per anchor, 128-bit loads/stores (HBM-bound).
// detect: a block reads an image's logits once and turns them into softmax scores in shared memory,
// counting them into a histogram per class on the way; then one warp per class (mode 1) or per image
// (mode 0) takes the top-k out of the scores by that histogram (warp_topk). Logits and boxes cross HBM
// once and nothing is staged in global memory.
// What bounds it is the number of instructions: 1024 images x 1917 anchors x 21 classes, top 200, took
// 428 us with a radix selection over registers and a radix sort of the survivors (238 k warp
// instructions per image); counting into the bins that the sort needs anyway took it to 192 us, kernels that know how many
// pieces a row of logits has to 155 with the decode (logits in and results out take 47 at the HBM rate).
#include <cstring>

#include "common.cuh"

namespace ogle {

__device__ __forceinline__ float4 decode_box(float4 p, float4 a, float4 var) {
    // decoder.glsl:21-27, products taken left to right as written there
    const float w = expf(p.z * var.z) * a.z;
    const float h = expf(p.w * var.w) * a.w;
    const float cx = p.x * var.x * a.z + a.x;
    const float cy = p.y * var.y * a.w + a.y;
    return make_float4(cx - 0.5f * w, cy - 0.5f * h, cx + 0.5f * w, cy + 0.5f * h);
}

__global__ void ssd_decode_kernel(const float4* __restrict__ pred, const float4* __restrict__ anchors,
                                  float4* __restrict__ out, long total, int A, float4 var) {
    grid_dependency_trigger();
    grid_dependency_wait();
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        out[i] = decode_box(pred[i], anchors[i % A], var);
    }
}

constexpr int kMaxTopK = 256;
constexpr int kBins = 512;               // of a score histogram: two 16-bit counts to a word
constexpr int kHistWords = kBins / 2;
constexpr int kListMax = 384;            // survivors a warp orders at once
constexpr int kEdgeMax = 96;             // of which at most this many share the bin that the k-th falls into

// Scores as keys: bits(score) - base with base = bits(threshold), so that positive floats order like their keys,
// candidates (score > threshold) have keys 1..max_key and everything else (NaN included) lies outside.
struct KeySpace {
    unsigned base, max_key;
    int shift;                           // key >> shift is the histogram bin
};

__device__ __forceinline__ void hist_add(unsigned* hist, unsigned bin) {
    atomicAdd(&hist[bin >> 1], 1u << ((bin & 1u) * 16u));
}
__device__ __forceinline__ unsigned hist_get(const unsigned* hist, unsigned bin) {
    return (hist[bin >> 1] >> ((bin & 1u) * 16u)) & 0xffffu;
}

// Warp-collective: the k largest candidates among vals[0..Ap) in order (score descending, equal scores by index)
// go to emit(rank, index); returns how many there are. vals: 16-byte aligned, Ap a multiple of 4, entries past the
// last score NaN. hist: the candidates' histogram by key >> shift, consumed; list: kListMax entries.
//  - A suffix sum over the bins finds the bin of the k-th candidate; candidates from that bin up - a few more than
//    k - are collected by one pass over the scores, each into its bin's place in descending bin order, so that a
//    candidate only has to be compared with the few that share its bin to know its rank.
//  - Where that bin holds too many (scores that all lie close together), the candidates above it are ranked as they
//    are and the bin itself is counted again over its own range, nine bits finer, and so on; at single keys the
//    rest are equal scores, taken in index order.
// kFour: four scores of a thread find their places at once, where registers allow it (1024 x 1917 x 21: 158 us, 154).
template <bool kFour, typename Emit>
__device__ __forceinline__ int warp_topk(const float* vals, int Ap, KeySpace ks, int k, unsigned* hist,
                                         unsigned short* list, Emit emit) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    unsigned lo = 0, hi = ks.max_key + 1;          // keys in question: [max(lo, 1), hi)
    int shift = ks.shift, done = 0, left = k;
    for (;;) {
        // lane owns bins [16 * lane, 16 * lane + 16)
        unsigned c[16], sum = 0;
        uint4* h4 = reinterpret_cast<uint4*>(hist + lane * 8);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint4 v = h4[q];
            const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                c[q * 8 + l * 2] = w[l] & 0xffffu;
                c[q * 8 + l * 2 + 1] = w[l] >> 16;
                sum += c[q * 8 + l * 2] + c[q * 8 + l * 2 + 1];
            }
        }
        unsigned incl = sum;                       // this lane's bins and all higher ones
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned t = __shfl_down_sync(full, incl, off);
            if (lane + off < 32) incl += t;
        }
        const unsigned total = __shfl_sync(full, incl, 0);
        unsigned run = incl - sum;
        int edge = -1;                             // the bin the last wanted candidate falls into
        unsigned above = 0, at_edge = 0;
        unsigned start[16];
#pragma unroll
        for (int q = 15; q >= 0; --q) {
            if (run < (unsigned)left && run + c[q] >= (unsigned)left) { edge = lane * 16 + q; above = run; at_edge = c[q]; }
            start[q] = run;
            run += c[q];
        }
        const unsigned who = __ballot_sync(full, edge >= 0);
        const bool all = who == 0;                 // fewer candidates than wanted: every one is taken
        if (all) { edge = 0; above = total; at_edge = 0; }
        else {
            const int src = __ffs(who) - 1;        // exactly one lane finds it
            edge = __shfl_sync(full, edge, src);
            above = __shfl_sync(full, above, src);
            at_edge = __shfl_sync(full, at_edge, src);
        }
        const bool last = at_edge <= (unsigned)kEdgeMax || shift == 0;
        const bool ties = last && at_edge > (unsigned)kEdgeMax;      // single keys: the edge bin holds equal scores
        const bool with_edge = all || (last && !ties);
        const unsigned first_bin = with_edge ? (unsigned)edge : (unsigned)edge + 1u;
        const int m = (int)(with_edge ? above + at_edge : above);    // at most 255 + kEdgeMax, or all of at most k
        if (m > 0) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                h4[q] = make_uint4(start[q * 8] | start[q * 8 + 1] << 16, start[q * 8 + 2] | start[q * 8 + 3] << 16,
                                   start[q * 8 + 4] | start[q * 8 + 5] << 16, start[q * 8 + 6] | start[q * 8 + 7] << 16);
            __syncwarp();
            unsigned from = lo + (first_bin << shift);
            if (from == 0) from = 1;
            const unsigned span = hi - from;
            for (int i = lane * 4; i < Ap; i += 128) {
                const float4 v = *reinterpret_cast<const float4*>(vals + i);
                const float f[4] = {v.x, v.y, v.z, v.w};
                if constexpr (kFour) {
                    // the four places come back one behind the other, not one after the other
                    unsigned pos[4];
                    bool in[4];
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        const unsigned key = __float_as_uint(f[l]) - ks.base;
                        in[l] = key - from < span;
                        const unsigned bin = (key - lo) >> shift, half = (bin & 1u) * 16u;
                        pos[l] = 0;
                        if (in[l]) pos[l] = atomicAdd(&hist[bin >> 1], 1u << half);
                        pos[l] = (pos[l] >> half) & 0xffffu;
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l)
                        if (in[l]) list[pos[l]] = (unsigned short)(i + l);
                } else {
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        const unsigned key = __float_as_uint(f[l]) - ks.base;
                        if (key - from < span) {
                            const unsigned bin = (key - lo) >> shift, half = (bin & 1u) * 16u;
                            const unsigned pos = (atomicAdd(&hist[bin >> 1], 1u << half) >> half) & 0xffffu;
                            list[pos] = (unsigned short)(i + l);
                        }
                    }
                }
            }
            __syncwarp();
            // a bin's candidates now lie in list[end of the bin above, end of the bin)
            for (int p = lane; p < m; p += 32) {
                const int idx = list[p];
                const unsigned bits = __float_as_uint(vals[idx]);
                const unsigned bin = (bits - ks.base - lo) >> shift;
                const int e = (int)hist_get(hist, bin);
                int rank = bin + 1 < (unsigned)kBins ? (int)hist_get(hist, bin + 1) : 0;
                for (int q = rank; q < e; ++q) {
                    const int other = list[q];
                    const unsigned b2 = __float_as_uint(vals[other]);
                    rank += (b2 > bits || (b2 == bits && other < idx)) ? 1 : 0;
                }
                if (rank < left) emit(done + rank, idx);
            }
            __syncwarp();
        }
        if (with_edge) return done + min(m, left);
        done += (int)above;
        left -= (int)above;
        lo += (unsigned)edge << shift;
        if (ties) {
            // equal scores with one key, lo: the first `left` of them by index
            for (int i0 = 0; i0 < Ap && left > 0; i0 += 32) {
                const int i = i0 + lane;
                const bool eq = i < Ap && __float_as_uint(vals[i]) - ks.base == lo;
                const unsigned mask = __ballot_sync(full, eq);
                const int rank = __popc(mask & ((1u << lane) - 1u));
                if (eq && rank < left) emit(done + rank, i);
                const int n = min(__popc(mask), left);
                done += n;
                left -= n;
            }
            return done;
        }
        hi = min(hi, lo + (1u << shift));
        shift = shift > 9 ? shift - 9 : 0;
        h4[0] = make_uint4(0, 0, 0, 0);
        h4[1] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        const unsigned from = lo == 0 ? 1u : lo, span = hi - from;
        for (int i = lane * 4; i < Ap; i += 128) {
            const float4 v = *reinterpret_cast<const float4*>(vals + i);
            const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const unsigned key = __float_as_uint(f[l]) - ks.base;
                if (key - from < span) hist_add(hist, (key - lo) >> shift);
            }
        }
        __syncwarp();
    }
}

struct DetectArgs {
    int N, A, Ap, C, logit_stride, top_k, image_w, image_h;
    int rows_fit;           // a row of logits is read in 128-bit pieces and kept in registers (at most 32 values)
    KeySpace ks;
    float nms_thr;
    int classes_per_pass;   // mode 1: foreground classes whose scores fit in shared memory at once
    int ahead;              // mode 1, kAhead: a block has the image this many further on fetched while it selects (0 = none)
    int parts;              // mode 1: blocks per image, each taking a contiguous range of the foreground classes
    const OgleImageDesc* frames;   // mode 0: per-image frame sizes, or null
    const float4* anchors;         // not null: `boxes` holds deltas, decoded against these as they are written
    float4 var;
};

__device__ __forceinline__ float4 result_box(const DetectArgs& a, const float4* bx, int anchor) {
    const float4 b = bx[anchor];
    return a.anchors ? decode_box(b, a.anchors[anchor], a.var) : b;
}

// The smaller of a score and one. NaN stays NaN and is no candidate: rows with a NaN logit, or with an exponential that
// overflows (inf / inf), have no scores, by either rule. (fminf would give them one in every class.)
__device__ __forceinline__ float at_most_one(float s) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(s), "f"(1.0f));
    return r;
}

// A row of kQuads * 4 - 3 to kQuads * 4 logits in registers by 128-bit loads, its exponentials taken once. How many there
// are is known when this is compiled but for the last three: with up to 32 of them told apart at run time the loops over
// a row were a sixth of the whole selection (1024 images, 1917 anchors, 21 classes 183 us, 154 with 24; 2 classes 77, 41).
template <int kQuads>
__device__ __forceinline__ bool is_class(int j, int C) { return j < kQuads * 4 - 3 || j < C; }
template <int kQuads>
__device__ __forceinline__ void load_row(const float* row, int C, float (&e)[kQuads * 4]) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
        const float4 v = row4[q];
        e[q * 4 + 0] = v.x; e[q * 4 + 1] = v.y; e[q * 4 + 2] = v.z; e[q * 4 + 3] = v.w;
    }
#pragma unroll
    for (int j = 0; j < kQuads * 4; ++j)
        if (is_class<kQuads>(j, C)) e[j] = expf(e[j]);
}
// (for the kernel that has one form for all)
template <int kQuads> struct Quads { static constexpr int value = kQuads; };
// f(Quads<number of 128-bit pieces of a row of C <= 32 logits>)
template <typename F>
__device__ __forceinline__ void by_quads(int C, F f) {
    switch ((C + 3) >> 2) {
        case 1: f(Quads<1>()); break;
        case 2: f(Quads<2>()); break;
        case 3: f(Quads<3>()); break;
        case 4: f(Quads<4>()); break;
        case 5: f(Quads<5>()); break;
        case 6: f(Quads<6>()); break;
        case 7: f(Quads<7>()); break;
        default: f(Quads<8>()); break;
    }
}

// Bytes [0, bytes) at p on their way into L2, a line a thread.
__device__ __forceinline__ void prefetch_l2(const void* p, long bytes) {
    for (long o = (long)threadIdx.x * 128; o < bytes; o += (long)blockDim.x * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(p) + o));
}

// Mode 1: per class. Dynamic shared memory: float scores[classes_per_pass][Ap], histograms of as many classes
// (kHistWords words each), one list of survivors per warp (kListMax 16-bit indices).
// kAhead: what the SM reads next is on its way into L2 while a block selects, at 72 to 96 registers a thread (a block an SM is all
// it is compiled for); else 48, for launches whose shared memory and threads let more blocks onto an SM than that (below).
// kPieces: 128-bit pieces of a row of logits (0: rows that are not read in such). A kernel for each, since the small ones
// otherwise get the registers of the large ones, or spill: 1024 images, 300 anchors, 21 classes 49.6 us with one for all, 45.8.
template <bool kAhead, int kPieces>
__global__ void __launch_bounds__(640, kAhead ? 1 : 2)
ssd_detect_kernel(const float* __restrict__ logits, const float4* __restrict__ boxes,
                  float* __restrict__ out_score, int* __restrict__ out_anchor, int* __restrict__ out_class,
                  float4* __restrict__ out_box, int* __restrict__ out_count, const DetectArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    grid_dependency_trigger();
    grid_dependency_wait();
    const int n = blockIdx.x / a.parts, part = blockIdx.x - n * a.parts;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const float* lg = logits + (long)n * a.A * a.logit_stride;
    const float4* bx = boxes + (long)n * a.A;
    float* scores = reinterpret_cast<float*>(smem);
    unsigned* hists = reinterpret_cast<unsigned*>(scores + (size_t)a.classes_per_pass * a.Ap);
    unsigned short* list = reinterpret_cast<unsigned short*>(hists + (size_t)a.classes_per_pass * kHistWords) + warp * kListMax;
    const int rows = (a.C - 1) * a.top_k;
    if (kAhead && a.ahead > 0) prefetch_l2(bx, (long)a.A * sizeof(float4));
    const int per_part = (a.C - 1 + a.parts - 1) / a.parts;
    const int c_lo = 1 + part * per_part, c_hi = min(a.C, c_lo + per_part);     // this block's classes
    for (int c0 = c_lo; c0 < c_hi; c0 += a.classes_per_pass) {
        const int nc = min(a.classes_per_pass, c_hi - c0);
        for (int i = tid; i < nc * (kHistWords / 4); i += blockDim.x) reinterpret_cast<uint4*>(hists)[i] = make_uint4(0, 0, 0, 0);
        if (a.Ap > a.A)
            for (int j = tid; j < nc * 4; j += blockDim.x)
                if (a.Ap - 4 + (j & 3) >= a.A) scores[(j >> 2) * a.Ap + a.Ap - 4 + (j & 3)] = __int_as_float(0x7fc00000);
        __syncthreads();
        auto put = [&](int j, int i, float s) {
            scores[j * a.Ap + i] = s;
            const unsigned key = __float_as_uint(s) - a.ks.base;
            if (key - 1u < a.ks.max_key) hist_add(hists + j * kHistWords, key >> a.ks.shift);
        };
        // softmax as the reference post-process does it - exp of the raw logits, summed in class
        // order - with the per-class divide replaced by one IEEE reciprocal of the sum and a
        // multiply per class (scores within one ulp of the reference's quotient)
        if constexpr (kPieces > 0) {
            auto rows_of = [&](auto wanted) {
                for (int i = tid; i < a.A; i += blockDim.x) {
                    float e[kPieces * 4];
                    load_row<kPieces>(lg + (long)i * a.logit_stride, a.C, e);
                    float total = 0.f;
#pragma unroll
                    for (int j = 0; j < kPieces * 4; ++j)
                        if (is_class<kPieces>(j, a.C)) total += e[j];
                    const float inv = 1.0f / total;
#pragma unroll
                    for (int j = 1; j < kPieces * 4; ++j)
                        if (wanted(j)) put(j - c0, i, at_most_one(e[j] * inv));
                }
            };
            if (nc == a.C - 1) rows_of([&](int j) { return is_class<kPieces>(j, a.C); });
            else rows_of([&](int j) { return j >= c0 && j < c0 + nc; });
        } else {
            for (int i = tid; i < a.A; i += blockDim.x) {
                const float* row = lg + (long)i * a.logit_stride;
                float total = 0.f;
                for (int j = 0; j < a.C; ++j) total += expf(row[j]);
                const float inv = 1.0f / total;
                for (int j = 0; j < nc; ++j) put(j, i, at_most_one(expf(row[c0 + j]) * inv));
            }
        }
        __syncthreads();
        if (kAhead && a.ahead > 0 && c0 == c_lo && n + a.ahead < a.N)
            prefetch_l2(lg + (long)a.ahead * a.A * a.logit_stride, ((long)(a.A - 1) * a.logit_stride + a.C) * sizeof(float));
        for (int j = warp; j < nc; j += nwarps) {
            const int cls = c0 + j;
            const float* vals = scores + j * a.Ap;
            const long base = (long)n * rows + (long)(cls - 1) * a.top_k;
            const int cnt = warp_topk<kAhead>(vals, a.Ap, a.ks, a.top_k, hists + j * kHistWords, list, [&](int r, int an) {
                out_score[base + r] = vals[an];
                out_anchor[base + r] = an;
                out_class[base + r] = cls;
                out_box[base + r] = result_box(a, bx, an);
            });
            for (int r = cnt + lane; r < a.top_k; r += 32) {
                out_score[base + r] = 0.f;
                out_anchor[base + r] = -1;
                out_class[base + r] = 0;
                out_box[base + r] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (lane == 0) out_count[(long)n * (a.C - 1) + cls - 1] = cnt;
            __syncwarp();
        }
        __syncthreads();
    }
}

// Mode 0: the reference Detector's rule (detector.cc:150-228), one block per image. Dynamic shared memory:
// float scores[Ap], int best[Ap], the histogram, the survivors' list, and of the selected: index, rectangle, keep flag.
__global__ void __launch_bounds__(512)
ssd_detect_rule_kernel(const float* __restrict__ logits, const float4* __restrict__ boxes,
                       float* __restrict__ out_score, int* __restrict__ out_anchor, int* __restrict__ out_class,
                       float4* __restrict__ out_box, int* __restrict__ out_count, const DetectArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_cnt;
    grid_dependency_trigger();
    const int n = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* lg = logits + (long)n * a.A * a.logit_stride;
    const float4* bx = boxes + (long)n * a.A;
    float* scores = reinterpret_cast<float*>(smem);
    int* best = reinterpret_cast<int*>(scores + a.Ap);
    unsigned* hist = reinterpret_cast<unsigned*>(best + a.Ap);
    int4* rect = reinterpret_cast<int4*>(hist + kHistWords);          // [kMaxTopK]
    int* keep = reinterpret_cast<int*>(rect + kMaxTopK);              // [kMaxTopK]
    int* picked = keep + kMaxTopK;                                    // [kMaxTopK]
    unsigned short* list = reinterpret_cast<unsigned short*>(picked + kMaxTopK);
    for (int i = tid; i < kHistWords; i += blockDim.x) hist[i] = 0;
    for (int i = a.A + tid; i < a.Ap; i += blockDim.x) scores[i] = __int_as_float(0x7fc00000);
    __syncthreads();
    grid_dependency_wait();
    auto put = [&](int i, float max_e, float total, int max_id) {
        const float s = max_e / total;
        scores[i] = s;
        best[i] = max_id;
        const unsigned key = __float_as_uint(s) - a.ks.base;
        if (key - 1u < a.ks.max_key) hist_add(hist, key >> a.ks.shift);
    };
    if (a.rows_fit) {
        by_quads(a.C, [&](auto quads) {
            constexpr int kQuads = decltype(quads)::value;
            for (int i = tid; i < a.A; i += blockDim.x) {
                float e[kQuads * 4];
                load_row<kQuads>(lg + (long)i * a.logit_stride, a.C, e);
                float total = e[0], max_e = 0.f;
                int max_id = 0;
#pragma unroll
                for (int j = 1; j < kQuads * 4; ++j)
                    if (is_class<kQuads>(j, a.C)) {
                        total += e[j];
                        if (max_e < e[j]) { max_e = e[j]; max_id = j; }
                    }
                put(i, max_e, total, max_id);
            }
        });
    } else {
        for (int i = tid; i < a.A; i += blockDim.x) {
            const float* row = lg + (long)i * a.logit_stride;
            float total = expf(row[0]), max_e = 0.f;
            int max_id = 0;
            for (int j = 1; j < a.C; ++j) {
                const float e = expf(row[j]);
                total += e;
                if (max_e < e) { max_e = e; max_id = j; }
            }
            put(i, max_e, total, max_id);
        }
    }
    __syncthreads();
    if (warp == 0) {
        const int cnt = warp_topk<true>(scores, a.Ap, a.ks, a.top_k, hist, list, [&](int r, int an) { picked[r] = an; });
        if (lane == 0) s_cnt = cnt;
    }
    __syncthreads();
    const int cnt = s_cnt;
    // integer pixel rectangles of the frame the image came from (detector.cc:179-180,199-214):
    // cv::Rect members are int, so float -> int truncates
    const int image_w = a.frames ? a.frames[n].width : a.image_w;
    const int image_h = a.frames ? a.frames[n].height : a.image_h;
    for (int r = tid; r < cnt; r += blockDim.x) {
        const float4 b = result_box(a, bx, picked[r]);
        const float xmin = b.x * image_w, ymin = b.y * image_h;
        const float xmax = b.z * image_w, ymax = b.w * image_h;
        rect[r] = make_int4((int)xmin, (int)ymin, (int)(xmax - xmin), (int)(ymax - ymin));
        keep[r] = 1;
    }
    __syncthreads();
    // detector.cc:127-148: box j is dropped if ANY earlier box i (dropped or not)
    // overlaps it by more than the threshold; eight threads share a j
    if (a.nms_thr > 0.f) {
        for (int t = tid; t < cnt * 8; t += blockDim.x) {
            const int j = t >> 3;
            const int4 rj = rect[j];
            const float xmin1 = rj.x, ymin1 = rj.y;
            const float xmax1 = rj.x + rj.z, ymax1 = rj.y + rj.w;
            for (int i = t & 7; i < j; i += 8) {
                const int4 ri = rect[i];
                const float xmin0 = ri.x, ymin0 = ri.y;
                const float xmax0 = ri.x + ri.z, ymax0 = ri.y + ri.w;
                const float w = fmaxf(0.0f, fminf(xmax0, xmax1) - fmaxf(xmin0, xmin1));
                const float h = fmaxf(0.0f, fminf(ymax0, ymax1) - fmaxf(ymin0, ymin1));
                const float inter = w * h;
                const float uni = (xmax0 - xmin0) * (ymax0 - ymin0) + (xmax1 - xmin1) * (ymax1 - ymin1) - inter;
                const float iou = uni <= 0.0f ? 0.0f : inter / uni;
                if (iou > a.nms_thr) { keep[j] = 0; break; }
            }
        }
        __syncthreads();
    }
    // ordered compaction of the survivors by warp 0
    if (warp == 0) {
        int nout = 0;
        const long base = (long)n * a.top_k;
        for (int b0 = 0; b0 < cnt; b0 += 32) {
            const int j = b0 + lane;
            const bool k = j < cnt && keep[j];
            const unsigned m = __ballot_sync(0xffffffffu, k);
            if (k) {
                const int pos = nout + __popc(m & ((1u << lane) - 1u));
                const int an = picked[j];
                out_score[base + pos] = scores[an];
                out_anchor[base + pos] = an;
                out_class[base + pos] = best[an];
                out_box[base + pos] = make_float4((float)rect[j].x, (float)rect[j].y, (float)rect[j].z, (float)rect[j].w);
            }
            nout += __popc(m);
        }
        for (int r = nout + lane; r < a.top_k; r += 32) {
            out_score[base + r] = 0.f; out_anchor[base + r] = -1; out_class[base + r] = 0;
            out_box[base + r] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (lane == 0) out_count[n] = nout;
    }
}

}  // namespace ogle

using namespace ogle;

extern "C" {

int ogle_cuda_ssd_decode(const float* pred, const float* anchors, float* out, int N, int A,
                         const float variances[4], ogle_stream_t stream) {
    if (!pred || !anchors || !out || !variances || N <= 0 || A <= 0) return OGLE_ERR_INVALID;
    if (!aligned16(pred) || !aligned16(anchors) || !aligned16(out)) return OGLE_ERR_ALIGNMENT;
    const long total = (long)N * A;
    const float4 var = make_float4(variances[0], variances[1], variances[2], variances[3]);
    launch_overlapped(ssd_decode_kernel, dim3(grid_for(total, 256)), dim3(256), 0, (cudaStream_t)stream,
                      reinterpret_cast<const float4*>(pred), reinterpret_cast<const float4*>(anchors),
                      reinterpret_cast<float4*>(out), total, A, var);
    return finish_launch();
}

typedef void (*DetectKernel)(const float*, const float4*, float*, int*, int*, float4*, int*, const DetectArgs);
#define DETECT_KERNELS(ahead) \
    {ssd_detect_kernel<ahead, 0>, ssd_detect_kernel<ahead, 1>, ssd_detect_kernel<ahead, 2>, ssd_detect_kernel<ahead, 3>, \
     ssd_detect_kernel<ahead, 4>, ssd_detect_kernel<ahead, 5>, ssd_detect_kernel<ahead, 6>, ssd_detect_kernel<ahead, 7>, ssd_detect_kernel<ahead, 8>}

static int launch_detect(const OgleDetectParams* p, const float* logits, const float* boxes, const float* anchors,
                         const float* variances, float* out_score, int* out_anchor, int* out_class, float* out_box,
                         int* out_count, ogle_stream_t stream) {
    if (!p || !logits || !boxes || !out_score || !out_anchor || !out_class || !out_box || !out_count)
        return OGLE_ERR_INVALID;
    if (p->N <= 0 || p->A <= 0 || p->C < 2 || p->top_k <= 0 || p->top_k > kMaxTopK) return OGLE_ERR_INVALID;
    if (p->mode < 0 || p->mode > 1) return OGLE_ERR_INVALID;
    const int ls = p->logit_stride ? p->logit_stride : p->C;
    if (ls < p->C) return OGLE_ERR_INVALID;
    if (!aligned16(boxes) || !aligned16(out_box) || (anchors && !aligned16(anchors))) return OGLE_ERR_ALIGNMENT;
    DetectArgs a = {};
    a.N = p->N; a.A = p->A; a.Ap = up4(p->A); a.C = p->C; a.logit_stride = ls; a.top_k = p->top_k;
    a.rows_fit = p->C <= 32 && (ls & 3) == 0 && ls <= 32 && aligned16(logits);
    a.image_w = p->image_w; a.image_h = p->image_h; a.nms_thr = p->nms_thr;
    a.frames = p->mode == 0 ? p->frame_sizes : nullptr;
    if (a.frames && (reinterpret_cast<uintptr_t>(a.frames) & 7)) return OGLE_ERR_ALIGNMENT;
    a.anchors = reinterpret_cast<const float4*>(anchors);
    if (anchors) a.var = make_float4(variances[0], variances[1], variances[2], variances[3]);
    // scores lie in [0, 1]; a negative threshold lets every one of them pass (base -1: key = bits + 1)
    const float thr = p->score_thr;
    uint32_t bits;
    memcpy(&bits, &thr, sizeof(bits));
    a.ks.base = thr < 0.f ? 0xffffffffu : (thr == 0.f ? 0u : bits);
    a.ks.max_key = thr < 1.f ? 0x3f800000u - a.ks.base : 0u;         // (NaN: nothing passes)
    int range_bits = 0;
    while (range_bits < 32 && (a.ks.max_key >> range_bits) != 0) ++range_bits;
    a.ks.shift = range_bits > 9 ? range_bits - 9 : 0;
    static const size_t kSmemBudget = 224 * 1024;
    static const size_t kSmemRule = 226 * 1024;                      // mode 0: up to 27936 anchors
    int threads;
    size_t smem;
    a.parts = 1;
    if (p->mode == 1) {
        // Two blocks per image, each with half of the foreground classes, when that lets two
        // blocks share an SM and the batch is a few rounds of SMs at most (more, smaller blocks
        // fill the last round better; for large batches the softmax done twice costs more than
        // that gains); one warp per class selects, ~100 registers a thread. An SM has registers for twenty warps: blocks of
        // fewer classes than its share of them take the rest for the softmax (N = 630, 2 classes, 1917 anchors: 105 us
        // with one warp a block, 45 with four).
        const size_t per_warp = kListMax * sizeof(unsigned short);
        const size_t per_class = (size_t)a.Ap * sizeof(float) + kHistWords * sizeof(unsigned);
        const int fg = p->C - 1;
        if (fg >= 8 && p->N <= 4 * kNumSMs) {
            const int half = (fg + 1) / 2;
            if ((size_t)half * (per_class + per_warp) <= 112 * 1024) a.parts = 2;
        }
        const int classes = (fg + a.parts - 1) / a.parts;
        // Where half as many warps as classes have a thread for every row, blocks of those, twice as many to an SM, keep more
        // of their threads busy through the softmax (1024 images, 300 anchors, 21 classes, top 100: 51.8 us, 48.0; 500
        // anchors 74.3, 82.2, so not there).
        int pickers = classes < 20 ? classes : 20;
        if (p->A <= 32 * ((classes + 1) / 2) && (classes + 1) / 2 < pickers) pickers = (classes + 1) / 2;
        const size_t block_bytes = classes * per_class + per_warp * (size_t)pickers + 1024;
        const long waiting = ((long)p->N * a.parts + kNumSMs - 1) / kNumSMs;       // blocks to an SM, and how many fit
        const long fitting = block_bytes < kSmemBudget ? (long)(kSmemBudget / block_bytes) : 1;
        const int share = (int)(20 / (waiting < fitting ? waiting : fitting));
        if (pickers < share) pickers = share;
        threads = 32 * pickers;
        const size_t warp_bytes = per_warp * (size_t)(pickers < classes ? pickers : classes);      // (only who picks needs a list)
        const size_t budget = a.parts == 2 && p->N * a.parts > kNumSMs ? 112 * 1024 : kSmemBudget;
        if (per_class + warp_bytes > budget) return OGLE_ERR_UNSUPPORTED;
        size_t cpp = (budget - warp_bytes) / per_class;
        if (cpp > (size_t)classes) cpp = classes;
        a.classes_per_pass = (int)cpp;
        smem = cpp * per_class + warp_bytes;
    } else {
        threads = 512;
        smem = (size_t)a.Ap * 8 + kHistWords * 4 + kMaxTopK * 6 * sizeof(int) + kListMax * sizeof(unsigned short);
        if (smem > kSmemRule) return OGLE_ERR_UNSUPPORTED;
    }
    static const DetectKernel per_class_kernels[2][9] = {DETECT_KERNELS(false), DETECT_KERNELS(true)};
    const int pieces = a.rows_fit ? (a.C + 3) >> 2 : 0;
    static thread_local int known_device = -1, regs[2][9];           // (0: not asked yet)
    static thread_local bool rule_set;
    int dev = 0;
    cudaGetDevice(&dev);
    if (known_device != dev) {
        memset(regs, 0, sizeof(regs));
        rule_set = false;
        known_device = dev;
    }
    if (p->mode == 0 ? !rule_set : regs[0][pieces] == 0) {
        cudaError_t e = cudaSuccess;
        if (p->mode == 0) {
            e = cudaFuncSetAttribute(ssd_detect_rule_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemRule);
        } else {
            int asked[2];
            for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
                cudaFuncAttributes fa;
                e = cudaFuncSetAttribute(per_class_kernels[i][pieces], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
                if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, per_class_kernels[i][pieces]);
                if (e == cudaSuccess) asked[i] = fa.numRegs;
            }
            if (e == cudaSuccess) { regs[0][pieces] = asked[0]; regs[1][pieces] = asked[1]; }
        }
        if (e != cudaSuccess) { set_last_error(e); return OGLE_ERR_CUDA; }
        if (p->mode == 0) rule_set = true;
    }
    bool wide = false;
    if (p->mode == 1) {
        // The kernel with more registers where that leaves as many blocks on an SM (of its shared memory, threads, and
        // registers by warps and quarters of the SM), or all there are: 1024 images, 1917 anchors, 21 classes 171.4 -> 162.6 us,
        // 12 classes 121.0 -> 109.2, 4000 anchors, 9 classes 229.5 -> 210.3. Where it does not, it loses what the blocks
        // gave (77 registers in every launch: 300 anchors, 21 classes 50.3 -> 70.9, 1917 anchors, 9 classes 92.8 -> 103.7).
        const int waiting = (p->N * a.parts + kNumSMs - 1) / kNumSMs;
        int blocks = (int)(228 * 1024 / (smem + 1024));
        if (blocks > 2048 / threads) blocks = 2048 / threads;
        if (blocks > waiting) blocks = waiting;
        int fit[2];
        for (int i = 0; i < 2; ++i) {
            const int warps = 4 * (16384 / ((regs[i][pieces] + 7) / 8 * 8 * 32)) / (threads / 32);
            fit[i] = blocks < warps ? blocks : warps;
        }
        wide = fit[1] >= fit[0];
        a.ahead = p->N > kNumSMs ? kNumSMs * fit[1] / a.parts : 0;
    }
    const DetectKernel kernel = p->mode != 1 ? ssd_detect_rule_kernel : per_class_kernels[wide ? 1 : 0][pieces];
    launch_overlapped(kernel, dim3(p->N * a.parts), dim3(threads), smem,
                      (cudaStream_t)stream, logits, reinterpret_cast<const float4*>(boxes), out_score, out_anchor, out_class,
                      reinterpret_cast<float4*>(out_box), out_count, a);
    return finish_launch();
}

int ogle_cuda_ssd_detect(const OgleDetectParams* p, const float* logits, const float* boxes,
                         float* out_score, int* out_anchor, int* out_class, float* out_box,
                         int* out_count, ogle_stream_t stream) {
    return launch_detect(p, logits, boxes, nullptr, nullptr, out_score, out_anchor, out_class, out_box, out_count, stream);
}

int ogle_cuda_ssd_decode_detect(const OgleDetectParams* p, const float* logits, const float* pred, const float* anchors,
                                const float variances[4], float* out_score, int* out_anchor, int* out_class,
                                float* out_box, int* out_count, ogle_stream_t stream) {
    if (!anchors || !variances) return OGLE_ERR_INVALID;
    return launch_detect(p, logits, pred, anchors, variances, out_score, out_anchor, out_class, out_box, out_count, stream);
}

}  // extern "C"
