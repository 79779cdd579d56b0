// [yolo] decode + per-class greedy NMS on the device.
//
// Reference semantics (lightnet-train/src/detect.rs): decode_yolo_head (:934-1016) emits one candidate per
// (head, anchor, cell, class) with objectness > thr and confidence = objectness * class_prob > thr, in that
// order; the list is stably sorted by confidence descending (:107) and apply_nms (:1449-1484) walks it: a
// candidate survives unless an earlier survivor of the same class overlaps it with IoU > nms_thr.
//
// Device formulation.  Every candidate gets the 64-bit key (order-preserving confidence bits << 32) |
// ~emission_index; descending key order is exactly the reference's sorted order, ties included.  Greedy NMS
// only ever needs candidates in that order, and only until top_k survivors exist, so they are consumed from
// the top in two stages:
//
//   pool  - two passes over the head tensors.  The first histograms the top 12 key bits of every candidate;
//           a walk down the histogram fixes a key `pool_lo` such that the candidates at or above it are a few
//           times what the survivors still wanted can need; the second pass writes exactly those keys to a
//           compact per-image pool (or, when they fit, straight into the band).  Should one histogram bin hold
//           more than a pool can (massive ties), the selection descends a digit with another pass.
//   band  - inside the pool a radix selection over the compact keys (cheap: the pool sits in L2) cuts bands
//           that fit in shared memory; each band is sorted (a bitonic network mostly in registers) and resolved
//           by one CTA per image in chunks of 512 candidates: each is tested against the survivors of its class
//           bucket, gets a row of bits with the earlier candidates of the chunk that suppress it, and the chunk is
//           resolved in rounds (kept once all its suppressors are out, out once one is kept).
//
// An image stops as soon as it has top_k survivors or runs out of candidates; a pool that is used up before
// that is followed by the next one further down.  The head tensors are the only large input: they are read
// twice per pool, and nothing of their size is written.
//
// At an ordinary threshold all candidates of an image fit in one band, and the selection has nothing to select: a call with a
// threshold of kDirectThr or more therefore starts with the fill pass alone (every candidate straight into the band) and NMS;
// an image with more candidates than a band holds falls back to the two stages above.  Host and device meet once per round: the
// kernels of a round are enqueued back to back (each skips the images that are not in its phase), records and per-image
// outcome are written to page-locked host memory by the NMS kernel itself.
//
// Most of the candidates only need their histogram bin, not their exact bits.  The passes over the heads
// therefore evaluate the class sigmoid with the hardware ex2 / rcp approximations first and fall back to the
// exact evaluation only when the approximate key is within kKeySlack units of a boundary that matters (a bin
// edge, the threshold, the ends of the range being collected).  Everything that is written anywhere -- pool
// and band keys, records -- comes from the exact evaluation: sigmoid, box decode and IoU use single IEEE-754
// operations in the reference's evaluation order, so a CPU evaluating the same expressions gets the same bits.
#include <cooperative_groups.h>

#include <cstdlib>
#include <ctime>

#include "ln_conv_plan.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kMaxHeads = 8;
constexpr int kBandMaxLarge = 16384;  // candidates of one band (sorted in shared memory) when at most 1024 survivors are wanted
constexpr int kBandMaxSmall = 8192;   // ... when more are wanted (their boxes need the room)
constexpr int kChunk = 512;      // candidates resolved together
constexpr int kBins = 4096;      // 12-bit radix digits
constexpr unsigned kPoolChunk = 8192;  // pool keys one block of the pool passes walks
constexpr int kLevels = 6;       // 5 x 12 bits + 4 bits = 64
// Largest distance, in units of the 32-bit confidence key, assumed between the key of the approximate score and
// the key of the exact one.  The approximations are good to a few units (measured by ln_debug_score_key_error).
constexpr unsigned kKeySlack = 256;
constexpr long long kPoolBytesTarget = 1ll << 30;  // pools of one call together, unless every candidate fits in less

enum { PHASE_POOL = 0, PHASE_FILL = 1, PHASE_SELECT = 2, PHASE_BAND = 3, PHASE_DONE = 4 };

// Smallest confidence threshold at which the direct fill is tried first.  Below it a detector head passes far more candidates than
// a band holds (the stress workload at 0.001: 150 k of 2 M per image), and the first pass over the heads would be for nothing; above
// it an overflow is rare and cheap, because a block that finds its image's band full leaves at once.
constexpr float kDirectThr = 0.04f;

struct HeadDev {
    const float* raw;  // [batch][n_anchor*(5+classes)][gh*gw]
    int gw, gh, classes, n_anchor, new_coords;
    // 0 = [yolo]; 1 = activated [yolox] head; 2 = predecoded distribution head ([ppyoloe] / [yolonas]).  Kinds 1 and 2 hold
    // probabilities already (new_coords = 1: values are used as they are) and have one box per cell.
    int kind;
    float scale_x_y;
    float anchors[16];
    int ca_base;  // number of (anchor, cell) slots in earlier heads
};

struct YoloParams {
    HeadDev heads[kMaxHeads];
    int n_heads, batch, total_ca, classes;
    int net_w, net_h, letterbox;
    float thr, nms_thr;
    int k_eff;          // survivors wanted per image
    int max_per_image;  // record capacity
    int band_max;       // capacity of one band
    int pool_max;       // capacity of one pool
    int hist_stride;    // the first histogram of a pool looks at every hist_stride-th block of 256 (anchor, cell) slots
};

struct ImgState {
    unsigned long long hi;       // keys >= hi have been consumed
    unsigned long long lo;       // current band is [lo, hi)
    unsigned long long prefix;   // digits fixed so far by the radix selection in progress (pool or band)
    unsigned long long pool_lo;  // the pool holds every candidate in [pool_lo, hi at the time it was filled)
    int level, phase, cap, above, band_count, kept, exhausted, img_w, img_h;
    int last_gain;   // survivors the previous band added
    int direct;      // the pool being filled is small enough to be the band itself
    int pool_count;  // keys in the pool
    int sampled;     // the histogram in progress is an estimate from a sample of the slots
    // band selection inside a pool starts at the first digit on which the pool's keys differ (all earlier digits = start_prefix)
    int start_level, fresh;
    unsigned long long start_prefix;
};

__device__ __forceinline__ int level_shift(int l) { return l < 5 ? 52 - 12 * l : 0; }
__device__ __forceinline__ int level_bits(int l) { return l < 5 ? 12 : 4; }

__device__ __forceinline__ float head_act(float raw, int new_coords) { return new_coords ? raw : ln_det_sigmoid(raw); }
// The objectness factor of a score.  The distribution heads gate on max(class, objectness * class) (detect.rs:1158-1162), which
// is the class score itself for an objectness in [0, 1]: their factor is 1 (a product with 1 is exact).
__device__ __forceinline__ float score_obj(const HeadDev& h, float raw_obj) { return h.kind == 2 ? 1.0f : head_act(raw_obj, h.new_coords); }

__device__ __forceinline__ unsigned conf_key(float c) {
    unsigned b = __float_as_uint(c);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_conf(unsigned k) {
    unsigned b = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(b);
}

struct Box { float x, y, w, h; };

// detect.rs:1288-1322 decode_bbox followed by :1414-1447 correct_bbox, operation for operation.
__device__ __forceinline__ Box decode_box(const HeadDev& h, const float* img, int a, int idx, int net_w, int net_h, int img_w, int img_h,
                                          int letterbox) {
    const int stride = h.gw * h.gh, epa = h.classes + 5;
    const int row = idx / h.gw, col = idx - row * h.gw;
    const float tx = img[(size_t)(a * epa + 0) * stride + idx], ty = img[(size_t)(a * epa + 1) * stride + idx];
    const float tw = img[(size_t)(a * epa + 2) * stride + idx], th = img[(size_t)(a * epa + 3) * stride + idx];
    const float s = h.scale_x_y, nw = (float)net_w, nh = (float)net_h, iw = (float)img_w, ih = (float)img_h;
    const float half = __fmul_rn(0.5f, __fsub_rn(s, 1.0f));
    float bx, by, bw, bh;
    const float aw = h.anchors[2 * a], ah = h.anchors[2 * a + 1];
    if (h.kind == 2) {  // final centre-size box of modern_yolo_predecode (dense_loss.rs:788)
        bx = tx; by = ty; bw = tw; bh = th;
    } else if (h.kind == 1) {  // decode_yolox_box (lightnet-layers/src/modern_yolo/cpu.rs:461-475), sanitised like cpu.rs:212-217
        const float cw = fminf(fmaxf(ln_finite_or_zero(tw), -10.0f), 10.0f), ch = fminf(fmaxf(ln_finite_or_zero(th), -10.0f), 10.0f);
        bx = ln_finite_or_zero(__fdiv_rn(__fadd_rn((float)col, ln_finite_or_zero(tx)), (float)h.gw));
        by = ln_finite_or_zero(__fdiv_rn(__fadd_rn((float)row, ln_finite_or_zero(ty)), (float)h.gh));
        bw = fmaxf(ln_finite_or_zero(__fdiv_rn(ln_det_expf(cw), (float)h.gw)), 1e-6f);
        bh = fmaxf(ln_finite_or_zero(__fdiv_rn(ln_det_expf(ch), (float)h.gh)), 1e-6f);
    } else {
    bx = __fdiv_rn(__fsub_rn(__fadd_rn((float)col, __fmul_rn(s, head_act(tx, h.new_coords))), half), (float)h.gw);
    by = __fdiv_rn(__fsub_rn(__fadd_rn((float)row, __fmul_rn(s, head_act(ty, h.new_coords))), half), (float)h.gh);
    if (h.new_coords) {
        bw = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(tw, tw), 4.0f), aw), nw);
        bh = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(th, th), 4.0f), ah), nh);
    } else {
        bw = __fdiv_rn(__fmul_rn(ln_det_expf(tw), aw), nw);
        bh = __fdiv_rn(__fmul_rn(ln_det_expf(th), ah), nh);
    }
    }
    float new_w, new_h;
    if (letterbox) {
        if (__fdiv_rn(nw, iw) < __fdiv_rn(nh, ih)) { new_w = nw; new_h = __fdiv_rn(__fmul_rn(ih, nw), iw); }
        else { new_w = __fdiv_rn(__fmul_rn(iw, nh), ih); new_h = nh; }
    } else { new_w = nw; new_h = nh; }
    const float delta_w = __fsub_rn(nw, new_w), delta_h = __fsub_rn(nh, new_h);
    const float ratio_w = __fdiv_rn(new_w, nw), ratio_h = __fdiv_rn(new_h, nh);
    bx = __fdiv_rn(__fsub_rn(bx, __fdiv_rn(__fdiv_rn(delta_w, 2.0f), nw)), ratio_w);
    by = __fdiv_rn(__fsub_rn(by, __fdiv_rn(__fdiv_rn(delta_h, 2.0f), nh)), ratio_h);
    bw = __fdiv_rn(bw, ratio_w);
    bh = __fdiv_rn(bh, ratio_h);
    Box b;
    b.x = __fmul_rn(bx, iw); b.y = __fmul_rn(by, ih); b.w = __fmul_rn(bw, iw); b.h = __fmul_rn(bh, ih);
    return b;
}

// detect.rs:1486-1503 bbox_iou with detection_geometry.rs:14-30 edges: intersection and union, whose quotient it is (0 when the
// intersection is not positive)
__device__ __forceinline__ void box_overlap(const Box& a, const Box& b, float& inter, float& denom) {
    const float al = __fsub_rn(a.x, __fmul_rn(a.w, 0.5f)), at = __fsub_rn(a.y, __fmul_rn(a.h, 0.5f));
    const float ar = __fadd_rn(a.x, __fmul_rn(a.w, 0.5f)), ab = __fadd_rn(a.y, __fmul_rn(a.h, 0.5f));
    const float bl = __fsub_rn(b.x, __fmul_rn(b.w, 0.5f)), bt = __fsub_rn(b.y, __fmul_rn(b.h, 0.5f));
    const float br = __fadd_rn(b.x, __fmul_rn(b.w, 0.5f)), bb = __fadd_rn(b.y, __fmul_rn(b.h, 0.5f));
    const float iw = fmaxf(__fsub_rn(fminf(ar, br), fmaxf(al, bl)), 0.0f), ih = fmaxf(__fsub_rn(fminf(ab, bb), fmaxf(at, bt)), 0.0f);
    inter = __fmul_rn(iw, ih);
    const float aa = __fmul_rn(fmaxf(a.w, 0.0f), fmaxf(a.h, 0.0f)), ba = __fmul_rn(fmaxf(b.w, 0.0f), fmaxf(b.h, 0.0f));
    denom = __fsub_rn(__fadd_rn(aa, ba), inter);
}

__device__ __forceinline__ int find_head(const YoloParams& p, int ca) {
    int h = 0;
    for (int k = 1; k < p.n_heads; ++k)
        if (ca >= p.heads[k].ca_base) h = k;
    return h;
}

// Band size wanted next: four candidates per survivor still wanted, or more when the previous band showed heavier suppression.
__device__ __forceinline__ int band_cap(const YoloParams& p, const ImgState& st) {
    long long want = 4ll * (p.k_eff - st.kept);
    if (st.last_gain >= 0) {
        const long long per = ((long long)st.band_count * 3 / 2) / (st.last_gain > 0 ? st.last_gain : 1) + 1;
        if (per > 4) want = per * (p.k_eff - st.kept);
    }
    return want < 1024 ? 1024 : (want > p.band_max ? p.band_max : (int)want);
}

// Confidence key of objectness * sigmoid(x) as an interval [klo, khi] that contains the exact key (valid for thresholds
// >= 1e-30, see approx_ok below).  Branch-free on the common path:
//   x >= 17   the exact sigmoid is 1, the score is the objectness itself: klo == khi
//   x <= -80  ex2 overflows, the approximate score is 0; the exact one is below 2e-35: both far under the threshold
//   NaN       not handled here: callers send NaN logits to the exact path
__device__ __forceinline__ void approx_score_key(float obj, float x, unsigned& klo, unsigned& khi) {
    const bool sat = x >= 17.0f;
    const float s = sat ? obj : obj * ln_rcp_ftz(1.0f + ln_ex2_ftz(x * -1.44269504f));
    const unsigned k = __float_as_uint(s) | 0x80000000u;  // s >= +0 (or NaN)
    const unsigned d = sat ? 0u : kKeySlack;
    klo = k - d;
    khi = k + d;
}

// The same interval for either kind of head: heads with new_coords take the class value as it is, so their score is one
// exact product and the interval a single key (NaN scores are left to the exact evaluation, which drops them).
__device__ __forceinline__ bool score_key_interval(float obj, float x, int new_coords, bool approx_ok, unsigned& klo, unsigned& khi) {
    if (new_coords) {
        const float conf = __fmul_rn(obj, x);
        klo = khi = conf_key(conf);
        return approx_ok && conf == conf;
    }
    approx_score_key(obj, x, klo, khi);
    return approx_ok && x == x;  // a NaN logit goes to the exact evaluation, whose clamps decide what it means
}

constexpr int kWarpBuf = 512;  // keys one warp of the fill pass buffers in shared memory before it reserves space in the pool

// Range of keys one pass over the heads is interested in, [rlo, rhi] inclusive, from the state of the image.
struct ScanRange {
    unsigned long long rlo, rhi;
    unsigned rlo_ck, rhi_ck;
};
template <int MODE>
__device__ __forceinline__ ScanRange scan_range(const ImgState& st) {
    ScanRange r;
    const int shift = level_shift(st.level), bits = level_bits(st.level);
    r.rhi = st.hi - 1ull;  // hi >= 1 whenever an image is still active
    if (MODE == 1) r.rlo = st.pool_lo;
    else if (st.level == 0) r.rlo = 0ull;
    else {
        r.rlo = st.prefix << (shift + bits);
        const unsigned long long pend = r.rlo | ((1ull << (shift + bits)) - 1ull);
        if (pend < r.rhi) r.rhi = pend;
    }
    r.rlo_ck = (unsigned)(r.rlo >> 32);
    r.rhi_ck = (unsigned)(r.rhi >> 32);
    return r;
}

// Exact key of one candidate, or 0 when it is not a candidate inside [rlo, rhi].
__device__ __forceinline__ unsigned long long exact_key_in_range(const YoloParams& p, const ScanRange& r, float obj, float x, int new_coords,
                                                                 unsigned ca, unsigned c) {
    const float conf = __fmul_rn(obj, head_act(x, new_coords));
    if (!(conf > p.thr)) return 0ull;
    const unsigned eidx = ca * (unsigned)p.classes + c;
    const unsigned long long key = ((unsigned long long)conf_key(conf) << 32) | (unsigned long long)(0xFFFFFFFFu - eidx);
    return (key < r.rlo || key > r.rhi) ? 0ull : key;  // a real key is never 0: its confidence bits are at least 0x80000000
}

// First pass over the head tensors for the images that need a pool: histogram of digit `level` (under `prefix`) of the
// unconsumed candidates (keys < hi).  One thread per (anchor, cell), all classes; blockIdx.y = image.  The common path of
// the class loop is branch-free: the flags of a score are computed unconditionally and only the rare score that needs the
// exact evaluation leaves it.
__global__ void __launch_bounds__(256) yolo_head_hist_kernel(const __grid_constant__ YoloParams p, const ImgState* __restrict__ states,
                                                             unsigned* __restrict__ hist) {
    const int img = blockIdx.y;
    const ImgState st = states[img];
    if (st.phase != PHASE_POOL) return;
    // an estimate is enough to place the pool's lower bound (the fill pass is exact whatever the bound): sampled images
    // histogram one block in hist_stride, offset by the image index
    if (st.sampled && (int)(blockIdx.x % p.hist_stride) != img % p.hist_stride) return;
    __shared__ unsigned s_hist[kBins + 1];  // slot kBins swallows the first, empty run of every thread
    for (int i = threadIdx.x; i <= kBins; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    const int shift = level_shift(st.level), bits = level_bits(st.level);
    const ScanRange r = scan_range<0>(st);
    const unsigned kthr = conf_key(p.thr);
    const bool approx_ok = p.thr >= 1e-30f;  // below that the exact exponential's clamp decides candidates
    const bool level0 = st.level == 0;
    const int ca = blockIdx.x * blockDim.x + threadIdx.x;
    if (ca < p.total_ca) {
        const HeadDev& h = p.heads[find_head(p, ca)];
        const int stride = h.gw * h.gh, new_coords = h.new_coords;
        const int epa = h.classes + 5, local = ca - h.ca_base;
        const int a = local / stride, idx = local - a * stride;
        const float* img_raw = h.raw + (size_t)img * h.n_anchor * epa * stride;
        const float obj = score_obj(h, __ldg(img_raw + (size_t)(a * epa + 4) * stride + idx));
        const float* __restrict__ cls_raw = img_raw + (size_t)(a * epa + 5) * stride + idx;
        if (obj > p.thr) {
            // consecutive classes often fall into the same bin (always, when scores saturate): runs are counted in registers
            unsigned run_bin = kBins, run_len = 0;
            // eight class logits are loaded before any of them is used: eight independent loads in flight per thread
            for (int c0 = 0; c0 < p.classes; c0 += 8) {
                float xs[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) xs[j] = c0 + j < p.classes ? __ldg(cls_raw + (size_t)j * stride) : 0.0f;
                cls_raw += (size_t)8 * stride;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float x = xs[j];
                    unsigned klo, khi;
                    const bool usable = score_key_interval(obj, x, new_coords, approx_ok, klo, khi);
                    const bool out = khi <= kthr || klo > r.rhi_ck || khi < r.rlo_ck;  // certainly not a candidate of interest
                    unsigned bin = klo >> 20;
                    const bool certain = level0 && klo > kthr && khi < r.rhi_ck && bin == (khi >> 20);  // the bin is all this pass needs
                    bool count = usable && !out && certain;
                    if (c0 + j < p.classes && !(usable && (out || certain))) {  // rare
                        const unsigned long long key = exact_key_in_range(p, r, obj, x, new_coords, (unsigned)ca, (unsigned)(c0 + j));
                        count = key != 0ull;
                        bin = (unsigned)(key >> shift) & ((1u << bits) - 1u);
                    }
                    count = count && c0 + j < p.classes;
                    const bool same = bin == run_bin;
                    if (count && !same) {
                        atomicAdd(&s_hist[run_bin], run_len);
                        run_bin = bin;
                        run_len = 0;
                    }
                    run_len += count ? 1u : 0u;
                }
            }
            atomicAdd(&s_hist[run_bin], run_len);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[(size_t)img * kBins + i], s_hist[i]);
}

// Second pass over the heads: write the exact keys of the candidates in [pool_lo, hi) to the pool, or to the band when
// `direct`.  A block first lists the (anchor, cell) slots of its 256 whose objectness reaches the range at all (a class
// probability never exceeds 1 where a sigmoid makes it), then walks (class, listed slot) pairs with all its threads, so
// that a few qualifying cells do not leave most lanes idle.  Keys are buffered per warp in shared memory and written
// out with one reservation per few hundred keys.
__global__ void __launch_bounds__(256) yolo_head_fill_kernel(const __grid_constant__ YoloParams p, const ImgState* __restrict__ states,
                                                             unsigned long long* __restrict__ band, int* __restrict__ band_fill,
                                                             unsigned long long* __restrict__ pool, int* __restrict__ pool_fill,
                                                             unsigned long long* __restrict__ key_and_or) {
    const int img = blockIdx.y;
    const ImgState st = states[img];
    if (st.phase != PHASE_FILL) return;
    __shared__ unsigned long long s_buf[8 * kWarpBuf];
    __shared__ int s_cnt[8];
    __shared__ const float* s_ptr[256];
    __shared__ float s_obj[256];
    __shared__ int s_stride[256];
    __shared__ int s_ca[256];   // slot index, with the head's new_coords flag in bit 31
    __shared__ int s_n, s_over;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* fill = st.direct ? band_fill + img : pool_fill + img;
    const int dst_cap = st.direct ? p.band_max : p.pool_max;
    if (lane == 0) s_cnt[warp] = 0;
    if (threadIdx.x == 0) {
        s_n = 0;
        s_over = *(volatile int*)fill > dst_cap;  // (other blocks are counting it up: one thread decides for the block)
    }
    __syncthreads();
    if (s_over) return;  // overflowed already: the image starts over, what is missing does not matter
    const ScanRange r = scan_range<1>(st);
    const unsigned kthr = conf_key(p.thr);
    const bool approx_ok = p.thr >= 1e-30f;
    unsigned long long* dst = st.direct ? band + (size_t)img * p.band_max : pool + (size_t)img * p.pool_max;
    const int ca = blockIdx.x * blockDim.x + threadIdx.x;
    if (ca < p.total_ca) {
        const HeadDev& h = p.heads[find_head(p, ca)];
        const int stride = h.gw * h.gh, new_coords = h.new_coords;
        const int epa = h.classes + 5, local = ca - h.ca_base;
        const int a = local / stride, idx = local - a * stride;
        const float* img_raw = h.raw + (size_t)img * h.n_anchor * epa * stride;
        const float obj = score_obj(h, __ldg(img_raw + (size_t)(a * epa + 4) * stride + idx));
        if (obj > p.thr && (new_coords || conf_key(obj) >= r.rlo_ck)) {
            const int slot = atomicAdd(&s_n, 1);
            s_ptr[slot] = img_raw + (size_t)(a * epa + 5) * stride + idx;
            s_obj[slot] = obj;
            s_stride[slot] = stride;
            s_ca[slot] = ca | (new_coords ? (int)0x80000000 : 0);
        }
    }
    __syncthreads();
    const int n_listed = s_n;
    if (n_listed == 0) return;
    unsigned long long t_and = ~0ull, t_or = 0ull;  // over the keys this thread emits
    auto emit = [&](unsigned long long key) {
        const int slot = atomicAdd(&s_cnt[warp], 1);  // stays below kWarpBuf, see the flush conditions
        s_buf[warp * kWarpBuf + slot] = key;
        t_and &= key;
        t_or |= key;
    };
    auto publish_and_or = [&]() {
        if (st.direct) return;  // (only the selection inside a pool uses them)
        for (int o = 16; o > 0; o >>= 1) {
            t_and &= __shfl_xor_sync(0xffffffffu, t_and, o);
            t_or |= __shfl_xor_sync(0xffffffffu, t_or, o);
        }
        if (lane == 0 && t_or != 0ull) { atomicAnd(&key_and_or[2 * img], t_and); atomicOr(&key_and_or[2 * img + 1], t_or); }
    };
    auto flush_if = [&](int limit, bool last) -> bool {
        // the warp writes its buffered keys out when the next step could overflow the buffer, and at the end; false (for the whole warp)
        // once the image has overflowed: it starts over, so that the rest of the pass would be for nothing
        __syncwarp();
        const int n = s_cnt[warp];
        if (n > limit || (n > 0 && last)) {
            int at = 0;
            if (lane == 0) at = atomicAdd(fill, n);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (at > dst_cap) return false;
            for (int k = lane; k < n; k += 32)
                if (at + k < dst_cap) dst[at + k] = s_buf[warp * kWarpBuf + k];
            __syncwarp();
            if (lane == 0) s_cnt[warp] = 0;
        }
        __syncwarp();
        return true;
    };
    if (n_listed >= 64) {
        // many listed slots: thread t takes listed slot t and walks its classes, eight loads in flight
        if (warp * 32 >= n_listed) return;
        const bool have = (int)threadIdx.x < n_listed;
        const int j = have ? (int)threadIdx.x : 0;
        const float obj = s_obj[j];
        const int new_coords = s_ca[j] < 0 ? 1 : 0, stride = s_stride[j];
        const unsigned cell = (unsigned)s_ca[j] & 0x7FFFFFFFu;
        const float* __restrict__ cls_raw = s_ptr[j];
        for (int c0 = 0; c0 < p.classes; c0 += 8) {
            if (have) {
                float xs[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) xs[q] = c0 + q < p.classes ? __ldg(cls_raw + (size_t)q * stride) : 0.0f;
                cls_raw += (size_t)8 * stride;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float x = xs[q];
                    unsigned klo, khi;
                    const bool out = score_key_interval(obj, x, new_coords, approx_ok, klo, khi) && (khi <= kthr || khi < r.rlo_ck || klo > r.rhi_ck);
                    if (!out && c0 + q < p.classes) {
                        const unsigned long long key = exact_key_in_range(p, r, obj, x, new_coords, cell, (unsigned)(c0 + q));
                        if (key != 0ull) emit(key);
                    }
                }
            }
            if (!flush_if(kWarpBuf - 256, c0 + 8 >= p.classes)) return;  // a step adds at most 8 x 32 keys
        }
        publish_and_or();
        return;
    }
    // few listed slots: all threads share the (class, listed slot) pairs
    const int items = n_listed * p.classes;
    for (int base = 0; base < items; base += 256) {  // uniform trip count
        const int i = base + (int)threadIdx.x;
        if (i < items) {
            const int c = i / n_listed, j = i - c * n_listed;
            const float obj = s_obj[j];
            const int new_coords = s_ca[j] < 0 ? 1 : 0;
            const unsigned cell = (unsigned)s_ca[j] & 0x7FFFFFFFu;
            const float x = __ldg(s_ptr[j] + (size_t)c * s_stride[j]);
            bool maybe = true;
            unsigned klo, khi;
            if (score_key_interval(obj, x, new_coords, approx_ok, klo, khi)) maybe = !(khi <= kthr || khi < r.rlo_ck || klo > r.rhi_ck);
            if (maybe) {
                const unsigned long long key = exact_key_in_range(p, r, obj, x, new_coords, cell, (unsigned)c);
                if (key != 0ull) emit(key);
            }
        }
        if (!flush_if(kWarpBuf - 32, base + 256 >= items)) return;  // a step adds at most 32 keys
    }
    publish_and_or();
}

// Loads the histogram of one image top bin first into shared memory (and zeroes it in global memory);
// s_part[t] = sum of the 16 slots thread t loaded.  Slot 0 is the top bin.
__device__ __forceinline__ void load_hist_desc(unsigned* h, int nb, unsigned* s_h, unsigned* s_part) {
    const int per = kBins / 256;
    unsigned sum = 0;
    for (int j = 0; j < per; ++j) {
        const int slot = threadIdx.x * per + j;
        const int bin = nb - 1 - slot;
        const unsigned v = bin >= 0 ? h[bin] : 0u;
        s_h[slot] = v;
        sum += v;
        if (bin >= 0) h[bin] = 0u;
    }
    s_part[threadIdx.x] = sum;
    __syncthreads();
}

// One block per image that needs a pool: walk the digit histogram from the top until the candidates counted reach the
// band size wanted; everything from that bin up is the pool.  A bin too large for a pool is descended into.
// With a sampled histogram the counts are estimates (scaled by the sampling stride): the target is doubled, sizes are
// compared with a margin of one half, and an image whose boundary bin looks too large for a pool starts over with the
// full histogram.  The fill pass counts exactly; should it overflow all the same, the image starts over as well.
__global__ void __launch_bounds__(256) yolo_pool_select_kernel(const __grid_constant__ YoloParams p, ImgState* __restrict__ states,
                                                               unsigned* __restrict__ hist) {
    const int img = blockIdx.x;
    ImgState st = states[img];
    if (st.phase != PHASE_POOL) return;
    __shared__ unsigned s_part[256];
    __shared__ unsigned s_h[kBins];
    const int nb = 1 << level_bits(st.level);
    load_hist_desc(hist + (size_t)img * kBins, nb, s_h, s_part);
    if (threadIdx.x != 0) return;
    if (st.level == 0) {
        st.cap = band_cap(p, st);
        st.above = 0;
        st.prefix = 0;
    }
    const long long scale = st.sampled ? p.hist_stride : 1;
    const int shift = level_shift(st.level), bits = level_bits(st.level);
    const long long want = st.sampled ? 2ll * st.cap : (long long)st.cap - st.above;  // > 0
    long long cum = 0;
    int b = -1;
    for (int t = 0; t < 256 && b < 0; ++t) {
        if ((cum + s_part[t]) * scale < want) { cum += s_part[t]; continue; }
        for (int j = 0; j < kBins / 256; ++j) {
            const int slot = t * (kBins / 256) + j;
            if ((cum + s_h[slot]) * scale >= want) { b = nb - 1 - slot; break; }
            cum += s_h[slot];
        }
    }
    const unsigned long long base = st.level == 0 ? 0ull : (st.prefix << (shift + bits));
    long long count;
    if (b < 0) {
        // everything that is left (under this prefix) is fewer than wanted: take all of it
        st.pool_lo = base;
        count = st.above + cum * scale;
    } else {
        const long long incl = st.above + (cum + s_h[nb - 1 - b]) * scale;
        long long fits = st.sampled ? incl + incl / 2 : incl;
        const long long all = (long long)p.total_ca * p.classes;  // an image has no more candidates than this, whatever the estimate says
        if (fits > all) fits = all;
        if (fits <= p.pool_max || (!st.sampled && st.level == kLevels - 1)) {
            st.pool_lo = base + ((unsigned long long)b << shift);
            count = incl;
        } else {
            if (st.sampled) st.sampled = 0;  // same level again, every block this time
            else {
                st.above += (int)cum;
                st.prefix = (st.level == 0 ? 0ull : (st.prefix << bits)) | (unsigned long long)b;
                st.level += 1;
            }
            states[img] = st;
            return;
        }
    }
    st.phase = PHASE_FILL;
    st.direct = (st.sampled ? count + count / 2 : count) <= p.band_max ? 1 : 0;
    if (st.direct) {
        st.lo = st.pool_lo;
        st.band_count = (int)count;
        st.exhausted = 1;
    }
    st.pool_count = 0;
    states[img] = st;
}

// After the fill pass: a filled pool goes to band selection, a directly filled band to NMS.  A fill that found more
// keys than its destination holds (after a histogram, possible only where that was sampled) is thrown away and the image starts
// over with the full histogram.
__global__ void yolo_after_fill_kernel(ImgState* __restrict__ states, int* __restrict__ band_fill, int* __restrict__ pool_fill, int batch,
                                       int band_max, int pool_max, int hist_stride, unsigned long long* __restrict__ key_and_or) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= batch || states[i].phase != PHASE_FILL) return;
    int* fill = states[i].direct ? band_fill + i : pool_fill + i;
    const int n = *fill;
    if (n > (states[i].direct ? band_max : pool_max)) {
        *fill = 0;
        key_and_or[2 * i] = ~0ull;
        key_and_or[2 * i + 1] = 0ull;
        states[i].phase = PHASE_POOL;
        states[i].sampled = 0;
        states[i].level = 0;
        return;
    }
    states[i].sampled = hist_stride > 1 ? 1 : 0;  // for the next pool of this image
    const unsigned long long k_and = key_and_or[2 * i], k_or = key_and_or[2 * i + 1];
    key_and_or[2 * i] = ~0ull;
    key_and_or[2 * i + 1] = 0ull;
    if (states[i].direct) {
        states[i].band_count = n;
        states[i].phase = PHASE_BAND;
    } else {
        // digits on which the AND and the OR of the pool's keys agree are shared by all of them: the selection starts below them
        int level = 0;
        unsigned long long prefix = 0ull;
        const unsigned long long diff = k_and ^ k_or;
        while (n > 0 && level < kLevels - 1) {
            const int sh = level_shift(level), bt = level_bits(level);
            const unsigned long long m = ((1ull << bt) - 1ull) << sh;
            if (diff & m) break;
            prefix = (prefix << bt) | ((k_and & m) >> sh);
            ++level;
        }
        states[i].pool_count = n;
        states[i].phase = PHASE_SELECT;
        states[i].level = states[i].start_level = level;
        states[i].prefix = states[i].start_prefix = prefix;
        states[i].fresh = 1;
    }
}

// Passes over the pool: one thread per two keys; integer work only.
// MODE 0: histogram of digit `level` under `prefix` of the unconsumed keys, plus the AND and OR of those keys (they tell
// the selection which further digits all of them share).  Lanes of a warp that fall into the same bin are merged into one
// shared-memory add.  MODE 1: collect the keys of the band [lo, hi).
template <int MODE>
__global__ void __launch_bounds__(256) yolo_pool_scan_kernel(const __grid_constant__ YoloParams p, const ImgState* __restrict__ states,
                                                             unsigned* __restrict__ hist, unsigned long long* __restrict__ key_and_or,
                                                             unsigned long long* __restrict__ band, int* __restrict__ band_fill,
                                                             const unsigned long long* __restrict__ pool) {
    const int img = blockIdx.y;
    const ImgState st = states[img];
    if (st.phase != (MODE == 0 ? PHASE_SELECT : PHASE_BAND) || (MODE == 1 && st.direct)) return;
    const unsigned n = (unsigned)st.pool_count;
    const unsigned chunk_begin = blockIdx.x * kPoolChunk;
    if (chunk_begin >= n) return;
    __shared__ unsigned s_hist[MODE == 0 ? kBins : 1];
    __shared__ unsigned long long s_and, s_or;
    if (MODE == 0) {
        for (int i = threadIdx.x; i < kBins; i += blockDim.x) s_hist[i] = 0;
        if (threadIdx.x == 0) { s_and = ~0ull; s_or = 0ull; }
        __syncthreads();
    }
    const int shift = level_shift(st.level), bits = level_bits(st.level);
    const unsigned long long* img_pool = pool + (size_t)img * p.pool_max;
    unsigned long long t_and = ~0ull, t_or = 0ull;
    for (unsigned base = chunk_begin; base < chunk_begin + kPoolChunk && base < n; base += 2u * blockDim.x) {  // uniform trip count
        const unsigned i0 = base + 2u * threadIdx.x;
        ulonglong2 v = make_ulonglong2(0ull, 0ull);
        if (i0 + 1 < n) v = *reinterpret_cast<const ulonglong2*>(img_pool + i0);
        else if (i0 < n) v.x = img_pool[i0];
        const unsigned long long ks[2] = {v.x, v.y};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const unsigned long long key = ks[e];
            bool valid = i0 + e < n && key < st.hi;
            if (MODE == 0) {
                valid = valid && (st.level == 0 || (key >> (shift + bits)) == st.prefix);
                unsigned bin = 0xFFFFFFFFu;
                if (valid) {
                    bin = (unsigned)(key >> shift) & ((1u << bits) - 1u);
                    t_and &= key;
                    t_or |= key;
                }
                const unsigned same = __match_any_sync(0xffffffffu, bin);
                if (valid && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&s_hist[bin], (unsigned)__popc(same));
            } else if (valid && key >= st.lo) {
                const int slot = atomicAdd(&band_fill[img], 1);
                if (slot < p.band_max) band[(size_t)img * p.band_max + slot] = key;
            }
        }
    }
    if (MODE == 0) {
        for (int o = 16; o > 0; o >>= 1) {
            t_and &= __shfl_xor_sync(0xffffffffu, t_and, o);
            t_or |= __shfl_xor_sync(0xffffffffu, t_or, o);
        }
        if ((threadIdx.x & 31) == 0) { atomicAnd(&s_and, t_and); atomicOr(&s_or, t_or); }
        __syncthreads();
        for (int b = threadIdx.x; b < kBins; b += blockDim.x)
            if (s_hist[b]) atomicAdd(&hist[(size_t)img * kBins + b], s_hist[b]);
        if (threadIdx.x == 0) { atomicAnd(&key_and_or[2 * img], s_and); atomicOr(&key_and_or[2 * img + 1], s_or); }
    }
}

// One block per image: walk the digit histogram of the pool from the top, either fix the band's lower bound or descend
// into the digit that holds too many candidates (skipping the digits all keys under it share).  Leaves the histogram zeroed.
__global__ void __launch_bounds__(256) yolo_select_kernel(const __grid_constant__ YoloParams p, ImgState* __restrict__ states,
                                                          unsigned* __restrict__ hist, unsigned long long* __restrict__ key_and_or) {
    const int img = blockIdx.x;
    ImgState st = states[img];
    if (st.phase != PHASE_SELECT) return;
    __shared__ unsigned s_part[256];
    __shared__ unsigned s_h[kBins];
    const int nb = 1 << level_bits(st.level);
    const int per = kBins / 256;
    load_hist_desc(hist + (size_t)img * kBins, nb, s_h, s_part);
    if (threadIdx.x != 0) return;
    const unsigned long long k_and = key_and_or[2 * img], k_or = key_and_or[2 * img + 1];
    key_and_or[2 * img] = ~0ull;
    key_and_or[2 * img + 1] = 0ull;
    // ---- one thread decides (a few hundred steps at most)
    if (st.fresh) {  // first pass of this band: level and prefix are the pool's starting point
        st.cap = band_cap(p, st);
        st.above = 0;
        st.fresh = 0;
    }
    const unsigned cap_left = (unsigned)(st.cap - st.above);
    const int shift = level_shift(st.level), bits = level_bits(st.level);
    unsigned cum = 0, everything = 0;
    int owner = -1;
    for (int t = 0; t < 256; ++t) everything += s_part[t];
    for (int t = 0; t < 256; ++t) {
        if (cum + s_part[t] > cap_left) { owner = t; break; }
        cum += s_part[t];
    }
    if (owner < 0) {
        // everything that is left of the pool (under this prefix) fits into the band
        const bool whole_pool = st.level == st.start_level;  // nothing was cut off above this level: the rest of the pool is the band
        st.lo = whole_pool ? st.pool_lo : (st.prefix << (shift + bits));
        st.band_count = st.above + (int)cum;
        st.exhausted = whole_pool ? 1 : 0;
        st.phase = PHASE_BAND;
        states[img] = st;
        return;
    }
    int b = -1;
    for (int j = 0; j < per; ++j) {
        const int slot = owner * per + j;
        if (cum + s_h[slot] > cap_left) { b = nb - 1 - slot; break; }
        cum += s_h[slot];
    }
    const int total = st.above + (int)cum;
    const bool last = st.level == kLevels - 1;
    if (total >= st.cap / 4 || last) {
        const unsigned long long base = st.level == 0 ? 0ull : (st.prefix << (shift + bits));
        st.lo = base + ((unsigned long long)(b + 1) << shift);  // b+1 == nb carries into the digit above: the band is `above` only
        st.band_count = total;
        st.exhausted = 0;
        st.phase = PHASE_BAND;
    } else {
        st.above = total;
        st.prefix = (st.level == 0 ? 0ull : (st.prefix << bits)) | (unsigned long long)b;
        st.level += 1;
        if (s_h[nb - 1 - b] == everything) {
            // every key of this pass sits in bin b: digits on which their AND and OR agree are shared by all of them
            const unsigned long long diff = k_and ^ k_or;
            while (st.level < kLevels - 1) {
                const int sh = level_shift(st.level), bt = level_bits(st.level);
                const unsigned long long m = ((1ull << bt) - 1ull) << sh;
                if (diff & m) break;
                st.prefix = (st.prefix << bt) | ((k_and & m) >> sh);
                st.level += 1;
            }
        }
    }
    states[img] = st;
}

// Sorts the n keys at `src` in descending order into shared memory.  Bitonic network over n_pow2 (a power of two >= n, at most
// 1024 * E) slots with E consecutive slots per thread in registers: distances below E are exchanges inside a thread, below 32 E
// shuffles, and only the rest goes through shared memory (slot e of thread t at e * 1024 + t: no bank conflicts).  Every step
// through shared memory moves the whole array twice and costs two barriers; with 16 K keys 15 of the 105 steps are left there.
template <int E>
__device__ __forceinline__ void block_sort_desc(const unsigned long long* __restrict__ src, int n, int n_pow2, unsigned long long* __restrict__ s) {
    const int t = (int)threadIdx.x;
    unsigned long long r[E];
#pragma unroll
    for (int e = 0; e < E; ++e) r[e] = t * E + e < n ? src[t * E + e] : 0ull;
    for (int k = 2; k <= n_pow2; k <<= 1) {
        int j = k >> 1;
        for (; j >= 32 * E; j >>= 1) {
            __syncthreads();
#pragma unroll
            for (int e = 0; e < E; ++e) s[e * 1024 + t] = r[e];
            __syncthreads();
            const bool keep_max = (((t * E) & j) == 0) == (((t * E) & k) == 0);
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const unsigned long long o = s[e * 1024 + (t ^ (j / E))];
                r[e] = keep_max ? (r[e] > o ? r[e] : o) : (r[e] < o ? r[e] : o);
            }
        }
        for (; j >= E; j >>= 1) {
            const bool keep_max = (((t * E) & j) == 0) == (((t * E) & k) == 0);
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, r[e], j / E);
                r[e] = keep_max ? (r[e] > o ? r[e] : o) : (r[e] < o ? r[e] : o);
            }
        }
#pragma unroll
        for (int jj = E / 2; jj >= 1; jj >>= 1) {
            if (jj > j) continue;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                if (e & jj) continue;
                const bool desc = ((t * E + e) & k) == 0;
                const unsigned long long lo = r[e], hi = r[e | jj];
                const bool swap = desc ? lo < hi : lo > hi;
                r[e] = swap ? hi : lo;
                r[e | jj] = swap ? lo : hi;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) s[t * E + e] = r[e];
    __syncthreads();
}

// box_iou(a, b) > thr with the division left out where it cannot matter: the rounded quotient of positive operands is within a few
// units in the last place of the real one, so a numerator 0.1 % away from thr * denominator decides by itself.
__device__ __forceinline__ bool iou_above(const float4& a4, const float4& b4, float thr) {
    Box a, b;
    a.x = a4.x; a.y = a4.y; a.w = a4.z; a.h = a4.w;
    b.x = b4.x; b.y = b4.y; b.w = b4.z; b.h = b4.w;
    float inter, denom;
    box_overlap(a, b, inter, denom);
    if (inter <= 0.0f) return 0.0f > thr;
    const float edge = thr * denom;
    if (denom > 0.0f && edge > 1e-30f) {
        if (inter < 0.999f * edge) return false;
        if (inter > 1.001f * edge) return true;
    }
    return __fdiv_rn(inter, denom) > thr;
}

constexpr int kBuckets = 128;  // survivors and chunk candidates are looked up by class modulo this

// Shared memory of the NMS kernel: sorted keys, survivors (box, class, list of the bucket), the chunk (box, class, objectness,
// suppressor rows, bucket bitmaps).
constexpr size_t nms_smem_bytes(int band_max, int k_eff) {
    return (size_t)band_max * 8 + (size_t)(k_eff + kChunk) * sizeof(float4) + (size_t)kChunk * (kChunk / 32) * 4 + (size_t)kBuckets * (kChunk / 32) * 4 +
           (size_t)k_eff * 8 + (size_t)kChunk * 12 + (size_t)kBuckets * 4 + 3 * (kChunk / 32) * 4;
}

// One CTA per image: sort the band, then greedy per-class NMS chunk by chunk.  Only candidates of one class can suppress one
// another, so a candidate is compared with the survivors of its class bucket (a linked list, both halves of the CTA taking every
// second entry) and with the earlier candidates of the chunk that share the bucket (128 bitmaps of 512 bits).  The chunk is then
// resolved in rounds instead of candidate by candidate: a candidate with a kept suppressor is out, one whose suppressors are all
// out is kept, and the chains are short.  (One image of 608 x 608 with 900 survivors: 515 us when every candidate was compared with
// every survivor and one warp walked the chunk.)
// Also takes images whose band was filled directly (PHASE_FILL): too many candidates send them back to PHASE_POOL.
// counts[img]: records kept once the image is done, -1 - phase while it is not.
__global__ void __launch_bounds__(1024, 1) yolo_nms_kernel(const __grid_constant__ YoloParams p, ImgState* __restrict__ states,
                                                           const unsigned long long* __restrict__ band, int* __restrict__ band_fill,
                                                           float4* __restrict__ kept_box, int* __restrict__ kept_cls,
                                                           float* __restrict__ records, int* __restrict__ counts) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int W = kChunk / 32;
    static_assert(kChunk * 28 <= kChunk * W * 4, "the record staging of a chunk reuses the suppressor rows");
    const int img = blockIdx.x, tid = (int)threadIdx.x;
    ImgState st = states[img];
    int n = band_fill[img];
    if (st.phase == PHASE_FILL && n > p.band_max) {
        if (tid == 0) {
            band_fill[img] = 0;
            states[img].phase = PHASE_POOL;
            counts[img] = -1 - PHASE_POOL;
        }
        return;
    }
    if (st.phase != PHASE_BAND && st.phase != PHASE_FILL) {
        if (tid == 0 && st.phase != PHASE_DONE) counts[img] = -1 - st.phase;
        return;
    }
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem);    // band_max
    float4* kbox = reinterpret_cast<float4*>(keys + p.band_max);               // k_eff survivors
    float4* cbox = kbox + p.k_eff;                                             // kChunk
    unsigned* mask = reinterpret_cast<unsigned*>(cbox + kChunk);               // kChunk x W words: row i = earlier candidates that suppress i
    unsigned* cbits = mask + kChunk * W;                                       // kBuckets x W words: candidates of the chunk by bucket
    int* kcls = reinterpret_cast<int*>(cbits + kBuckets * W);                  // k_eff
    int* knext = kcls + p.k_eff;                                               // k_eff: next survivor of the bucket, -1 = last
    int* ccls = knext + p.k_eff;                                               // kChunk
    float* cobj = reinterpret_cast<float*>(ccls + kChunk);                     // kChunk
    unsigned* row_words = reinterpret_cast<unsigned*>(cobj + kChunk);          // kChunk: which words of the row are not zero
    int* khead = reinterpret_cast<int*>(row_words + kChunk);                   // kBuckets
    unsigned* alive_words = reinterpret_cast<unsigned*>(khead + kBuckets);     // W
    volatile unsigned* kept_words = alive_words + W;                           // W
    volatile unsigned* out_words = alive_words + 2 * W;                        // W

    if (n > p.band_max) n = p.band_max;
    int n2 = 32;
    while (n2 < n) n2 <<= 1;
    for (int i = tid; i < kBuckets; i += 1024) khead[i] = -1;
    __syncthreads();
    for (int i = tid; i < st.kept; i += 1024) {
        const int c = kept_cls[(size_t)img * p.k_eff + i];
        kbox[i] = kept_box[(size_t)img * p.k_eff + i];
        kcls[i] = c;
        knext[i] = atomicExch(&khead[c % kBuckets], i);
    }
    const unsigned long long* src = band + (size_t)img * p.band_max;
    if (n2 <= 1024) block_sort_desc<1>(src, n, n2, keys);
    else if (n2 == 2048) block_sort_desc<2>(src, n, n2, keys);
    else if (n2 == 4096) block_sort_desc<4>(src, n, n2, keys);
    else if (n2 == 8192) block_sort_desc<8>(src, n, n2, keys);
    else block_sort_desc<16>(src, n, n2, keys);

    int kept = st.kept;
    for (int base = 0; base < n && kept < p.k_eff; base += kChunk) {
        const int m = min(kChunk, n - base);
        const int slot = tid & (kChunk - 1), half = tid / kChunk;  // threads 512 and up help candidate slot
        for (int i = tid; i < kBuckets * W; i += 1024) cbits[i] = 0u;
        if (tid < W) { alive_words[tid] = 0u; kept_words[tid] = 0u; }
        // ---- decode the chunk
        if (tid < kChunk) {
            row_words[tid] = 0u;
            if (tid < m) {
                const unsigned eidx = 0xFFFFFFFFu - (unsigned)(keys[base + tid] & 0xFFFFFFFFull);
                const int cls = (int)(eidx % (unsigned)p.classes), ca = (int)(eidx / (unsigned)p.classes);
                const HeadDev& h = p.heads[find_head(p, ca)];
                const int stride = h.gw * h.gh, epa = h.classes + 5;
                const int local = ca - h.ca_base, a = local / stride, idx = local - a * stride;
                const float* img_raw = h.raw + (size_t)img * h.n_anchor * epa * stride;
                const float obj_raw = img_raw[(size_t)(a * epa + 4) * stride + idx];
                const Box b = decode_box(h, img_raw, a, idx, p.net_w, p.net_h, st.img_w, st.img_h, p.letterbox);
                cbox[tid] = make_float4(b.x, b.y, b.w, b.h);
                ccls[tid] = cls;
                cobj[tid] = head_act(obj_raw, h.new_coords);
            }
        }
        __syncthreads();
        // ---- against the survivors so far
        bool hit = false;
        if (slot < m) {
            const int cls = ccls[slot];
            const float4 b = cbox[slot];
            for (int k = khead[cls % kBuckets]; k >= 0 && !hit; k = knext[k])
                if ((k & 1) == half && kcls[k] == cls) hit = iou_above(kbox[k], b, p.nms_thr);
        }
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (half == 0 && (tid & 31) == 0) out_words[slot >> 5] = bal;
        __syncthreads();
        if (half == 1 && (tid & 31) == 0) out_words[slot >> 5] |= bal;
        __syncthreads();
        const bool alive = tid < m && !((out_words[(tid & (kChunk - 1)) >> 5] >> (tid & 31)) & 1u);
        if (alive) atomicOr(&cbits[(ccls[tid] % kBuckets) * W + (tid >> 5)], 1u << (tid & 31));
        if (tid < kChunk) {
            const unsigned ab = __ballot_sync(0xffffffffu, alive);
            if ((tid & 31) == 0) alive_words[tid >> 5] = ab;
        }
        __syncthreads();
        // ---- suppressor rows: bit j of row i set when the earlier candidate j suppresses i if it is kept
        for (int item = tid; item < kChunk * W; item += 1024) {
            const int i = item / W, wd = item & (W - 1);
            unsigned bitsv = 0u;
            if (i < m && wd <= (i >> 5) && ((alive_words[i >> 5] >> (i & 31)) & 1u)) {
                const int ci = ccls[i];
                unsigned cand = cbits[(ci % kBuckets) * W + wd];
                if (wd == (i >> 5)) cand &= (1u << (i & 31)) - 1u;
                if (cand) {
                    const float4 bi = cbox[i];
                    while (cand) {
                        const int b = __ffs(cand) - 1, j = wd * 32 + b;
                        cand &= cand - 1u;
                        if (ccls[j] == ci && iou_above(cbox[j], bi, p.nms_thr)) bitsv |= 1u << b;
                    }
                    if (bitsv) atomicOr(&row_words[i], 1u << wd);
                }
            }
            mask[item] = bitsv;
        }
        __syncthreads();
        // ---- resolve: facts only ever get added to kept_words / out_words, so reading them while others write is harmless
        bool undecided = alive;
        bool is_kept = false;
        if (tid < W) out_words[tid] = ~alive_words[tid];
        __syncthreads();
        for (int round = 0; round < kChunk; ++round) {  // (every round decides at least the first undecided candidate)
            bool k = false, o = false;
            if (undecided) {
                bool open = false;
                for (unsigned ws = row_words[tid]; ws && !o; ws &= ws - 1u) {
                    const int wd = __ffs(ws) - 1;
                    const unsigned sup = mask[tid * W + wd];
                    o = (sup & kept_words[wd]) != 0u;
                    open = open || (sup & ~out_words[wd]) != 0u;
                }
                k = !o && !open;
                undecided = !(k || o);
                is_kept = is_kept || k;
            }
            if (tid < kChunk) {
                const unsigned kb = __ballot_sync(0xffffffffu, k), ob = __ballot_sync(0xffffffffu, o);
                if ((tid & 31) == 0) {
                    if (kb) kept_words[tid >> 5] |= kb;
                    if (ob) out_words[tid >> 5] |= ob;
                }
            }
            if (!__syncthreads_or(undecided ? 1 : 0)) break;
        }
        // ---- append the new survivors, in order, up to k_eff; their records leave through shared memory as one contiguous range
        const int kept_before = kept;
        int before = 0, total = 0;
        for (int w = 0; w < W; ++w) {
            const int c = __popc(kept_words[w]);
            if (w < (tid >> 5)) before += c;
            total += c;
        }
        kept = min(kept_before + total, p.k_eff);
        float* stage = reinterpret_cast<float*>(mask);
        if (is_kept) {
            const int rank = before + __popc(kept_words[tid >> 5] & ((1u << (tid & 31)) - 1u)), pos = kept_before + rank;
            if (pos < p.k_eff) {
                const float4 b = cbox[tid];
                const int cls = ccls[tid];
                kbox[pos] = b;
                kcls[pos] = cls;
                knext[pos] = atomicExch(&khead[cls % kBuckets], pos);
                kept_box[(size_t)img * p.k_eff + pos] = b;
                kept_cls[(size_t)img * p.k_eff + pos] = cls;
                float* d = stage + rank * 7;  // ln_detection
                d[0] = (float)cls;
                d[1] = key_conf((unsigned)(keys[base + tid] >> 32));
                d[2] = cobj[tid];
                d[3] = b.x; d[4] = b.y; d[5] = b.z; d[6] = b.w;
            }
        }
        __syncthreads();
        float* dst = records + ((size_t)img * p.max_per_image + kept_before) * 7;
        for (int i = tid; i < (kept - kept_before) * 7; i += 1024) dst[i] = stage[i];
        __syncthreads();
    }
    if (tid == 0) {
        st.last_gain = kept - st.kept;
        st.band_count = n;
        st.kept = kept;
        st.hi = st.lo;
        band_fill[img] = 0;
        if (st.kept >= p.k_eff || (st.exhausted && st.pool_lo == 0ull)) st.phase = PHASE_DONE;
        else {
            st.level = 0;
            if (st.exhausted) {  // the pool is used up: the next one starts below it
                st.phase = PHASE_POOL;
                st.prefix = 0;
                st.above = 0;
            } else {
                st.phase = PHASE_SELECT;
                st.level = st.start_level;
                st.prefix = st.start_prefix;
                st.fresh = 1;
            }
        }
        states[img] = st;
        counts[img] = st.phase == PHASE_DONE ? min(kept, p.max_per_image) : -1 - st.phase;
    }
}

// Starts every image: with `direct` by the fill pass over everything above the threshold, else by the histogram of a pool.
__global__ void yolo_init_states_kernel(ImgState* states, unsigned long long* key_and_or, int* fills, const int* img_w, const int* img_h, int batch, int hist_stride,
                                        int direct) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= batch) return;
    ImgState s;
    s.hi = ~0ull; s.lo = 0; s.prefix = 0; s.pool_lo = 0;
    s.level = 0; s.phase = direct ? PHASE_FILL : PHASE_POOL; s.cap = 0; s.above = 0; s.band_count = 0; s.kept = 0; s.exhausted = direct;
    s.img_w = img_w[i]; s.img_h = img_h[i]; s.last_gain = -1; s.direct = direct; s.pool_count = 0; s.sampled = hist_stride > 1 ? 1 : 0;
    s.start_level = 0; s.fresh = 1; s.start_prefix = 0;
    states[i] = s;
    fills[i] = 0;
    fills[batch + i] = 0;
    key_and_or[2 * i] = ~0ull;
    key_and_or[2 * i + 1] = 0ull;
}

// Largest distance between the approximate and the exact confidence key over a sweep of logits (debug aid that
// justifies kKeySlack): objectness sweeps [obj_lo, obj_hi], class logit sweeps [x_lo, x_hi].
__global__ void yolo_key_error_kernel(float obj_lo, float obj_hi, float x_lo, float x_hi, int n_obj, int n_x, unsigned* __restrict__ worst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_obj * n_x) return;
    const int io = i / n_x, ix = i - io * n_x;
    const float o = obj_lo + (obj_hi - obj_lo) * ((float)io / (float)(n_obj > 1 ? n_obj - 1 : 1));
    const float x = x_lo + (x_hi - x_lo) * ((float)ix / (float)(n_x > 1 ? n_x - 1 : 1));
    const float obj = ln_det_sigmoid(o);
    unsigned klo, khi;
    approx_score_key(obj, x, klo, khi);
    const unsigned mid = klo + (khi - klo) / 2u;
    const unsigned exact = conf_key(__fmul_rn(obj, ln_det_sigmoid(x)));
    const unsigned d = mid > exact ? mid - exact : exact - mid;
    atomicMax(worst, d);
}

// ---- decode only (parity helper): per (anchor, cell) counts, then ordered writes ---------------
__global__ void yolo_decode_count_kernel(const __grid_constant__ YoloParams p, int img, int* __restrict__ counts) {
    const int ca = blockIdx.x * blockDim.x + threadIdx.x;
    if (ca >= p.total_ca) return;
    const HeadDev& h = p.heads[find_head(p, ca)];
    const int stride = h.gw * h.gh, epa = h.classes + 5;
    const int local = ca - h.ca_base, a = local / stride, idx = local - a * stride;
    const float* img_raw = h.raw + (size_t)img * h.n_anchor * epa * stride;
    const float obj = score_obj(h, img_raw[(size_t)(a * epa + 4) * stride + idx]);
    int n = 0;
    if (obj > p.thr)
        for (int c = 0; c < h.classes; ++c)
            if (__fmul_rn(obj, head_act(img_raw[(size_t)(a * epa + 5 + c) * stride + idx], h.new_coords)) > p.thr) ++n;
    counts[ca] = n;
}
__global__ void yolo_decode_write_kernel(const __grid_constant__ YoloParams p, int img, int img_w, int img_h, const long long* __restrict__ offsets,
                                         ln_detection* __restrict__ out, long long capacity) {
    const int ca = blockIdx.x * blockDim.x + threadIdx.x;
    if (ca >= p.total_ca) return;
    const HeadDev& h = p.heads[find_head(p, ca)];
    const int stride = h.gw * h.gh, epa = h.classes + 5;
    const int local = ca - h.ca_base, a = local / stride, idx = local - a * stride;
    const float* img_raw = h.raw + (size_t)img * h.n_anchor * epa * stride;
    const float obj = score_obj(h, img_raw[(size_t)(a * epa + 4) * stride + idx]);
    const float obj_reported = head_act(img_raw[(size_t)(a * epa + 4) * stride + idx], h.new_coords);
    if (!(obj > p.thr)) return;
    long long o = offsets[ca];
    Box b;
    bool have = false;
    for (int c = 0; c < h.classes; ++c) {
        const float conf = __fmul_rn(obj, head_act(img_raw[(size_t)(a * epa + 5 + c) * stride + idx], h.new_coords));
        if (!(conf > p.thr)) continue;
        if (!have) { b = decode_box(h, img_raw, a, idx, p.net_w, p.net_h, img_w, img_h, p.letterbox); have = true; }
        if (o < capacity) {
            ln_detection d;
            d.class_id = (float)c; d.confidence = conf; d.objectness = obj_reported; d.x = b.x; d.y = b.y; d.w = b.w; d.h = b.h;
            out[o] = d;
        }
        ++o;
    }
}

int fill_params(ln_ctx* ctx, YoloParams* p, const ln_yolo_head* heads, int32_t n_heads, int32_t net_w, int32_t net_h, const char* who) {
    if (n_heads < 1 || n_heads > kMaxHeads) return ln_fail(ctx, LN_ERR_ARG, "%s: between 1 and %d heads are supported", who, kMaxHeads);
    memset(p, 0, sizeof *p);
    p->n_heads = n_heads; p->net_w = net_w; p->net_h = net_h;
    int ca = 0;
    for (int k = 0; k < n_heads; ++k) {
        const ln_yolo_head& s = heads[k];
        if (!s.raw || s.raw->dtype != LN_F32) return ln_fail(ctx, LN_ERR_ARG, "%s: head %d is not an f32 tensor", who, k);
        if (s.n_anchor < 1 || s.n_anchor > 8 || s.classes < 1) return ln_fail(ctx, LN_ERR_ARG, "%s: head %d has %d anchors / %d classes", who, k, s.n_anchor, s.classes);
        // decode_yolo_head's length check (detect.rs:950-959)
        if (s.raw->c != (int64_t)s.n_anchor * (s.classes + 5)) return ln_fail(ctx, LN_ERR_SHAPE, "YOLO head tensor length mismatch: head %d has %lld channels, expected %d", k, (long long)s.raw->c, s.n_anchor * (s.classes + 5));
        if (k > 0 && (s.raw->n != heads[0].raw->n || s.classes != heads[0].classes)) return ln_fail(ctx, LN_ERR_SHAPE, "%s: heads disagree on batch or class count", who);
        HeadDev& h = p->heads[k];
        h.raw = (const float*)s.raw->ptr;
        if (s.kind < 0 || s.kind > 2) return ln_fail(ctx, LN_ERR_ARG, "%s: head %d has kind %d (0 = yolo, 1 = yolox, 2 = predecoded distribution head)", who, k, s.kind);
        if (s.kind != 0 && s.n_anchor != 1) return ln_fail(ctx, LN_ERR_ARG, "%s: head %d is anchor-free and takes n_anchor = 1", who, k);
        h.gw = (int)s.raw->w; h.gh = (int)s.raw->h; h.classes = s.classes; h.n_anchor = s.n_anchor;
        h.kind = s.kind;
        h.new_coords = s.kind != 0 ? 1 : s.new_coords;  // the modern heads hold probabilities already
        h.scale_x_y = s.scale_x_y;
        for (int i = 0; i < 2 * s.n_anchor; ++i) h.anchors[i] = s.anchors[i];
        h.ca_base = ca;
        ca += s.n_anchor * h.gw * h.gh;
    }
    p->total_ca = ca;
    p->classes = heads[0].classes;
    p->batch = (int)heads[0].raw->n;
    if ((int64_t)ca * p->classes >= 0xFFFFFFFFll) return ln_fail(ctx, LN_ERR_UNSUPPORTED, "%s: more than 2^32 candidates per image", who);
    return LN_OK;
}

struct Scratch {
    size_t sz_states, sz_hist, sz_band, sz_fill, sz_kbox, sz_kcls, sz_rec, sz_dims, sz_cnt, sz_andor, sz_pool, total;
};

// Sizes of the working arrays of one call.  pool_entries = 0 picks the pool size: every candidate of an image when that
// keeps the pools of the call within kPoolBytesTarget, otherwise that budget split over the images (at least 65536 keys).
void scratch_layout(YoloParams* p, int pool_entries, Scratch* s) {
    const int64_t B = p->batch;
    const int64_t per_image = (int64_t)p->total_ca * p->classes;
    int64_t pm = pool_entries;
    if (pm <= 0) {
        pm = kPoolBytesTarget / 8 / B;
        if (pm < 65536) pm = 65536;
    }
    if (pm > per_image) pm = per_image;
    if (pm < p->band_max + 1) pm = p->band_max + 1;  // a pool is only used for more than a band holds
    pm = ln_round_up(pm, 2);                         // 16-byte rows
    p->pool_max = (int)pm;
    // sampling pays once an image has many blocks of slots; small images are histogrammed in full
    p->hist_stride = (p->total_ca + 255) / 256 >= 64 ? 8 : 1;
    s->sz_states = (size_t)ln_round_up(B * (int64_t)sizeof(ImgState), 256);
    s->sz_hist = (size_t)B * kBins * 4;
    s->sz_band = (size_t)B * p->band_max * 8;
    s->sz_fill = (size_t)ln_round_up(B * 8, 256);  // band_fill, pool_fill
    s->sz_kbox = (size_t)B * p->k_eff * sizeof(float4);
    s->sz_kcls = (size_t)ln_round_up(B * p->k_eff * 4, 256);
    s->sz_rec = (size_t)ln_round_up(B * p->max_per_image * (int64_t)sizeof(ln_detection), 256);
    s->sz_dims = (size_t)ln_round_up(B * 8, 256);
    s->sz_cnt = (size_t)ln_round_up(B * 4, 256);
    s->sz_andor = (size_t)ln_round_up(B * 16, 256);
    s->sz_pool = (size_t)B * (size_t)pm * 8;
    s->total = s->sz_states + s->sz_hist + s->sz_band + s->sz_fill + s->sz_kbox + s->sz_kcls + s->sz_rec + s->sz_dims + s->sz_cnt + s->sz_andor +
               s->sz_pool;
}

int check_options(ln_ctx* ctx, YoloParams* p, const ln_detect_options* opts, const int32_t* image_w, const int32_t* image_h, int band_max, const char* who) {
    p->thr = opts->confidence_threshold;
    // apply_nms returns at once for a threshold <= 0 (detect.rs:1449-1452): nothing is suppressed.  The kernels test
    // `iou > nms_thr`, which no IoU passes when the threshold is +infinity.
    p->nms_thr = opts->nms_threshold > 0.0f ? opts->nms_threshold : INFINITY;
    p->letterbox = opts->letterbox;
    p->max_per_image = opts->max_per_image;
    p->k_eff = opts->top_k > 0 && opts->top_k < opts->max_per_image ? opts->top_k : opts->max_per_image;
    p->band_max = band_max ? band_max : (p->k_eff <= 1024 ? kBandMaxLarge : kBandMaxSmall);
    if (p->k_eff > 4096) return ln_fail(ctx, LN_ERR_UNSUPPORTED, "%s: at most 4096 detections per image (top_k / max_per_image)", who);
    for (int i = 0; i < p->batch; ++i)
        if (image_w[i] <= 0 || image_h[i] <= 0) return ln_fail(ctx, LN_ERR_ARG, "image dimensions must be positive for network detection decoding");
    return LN_OK;
}

// Page-locked host memory of one call: image sizes in, outcome per image and records out.  Kernels read and write it directly.
size_t stage_bytes(const YoloParams& p) { return (size_t)ln_round_up((int64_t)p.batch * 12, 128) + (size_t)p.batch * p.max_per_image * sizeof(ln_detection); }

// Device address of `bytes` of page-locked host memory that a kernel may write as floats; null when any of it is not (a caller may have
// registered only the beginning of its array, and a kernel that runs past the end faults where a copy would have returned an error).
void* mapped_floats(const ln_ctx* ctx, void* host, size_t bytes) {
    cudaPointerAttributes a;
    const bool ok = cudaPointerGetAttributes(&a, host) == cudaSuccess && a.type == cudaMemoryTypeHost && a.devicePointer;
    (void)cudaGetLastError();  // (an unregistered pointer is not an error here)
    if (!ok || ((uintptr_t)a.devicePointer & 3) != 0) return nullptr;
    CUdeviceptr start = 0;
    size_t size = 0;
    const CUdeviceptr at = (CUdeviceptr)a.devicePointer;
    if (ctx->pointer_attribute(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, at) != CUDA_SUCCESS ||
        ctx->pointer_attribute(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, at) != CUDA_SUCCESS)
        return nullptr;
    return at >= start && at - start <= size && bytes <= size - (at - start) ? a.devicePointer : nullptr;
}

// The whole decode + NMS call over working memory that the caller provides (s.total bytes at `scratch`, 256-byte aligned).
// `stage`: stage_bytes(p) of page-locked memory, or null (sizes and results then go through device memory and copies).
int run_decode_nms(ln_ctx* ctx, const YoloParams& p, const Scratch& s, unsigned char* scratch, const int32_t* image_w, const int32_t* image_h,
                   ln_detection* records_host, int32_t* counts_host, const char* who, void* stage = nullptr) {
    const int B = p.batch;
    unsigned char* q = scratch;
    ImgState* states = (ImgState*)q; q += s.sz_states;
    unsigned* hist = (unsigned*)q; q += s.sz_hist;
    unsigned long long* band = (unsigned long long*)q; q += s.sz_band;
    int* band_fill = (int*)q; int* pool_fill = band_fill + B; q += s.sz_fill;
    float4* kept_box = (float4*)q; q += s.sz_kbox;
    int* kept_cls = (int*)q; q += s.sz_kcls;
    float* records = (float*)q; q += s.sz_rec;
    int* dims = (int*)q; q += s.sz_dims;
    int* counts = (int*)q; q += s.sz_cnt;
    unsigned long long* key_and_or = (unsigned long long*)q; q += s.sz_andor;
    unsigned long long* pool = (unsigned long long*)q;
#define LN_Y(call)                                                                                     \
    do {                                                                                               \
        cudaError_t e__ = (call);                                                                      \
        if (e__ != cudaSuccess) return ln_fail(ctx, LN_ERR_CUDA, "%s: %s: %s", who, #call, cudaGetErrorString(e__)); \
    } while (0)
    const bool dbg = getenv("LN_DEBUG_NMS") != nullptr;
    auto now = []() { timespec ts; clock_gettime(CLOCK_MONOTONIC, &ts); return ts.tv_sec * 1e3 + ts.tv_nsec * 1e-6; };
    const double t_begin = dbg ? now() : 0;
    const int* outcome = counts_host;  // what the host reads after a round
    float* stage_records = nullptr;    // records wait here for the copy into the caller's array
    if (stage) {
        int* st = (int*)stage;
        memcpy(st, image_w, (size_t)B * 4);
        memcpy(st + B, image_h, (size_t)B * 4);
        dims = st;
        counts = st + 2 * B;
        outcome = counts;
        // a caller that passes a page-locked record array gets its records written in place
        if (void* m = mapped_floats(ctx, records_host, (size_t)B * p.max_per_image * sizeof(ln_detection))) records = (float*)m;
        else records = stage_records = (float*)((unsigned char*)stage + ln_round_up((int64_t)B * 12, 128));
    } else {
        LN_Y(cudaMemcpyAsync(dims, image_w, (size_t)B * 4, cudaMemcpyHostToDevice, ctx->stream));
        LN_Y(cudaMemcpyAsync(dims + B, image_h, (size_t)B * 4, cudaMemcpyHostToDevice, ctx->stream));
    }
    const bool direct = p.thr >= kDirectThr;
    yolo_init_states_kernel<<<(B + 127) / 128, 128, 0, ctx->stream>>>(states, key_and_or, band_fill, dims, dims + B, B, p.hist_stride, direct ? 1 : 0);
    ctx->launches++;

    const size_t nms_smem = nms_smem_bytes(p.band_max, p.k_eff);
    LN_Y(cudaFuncSetAttribute(yolo_nms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nms_smem));
    const dim3 scan_grid((p.total_ca + 255) / 256, B);
    const dim3 pool_grid((unsigned)((p.pool_max + kPoolChunk - 1) / kPoolChunk), B);
    const int max_rounds = 1 << 16;
    // with LN_DEBUG_NMS set, every kernel is followed by a synchronize and its wall time is added to its class
    double t_k[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    double t_mark = 0;
    auto tick = [&]() { if (dbg) { cudaStreamSynchronize(ctx->stream); t_mark = now(); } };
    auto tock = [&](int k) { if (dbg) { cudaStreamSynchronize(ctx->stream); t_k[k] += now() - t_mark; } };
    int n_full = 0, n_pool_passes = 0, round = 0;
    bool need_pool = !direct, hist_clear = false;
    for (; round < max_rounds; ++round) {
        if (direct && round == 0) {
            tick();
            yolo_head_fill_kernel<<<scan_grid, 256, 0, ctx->stream>>>(p, states, band, band_fill, pool, pool_fill, key_and_or);
            tock(2);
            ctx->launches++;
            n_full++;
        } else {
            // selection: pools for the images that need one, then a band inside every pool (one digit per round; an image that has to
            // descend another digit sits out the rest of the round)
            if (!hist_clear) {  // (the selections leave the histograms zeroed)
                LN_Y(cudaMemsetAsync(hist, 0, s.sz_hist, ctx->stream));
                hist_clear = true;
            }
            if (need_pool) {
                if (round > 0) LN_Y(cudaMemsetAsync(pool_fill, 0, (size_t)B * 4, ctx->stream));
                tick();
                yolo_head_hist_kernel<<<scan_grid, 256, 0, ctx->stream>>>(p, states, hist);
                tock(0); tick();
                yolo_pool_select_kernel<<<B, 256, 0, ctx->stream>>>(p, states, hist);
                tock(1); tick();
                yolo_head_fill_kernel<<<scan_grid, 256, 0, ctx->stream>>>(p, states, band, band_fill, pool, pool_fill, key_and_or);
                tock(2);
                yolo_after_fill_kernel<<<(B + 127) / 128, 128, 0, ctx->stream>>>(states, band_fill, pool_fill, B, p.band_max, p.pool_max, p.hist_stride, key_and_or);
                ctx->launches += 4;
                n_full += 2;
            }
            tick();
            yolo_pool_scan_kernel<0><<<pool_grid, 256, 0, ctx->stream>>>(p, states, hist, key_and_or, band, band_fill, pool);
            tock(3); tick();
            yolo_select_kernel<<<B, 256, 0, ctx->stream>>>(p, states, hist, key_and_or);
            tock(4); tick();
            yolo_pool_scan_kernel<1><<<pool_grid, 256, 0, ctx->stream>>>(p, states, hist, key_and_or, band, band_fill, pool);
            tock(5);
            ctx->launches += 3;
            ++n_pool_passes;
        }
        tick();
        yolo_nms_kernel<<<B, 1024, nms_smem, ctx->stream>>>(p, states, band, band_fill, kept_box, kept_cls, records, counts);
        tock(6);
        ctx->launches++;
        LN_Y(cudaGetLastError());
        if (!stage) LN_Y(cudaMemcpyAsync(counts_host, counts, (size_t)B * 4, cudaMemcpyDeviceToHost, ctx->stream));
        LN_Y(cudaStreamSynchronize(ctx->stream));
        bool active = false;
        need_pool = false;
        for (int i = 0; i < B; ++i) {
            active = active || outcome[i] < 0;
            need_pool = need_pool || outcome[i] == -1 - PHASE_POOL;
        }
        if (!active) break;
    }
    const double t_loop = dbg ? now() : 0;
    if (dbg) fprintf(stderr, "[ln_yolo] batch %d: %d rounds, %d passes over the heads, %d pool passes; ms: head histogram %.3f, pool select %.3f, head fill %.3f, "
                     "pool histogram %.3f, band select %.3f, band collect %.3f, sort + nms %.3f; band_max %d, pool_max %d, k_eff %d\n",
                     B, round + 1, n_full, n_pool_passes, t_k[0], t_k[1], t_k[2], t_k[3], t_k[4], t_k[5], t_k[6], p.band_max, p.pool_max, p.k_eff);
    if (round == max_rounds) return ln_fail(ctx, LN_ERR_TIMEOUT, "%s: NMS did not finish in %d rounds", who, max_rounds);
    if (stage) {
        memcpy(counts_host, counts, (size_t)B * 4);
        if (stage_records)
            for (int i = 0; i < B; ++i)
                memcpy(records_host + (size_t)i * p.max_per_image, stage_records + (size_t)i * p.max_per_image * 7, (size_t)counts_host[i] * sizeof(ln_detection));
    } else {
        LN_Y(cudaMemcpyAsync(records_host, records, (size_t)B * p.max_per_image * sizeof(ln_detection), cudaMemcpyDeviceToHost, ctx->stream));
        LN_Y(cudaStreamSynchronize(ctx->stream));
    }
    if (dbg) fprintf(stderr, "[ln_yolo] whole call %.3f ms, of which handing over counts and records %.3f ms\n", now() - t_begin, now() - t_loop);
#undef LN_Y
    return LN_OK;
}

}  // namespace

extern "C" {

int32_t ln_yolo_decode_nms(ln_ctx* ctx, const ln_yolo_head* heads, int32_t n_heads, int32_t net_w, int32_t net_h, const int32_t* image_w,
                           const int32_t* image_h, const ln_detect_options* opts, ln_detection* records_host, int32_t* counts_host) {
    const char* who = "ln_yolo_decode_nms";
    if (!ctx || !heads || !image_w || !image_h || !opts || !records_host || !counts_host) return ln_fail(ctx, LN_ERR_ARG, "%s: NULL argument", who);
    if (opts->max_per_image < 1) return ln_fail(ctx, LN_ERR_ARG, "%s: max_per_image must be positive", who);
    YoloParams p;
    int rc = fill_params(ctx, &p, heads, n_heads, net_w, net_h, who);
    if (rc) return rc;
    rc = check_options(ctx, &p, opts, image_w, image_h, 0, who);
    if (rc) return rc;
    Scratch s;
    scratch_layout(&p, ctx->nms_pool_entries, &s);
    cudaSetDevice(ctx->device);
    unsigned char* scratch = (unsigned char*)ln_pool_alloc(ctx, s.total);
    if (!scratch) return LN_ERR_CUDA;
    const size_t need = stage_bytes(p);
    if (ctx->h_stage_bytes < need) {
        if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
        ctx->h_stage = nullptr;
        ctx->h_stage_bytes = 0;
        if (cudaMallocHost(&ctx->h_stage, need) == cudaSuccess) ctx->h_stage_bytes = need;
        else { ctx->h_stage = nullptr; cudaGetLastError(); }  // no pinned memory to be had: read back directly
    }
    rc = run_decode_nms(ctx, p, s, scratch, image_w, image_h, records_host, counts_host, who, ctx->h_stage);
    ln_pool_free(ctx, scratch, s.total);
    return rc;
}

// ---- decode + NMS without any allocation ------------------------------------------------------------
// Working memory of ln_yolo_decode_nms_noalloc: a fixed array that is part of the loaded module.  Every GPU
// that loads this library carries these 64 MiB until the process exits, whether or not the entry point is used.
#define LN_NOALLOC_SCRATCH_BYTES (64u * 1024u * 1024u)
static __device__ __align__(256) unsigned char ln_noalloc_scratch[LN_NOALLOC_SCRATCH_BYTES];
// Device address of the array above, per device ordinal.  In host code the name `ln_noalloc_scratch` is only a
// stand-in for the symbol, not a pointer a kernel could use; the address has to be asked for, once per device.
static unsigned char* g_noalloc_ptr[64] = {nullptr};

int32_t ln_yolo_decode_nms_noalloc(ln_ctx* ctx, const ln_yolo_head* heads, int32_t n_heads, int32_t net_w, int32_t net_h, const int32_t* image_w,
                                   const int32_t* image_h, const ln_detect_options* opts, ln_detection* records_host, int32_t* counts_host) {
    const char* who = "ln_yolo_decode_nms_noalloc";
    if (!ctx || !heads || !image_w || !image_h || !opts || !records_host || !counts_host) return ln_fail(ctx, LN_ERR_ARG, "%s: NULL argument", who);
    if (opts->max_per_image < 1) return ln_fail(ctx, LN_ERR_ARG, "%s: max_per_image must be positive", who);
    if (ctx->device < 0 || ctx->device >= 64) return ln_fail(ctx, LN_ERR_UNSUPPORTED, "%s: device ordinal %d is outside the table of 64", who, ctx->device);
    YoloParams p;
    int rc = fill_params(ctx, &p, heads, n_heads, net_w, net_h, who);
    if (rc) return rc;
    rc = check_options(ctx, &p, opts, image_w, image_h, kBandMaxSmall, who);
    if (rc) return rc;
    // the pool gets what the fixed array has left after the other working arrays, and must hold every candidate of an
    // image: this entry point never takes the extra passes a smaller pool can need
    Scratch s;
    scratch_layout(&p, 0, &s);
    const int64_t per_image = (int64_t)p.total_ca * p.classes;
    if (p.pool_max < per_image || s.total > (size_t)LN_NOALLOC_SCRATCH_BYTES)
        return ln_fail(ctx, LN_ERR_UNSUPPORTED,
                       "%s: this call needs %zu bytes of working memory (batch %d, %lld candidates per image, %d records per image) but the fixed "
                       "array holds %u; use a smaller batch, fewer records, or ln_yolo_decode_nms",
                       who, s.total - s.sz_pool + (size_t)p.batch * (size_t)ln_round_up(per_image, 2) * 8, p.batch, (long long)per_image, p.max_per_image,
                       LN_NOALLOC_SCRATCH_BYTES);
    cudaSetDevice(ctx->device);
    if (!g_noalloc_ptr[ctx->device]) {
        // once per device, with that device current: the address of the module's array on this device
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, ln_noalloc_scratch);
        if (e != cudaSuccess || !ptr) return ln_fail(ctx, LN_ERR_CUDA, "%s: cudaGetSymbolAddress: %s", who, cudaGetErrorString(e));
        g_noalloc_ptr[ctx->device] = (unsigned char*)ptr;
    }
    return run_decode_nms(ctx, p, s, g_noalloc_ptr[ctx->device], image_w, image_h, records_host, counts_host, who);
}

// Debug aid: largest distance (in confidence-key units) between the approximate and the exact score over a sweep.
int32_t ln_debug_score_key_error(ln_ctx* ctx, float obj_lo, float obj_hi, float x_lo, float x_hi, int32_t n_obj, int32_t n_x, uint32_t* worst) {
    if (!ctx || !worst || n_obj < 1 || n_x < 1) return ln_fail(ctx, LN_ERR_ARG, "ln_debug_score_key_error: bad argument");
    cudaSetDevice(ctx->device);
    unsigned* d = (unsigned*)ln_pool_alloc(ctx, 256);
    if (!d) return LN_ERR_CUDA;
    cudaMemsetAsync(d, 0, 4, ctx->stream);
    const long long total = (long long)n_obj * n_x;
    yolo_key_error_kernel<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(obj_lo, obj_hi, x_lo, x_hi, n_obj, n_x, d);
    ctx->launches++;
    cudaError_t e = cudaMemcpyAsync(worst, d, 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    ln_pool_free(ctx, d, 256);
    if (e != cudaSuccess) return ln_fail(ctx, LN_ERR_CUDA, "ln_debug_score_key_error: %s", cudaGetErrorString(e));
    return LN_OK;
}

int32_t ln_ctx_set_nms_pool_entries(ln_ctx* ctx, int64_t entries) {
    if (!ctx || entries < 0 || entries > (1ll << 30)) return ln_fail(ctx, LN_ERR_ARG, "ln_ctx_set_nms_pool_entries: entries must be in [0, 2^30]");
    ctx->nms_pool_entries = (int)entries;
    return LN_OK;
}

int32_t ln_yolo_decode_only(ln_ctx* ctx, const ln_yolo_head* heads, int32_t n_heads, int32_t image_index, int32_t net_w, int32_t net_h,
                            int32_t image_w, int32_t image_h, float confidence_threshold, int32_t letterbox, ln_detection* records_host,
                            int64_t capacity, int64_t* count) {
    if (!ctx || !heads || !records_host || !count) return ln_fail(ctx, LN_ERR_ARG, "ln_yolo_decode_only: NULL argument");
    YoloParams p;
    int rc = fill_params(ctx, &p, heads, n_heads, net_w, net_h, "ln_yolo_decode_only");
    if (rc) return rc;
    if (image_index < 0 || image_index >= p.batch) return ln_fail(ctx, LN_ERR_ARG, "batch index %d is outside YOLO head batch %d", image_index, p.batch);
    if (image_w <= 0 || image_h <= 0) return ln_fail(ctx, LN_ERR_ARG, "image dimensions must be positive for network detection decoding");
    p.thr = confidence_threshold;
    p.letterbox = letterbox;
    cudaSetDevice(ctx->device);
    const int n = p.total_ca;
    int* d_counts = (int*)ln_pool_alloc(ctx, (size_t)n * 4);
    long long* d_off = (long long*)ln_pool_alloc(ctx, (size_t)n * 8);
    ln_detection* d_out = (ln_detection*)ln_pool_alloc(ctx, (size_t)(capacity > 0 ? capacity : 1) * sizeof(ln_detection));
    auto cleanup = [&]() {
        ln_pool_free(ctx, d_counts, (size_t)n * 4);
        ln_pool_free(ctx, d_off, (size_t)n * 8);
        ln_pool_free(ctx, d_out, (size_t)(capacity > 0 ? capacity : 1) * sizeof(ln_detection));
    };
    if (!d_counts || !d_off || !d_out) { cleanup(); return LN_ERR_CUDA; }
    yolo_decode_count_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(p, image_index, d_counts);
    ctx->launches++;
    std::vector<int> h_counts((size_t)n);
    std::vector<long long> h_off((size_t)n);
    cudaError_t e = cudaMemcpyAsync(h_counts.data(), d_counts, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    long long total = 0;
    for (int i = 0; i < n; ++i) { h_off[i] = total; total += h_counts[i]; }
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_off, h_off.data(), (size_t)n * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        yolo_decode_write_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(p, image_index, image_w, image_h, d_off, d_out, capacity);
        ctx->launches++;
        e = cudaGetLastError();
    }
    const long long ncopy = total < capacity ? total : capacity;
    if (e == cudaSuccess && ncopy > 0) e = cudaMemcpyAsync(records_host, d_out, (size_t)ncopy * sizeof(ln_detection), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cleanup();
    if (e != cudaSuccess) return ln_fail(ctx, LN_ERR_CUDA, "ln_yolo_decode_only: %s", cudaGetErrorString(e));
    *count = total;
    return LN_OK;
}

}  // extern "C"
