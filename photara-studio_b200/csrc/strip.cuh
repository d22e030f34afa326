// Front-to-back compositing and its reverse-order adjoint for one strip of a
// tile, as the work of ONE warp (a CTA of 32 threads), shared by the
// single-view and the batched kernels.
//
// Forward numerics follow blend_tile pass 1
// (third_party/splat_drender/src/render_forward.cu:341-416, :508-525):
//   power = gaussian_power(conic, mean - pixel); skip power > 0;
//   alpha = min(alpha_clip, o * exp(power)); skip alpha < 1/255;
//   T' = T (1 - alpha); T' < 1e-4 ends the pixel WITHOUT blending;
//   C += rgb * alpha * T;  out = C + T * bg, alpha_out = 1 - T.
//
// Organisation. A strip is TW columns by (32 / TW) * PX rows: lane l owns
// column l % TW and PX pixels, taken in vertical pairs (f32x2 registers); pair
// p of all lanes covers one band of consecutive rows. With TW = 16 and PX = 8
// a strip is a whole 16x16 tile and a band four rows; frames with few tiles
// take fewer pixels per thread, hence more strips. The strips of a tile share
// nothing, so no barrier is wider than a warp.
//  * The tile's Gaussians arrive in batches of 32 by TMA gathers of their
//    64-byte records (tile::gather4), one batch ahead of the blend.
//  * Lane k tests Gaussian k of the batch against the strip: the row interval
//    of its alpha >= 1/255 ellipse over the strip's columns, widened by a
//    pixel, so the test only drops work that the per-pixel test would drop.
//    One ballot per band makes the visit masks; the blend walks their set bits.
//  * The adjoint walks back from every pixel's recorded last entry and recovers
//    T by T_i = T_{i+1} / (1 - a_i) (the reference restarts from stored
//    32-instance snapshots, render_backward.cu:156-519). A pixel adds only
//    s = o G dL/dalpha and its moments in dy, the refine norm and three colour
//    terms; dx is the lane's own, so the ten partial gradients of a Gaussian
//    are formed once per lane, reduce-scattered over the warp and added to
//    its gradient row by one 10-lane atomic.
// Bound: instruction issue. At 1M Gaussians / 1080p a tile blends about 106 of
// its 1,010 listed Gaussians, nearly all over the whole tile, so time is visits
// times instructions. Before, two-warp CTAs of four pixels per thread shared
// staging and shared-memory accumulators: forward 280 us, adjoint 592 us, now
// 217 and 384 us (at 8.4M / 2160p 903 and 1,991 us, now 663 and 1,228 us; at
// 16K / 256x256 88 and 161 us, now 44 and 114 us).
#pragma once

#include "composite.cuh"
#include "kernels.h"

namespace gsb {

template <int TW, int PX> struct StripGeom {
    static_assert(TW == 8 || TW == 16 || TW == 32, "strip width must be 8, 16 or 32");
    static_assert(PX == 1 || PX % 2 == 0, "one pixel per thread or vertical pairs");
    static constexpr int kRowGroups = 32 / TW;
    static constexpr int kRows = kRowGroups * PX;
    static constexpr int kBands = PX == 1 ? 1 : PX / 2;
    static constexpr int kBandRows = kRows / kBands;
};

constexpr int kStripBatch = 32; // Gaussians per batch: one per lane

// Two batches of records (one blended while the next arrives) and their mbarriers.
struct __align__(128) StripStage {
    SplatRec rec[2][kStripBatch];
    unsigned long long bar[2];
};

// The warp's double-buffered TMA staging.
struct StripFeed {
    StripStage& s;
    const CUtensorMap* map;
    unsigned* err;
    unsigned parity = 0; // bit b: parity of buffer b's next phase

    __device__ __forceinline__ void init() {
        if (lane_id() == 0) {
            mbar_init(&s.bar[0], 1);
            mbar_init(&s.bar[1], 1);
        }
        __syncwarp();
    }
    // Starts the copy of records order[first, first + cnt) into buffer b (its
    // previous batch is no longer read); returns lane k's Gaussian (k < cnt).
    // The last gather repeats the batch's last row where cnt is not a
    // multiple of four.
    __device__ __forceinline__ unsigned issue(int b, const unsigned* __restrict__ order,
                                              unsigned first, int cnt) {
        const int lane = int(lane_id());
        const unsigned id = order[first + unsigned(min(lane, cnt - 1))];
        const int ops = (cnt + 3) >> 2;
        int r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            r[q] = int(__shfl_sync(0xffffffffu, id, (4 * lane + q) & 31));
        if (lane == 0)
            mbar_arrive_expect_tx(&s.bar[b], unsigned(ops) * 4u * unsigned(sizeof(SplatRec)));
        __syncwarp();
        // the warp's reads of the buffer come before the asynchronous writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (lane < ops)
            tma_gather4(&s.rec[b][4 * lane], map, r[0], r[1], r[2], r[3], &s.bar[b]);
        return id;
    }
    // Waits (bounded) for buffer b's batch; false in every lane, with
    // kDevStageTimeout set, if it did not arrive.
    __device__ __forceinline__ bool wait(int b) {
        const bool ok = mbar_wait_bounded(&s.bar[b], (parity >> b) & 1u, kStageWaitLimit);
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane_id() == 0)
                atomicOr(err, kDevStageTimeout);
            mbar_wait_bounded(&s.bar[b], (parity >> b) & 1u, kStageWaitLimit);
            return false;
        }
        parity ^= 1u << b;
        return true;
    }
};

// Bit p: the Gaussian's alpha >= 1/255 ellipse, widened by a pixel, reaches
// band p of the strip with origin (x0, y0). The box of the record bounds the
// columns and rows; the ellipse's rows over the strip's columns (the walk's
// column interval, tiles.cuh:18-179) sharpen it for tilted ones. A NaN counts
// as reaching.
// Both are worked out in 32 bits, and for a tilted needle the determinant
// cancels: with d = det / (xx zz), the box (from the covariance), det here and
// the exponent of the per-pixel test are each off by some 2^-22 / d. Below
// kNeedleDet every band counts as reached. Above it the errors stay under 5e-4
// of an extent squared in all: the threshold is raised by 2e-3, and the box's
// extents, at most 1,205 pixels (the covariance is capped), are within the
// pixel that it is widened by. Without the rule aspects of 1,000 and more lost
// blends (minor axis 0.05 pixels, aspect 3,000: 46 of 41,818 pixels).
constexpr float kNeedleDet = 1.f / 1024.f;

template <int TW, int PX>
__device__ __forceinline__ unsigned strip_bands(const SplatRec& rec, int x0, int y0) {
    using G = StripGeom<TW, PX>;
    const float4 co = rec.co;
    const float2 m = rec.xy;
    const ushort4 box = rec.bounds;
    const float det = co.x * co.z - co.y * co.y;
    if (!(det > kNeedleDet * co.x * co.z))
        return (1u << G::kBands) - 1u;
    if (int(box.x) - 1 >= x0 + TW || int(box.y) + 1 <= x0)
        return 0u;
    const float thr = 2.004f * logf(co.w * 255.f);
    const float ex = sqrtf(thr * co.z / det), ey = sqrtf(thr * co.x / det);
    const float d0 = fmaxf(-ex, float(x0 - 1) - m.x), d1 = fminf(ex, float(x0 + TW) - m.x);
    const float r0 = sqrtf(fmaxf(0.f, co.z * thr - det * d0 * d0));
    const float r1 = sqrtf(fmaxf(0.f, co.z * thr - det * d1 * d1));
    const float ic = 1.f / co.z;
    float lo = fminf(-co.y * d0 - r0, -co.y * d1 - r1) * ic;
    float hi = fmaxf(-co.y * d0 + r0, -co.y * d1 + r1) * ic;
    const float tip = co.y * ey / co.x; // column of the lowest point; the highest is at -tip
    if (!(tip < d0) && !(tip > d1))
        lo = -ey;
    if (!(-tip < d0) && !(-tip > d1))
        hi = ey;
    lo += m.y - 1.f;
    hi += m.y + 1.f;
    unsigned bits = 0;
#pragma unroll
    for (int p = 0; p < G::kBands; ++p) {
        const int ya = y0 + p * G::kBandRows, yb = ya + G::kBandRows;
        if (int(box.z) - 1 < yb && int(box.w) + 1 > ya && !(lo > float(yb - 1)) &&
            !(hi < float(ya)))
            bits |= 1u << p;
    }
    return bits;
}

// The batch's visit masks: bit k of mask[p] is set when Gaussian k reaches
// band p, of `all` when it reaches every band; returns their union.
template <int TW, int PX>
__device__ __forceinline__ unsigned strip_masks(const SplatRec* rec, int cnt, int x0, int y0,
                                                unsigned (&mask)[StripGeom<TW, PX>::kBands],
                                                unsigned& all) {
    const int lane = int(lane_id());
    const unsigned bits = lane < cnt ? strip_bands<TW, PX>(rec[lane], x0, y0) : 0u;
    unsigned any = 0;
    all = 0xffffffffu;
#pragma unroll
    for (int p = 0; p < StripGeom<TW, PX>::kBands; ++p) {
        mask[p] = __ballot_sync(0xffffffffu, (bits >> p) & 1u);
        any |= mask[p];
        all &= mask[p];
    }
    return any;
}

// A pixel that does not blend a Gaussian multiplies its values by zero, which
// an infinity or a NaN would turn into a NaN there. Frames with a colour that is
// not finite (finite_colour, in the preprocess) take a forward with the guarded blend, a
// kernel of its own: both in one slowed the other down (1M / 1080p 217 -> 230
// us, by registers and code that the plain loop then shares).
// The adjoint takes guarded steps in batches with a colour, and strips with a
// gradient, that is not below this bound (products of two such values and an image's size stay
// finite).
constexpr float kTame = 1e15f;

__device__ __forceinline__ bool tame(float a, float b, float c) {
    return fabsf(a) + fabsf(b) + fabsf(c) < kTame;
}

// Whether the batch's colours are all below the bound.
__device__ __forceinline__ bool tame_colours(const SplatRec* rec, int cnt) {
    const float4 c = rec[min(int(lane_id()), cnt - 1)].rgb;
    return __all_sync(0xffffffffu, tame(c.x, c.y, c.z));
}

// Strips by their adjoint work, heaviest first: the forward appends each strip
// to the list of its work class (four classes per power of two, so within a
// quarter of each other) and the adjoint's blocks take the classes in
// descending order, so the kernel's tail is made of the shortest strips.
// Replaces a one-block sort of the tiles between the two (8 us at 8,160
// tiles, 22 us at 32,400).
constexpr int kWorkClasses = kWorkListZeroed;
static_assert(kWorkClasses == 64, "two classes per lane");

struct StripOrder {
    unsigned* count = nullptr; // [kWorkClasses], zero before the forward
    unsigned* list = nullptr;  // [kWorkClasses][strips]
    unsigned strips = 0;
};

__device__ __forceinline__ void strip_order_add(const StripOrder& o, unsigned strip,
                                                unsigned work) {
    if (work == 0) // no pixel blended anything: the adjoint has nothing to do
        return;
    const int e = 31 - __clz(int(work));
    const int m = int(e >= 2 ? work >> (e - 2) : work << (2 - e)) & 3;
    const int cls = kWorkClasses - 1 - min(kWorkClasses - 1, 4 * e + m);
    o.list[size_t(cls) * o.strips + atomicAdd(&o.count[cls], 1u)] = strip;
}

// The strip at place `rank` of the descending order (every lane of a warp
// calls this); ~0u past the end.
__device__ __forceinline__ unsigned strip_order_get(const StripOrder& o, unsigned rank) {
    const unsigned lane = lane_id();
    const uint2 c = reinterpret_cast<const uint2*>(o.count)[lane];
    const unsigned incl = warp_incl_scan(c.x + c.y);
    const unsigned before = __ballot_sync(0xffffffffu, incl <= rank);
    const int src = __popc(before);
    if (src == 32)
        return 0xffffffffu;
    unsigned at = rank - __shfl_sync(0xffffffffu, incl - c.x - c.y, src);
    const unsigned cx = __shfl_sync(0xffffffffu, c.x, src);
    const unsigned cls = 2u * unsigned(src) + (at >= cx ? 1u : 0u);
    if (at >= cx)
        at -= cx;
    return o.list[size_t(cls) * o.strips + at];
}

// Checkpoints of a training forward, for frames with so few tiles that the
// adjoint's time is the longest strip's serial walk: the list positions are cut
// into segments of kSegment (the last level takes the rest), and at the end of
// each one the forward stores, per pixel, the colour blended inside it and the
// transmittance left. The adjoint then walks every segment of a strip in its own
// warp: it starts from the stored transmittance, and the colour behind is the
// sum over the later segments (no differences of large sums are taken).
constexpr int kSegment = 64;
static_assert(kSegment % kStripBatch == 0, "segments end with a batch");

struct Checkpoints {
    float4* data = nullptr;      // [levels][H * W] colour in the segment, T at its end
    unsigned* tile_last = nullptr; // [tiles], zero before the forward: largest pix_last
    int levels = 0;
};

// ---------------------------------------------------------------- forward --
// A Gaussian's exponent at a vertical pixel pair, in gaussian_power's rounding
// (element by element on f32x2 instructions).
__device__ __forceinline__ float2 pair_power(float4 co, float dx, float xx, float nxy, float2 dy) {
    const float2 yy = __fmul2_rn(__fmul2_rn(f2s(co.z), dy), dy);
    return __fadd2_rn(__fmul2_rn(f2s(-0.5f), __ffma2_rn(f2s(dx), f2s(xx), yy)),
                      __fmul2_rn(f2s(nxy), dy));
}

// min(clip, o exp(power)) at the pair, 0 where the power or the 1/255 test
// drops the Gaussian.
__device__ __forceinline__ float2 pair_alpha(float4 co, float dx, float xx, float nxy, float2 dy,
                                             float clip) {
    const float2 power = pair_power(co, dx, xx, nxy, dy);
    const float2 og = __fmul2_rn(f2s(co.w), f2(expf(power.x), expf(power.y)));
    const float2 a = f2(fminf(clip, og.x), fminf(clip, og.y));
    return f2(!(power.x > 0.f) && !(a.x < kAlphaFloor) ? a.x : 0.f,
              !(power.y > 0.f) && !(a.y < kAlphaFloor) ? a.y : 0.f);
}

// Blends the pair, in draw order. A dropped Gaussian has alpha 0 and leaves T
// as it was (a live T is at least 1e-4, so it passes the test). A pixel that
// has ended keeps its transmittance with the sign set: its T (1 - alpha) is
// negative, so it never passes again and needs no flag. la, lb: 1 + position
// of the last Gaussian taken while the pixel was open, at or behind the last
// one blended (testing the weight instead: forward at 1M / 1080p 214 -> 228
// us, the adjoint's walk no shorter where pixels fill up). Returns the bits of
// the pair's blend weights (zero apart from the sign: nothing blended).
// Selects on values instead of flags kept across the pairs: eight pixels'
// flags exceed the predicate registers and were moved through general ones
// (179 ALU instructions per visit of a whole tile).
// kSeg: also adds the blend to the segment's colour sums. kGuard: the colour
// reaches the pixels that blend it only (see finite_colour).
struct SegSums {
    float2 r, g, b;
};

template <bool kSeg, bool kGuard>
__device__ __forceinline__ int pair_blend(float2 a, float4 c, unsigned pos, float2& T, float2& r,
                                          float2& g, float2& b, unsigned& la, unsigned& lb,
                                          SegSums& seg) {
    const float2 tt = __fmul2_rn(T, __ffma2_rn(a, f2s(-1.f), f2s(1.f)));
    const bool ba = !(tt.x < kTransmittanceFloor);
    const bool bb = !(tt.y < kTransmittanceFloor);
    const float2 w = __fmul2_rn(f2(ba ? a.x : 0.f, bb ? a.y : 0.f), T);
    auto at = [&](float v) {
        return kGuard ? f2(w.x > 0.f ? v : 0.f, w.y > 0.f ? v : 0.f) : f2s(v);
    };
    r = __ffma2_rn(at(c.x), w, r);
    g = __ffma2_rn(at(c.y), w, g);
    b = __ffma2_rn(at(c.z), w, b);
    if constexpr (kSeg) {
        seg.r = __ffma2_rn(at(c.x), w, seg.r);
        seg.g = __ffma2_rn(at(c.y), w, seg.g);
        seg.b = __ffma2_rn(at(c.z), w, seg.b);
    }
    T.x = ba ? tt.x : -fabsf(T.x);
    T.y = bb ? tt.y : -fabsf(T.y);
    la = ba ? pos : la;
    lb = bb ? pos : lb;
    return __float_as_int(w.x) | __float_as_int(w.y);
}

// Forward of the strip with origin (x0, y0) over instances [range.x, range.y)
// of `order`. kCount: also adds to *pairs the (Gaussian, pixel) pairs whose
// alpha test runs on a pixel that has not ended, for the roofline figures.
// sched (count may be NULL): receives the strip (index `strip`) with its
// adjoint work. False: the staging gave up (the strip was not written).
// kSeg: stores the checkpoints and adds the strip to tile_last[tile]. kGuard:
// the guarded blend (one pixel per thread guards its blend anyway).
template <int TW, int PX, bool kCount = false, bool kSeg = false, bool kGuard = false>
__device__ __forceinline__ bool composite_forward_strip(
    StripFeed& feed, int x0, int y0, uint2 range, const unsigned* __restrict__ order,
    const ViewTarget& o, float* __restrict__ visibility, const StripOrder& sched, unsigned strip,
    unsigned long long* __restrict__ pairs = nullptr, const Checkpoints* cp = nullptr,
    int tile = 0) {
    using G = StripGeom<TW, PX>;
    constexpr int NP = G::kBands;
    constexpr unsigned full = 0xffffffffu;
    const int lane = int(lane_id());
    const int px = x0 + lane % TW;
    const int py = y0 + (PX == 1 ? 1 : 2) * (lane / TW); // pair p adds p * kBandRows
    const float fx = float(px);
    const float clip = o.clip;
    // a clip below the blend threshold blends nothing
    const int n = clip < kAlphaFloor ? 0 : int(range.y - range.x);

    // Pixels outside the image count as ended.
    float2 T[NP], r[NP], g[NP], b[NP], nfy[NP];
    unsigned la[NP], lb[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int y = py + p * G::kBandRows;
        T[p] = f2(px < o.width && y < o.height ? 1.f : -1.f,
                  PX > 1 && px < o.width && y + 1 < o.height ? 1.f : -1.f);
        r[p] = g[p] = b[p] = f2s(0.f);
        nfy[p] = f2(-float(y), -float(y + 1));
        la[p] = lb[p] = 0;
    }
    auto ended = [&]() {
        int s = -1;
#pragma unroll
        for (int p = 0; p < NP; ++p)
            s &= __float_as_int(T[p].x) & (PX > 1 ? __float_as_int(T[p].y) : -1);
        return s < 0;
    };
    unsigned long long evaluated = 0;
    SegSums seg[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p)
        seg[p].r = seg[p].g = seg[p].b = f2s(0.f);
    // Stores segment `level`'s sums and the transmittance, and starts the next.
    auto checkpoint = [&](int level) {
        float4* dst = cp->data + size_t(level) * o.width * o.height;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
#pragma unroll
            for (int q = 0; q < (PX > 1 ? 2 : 1); ++q) {
                const int y = py + p * G::kBandRows + q;
                if (px < o.width && y < o.height)
                    dst[size_t(y) * o.width + px] =
                        make_float4(q ? seg[p].r.y : seg[p].r.x, q ? seg[p].g.y : seg[p].g.x,
                                    q ? seg[p].b.y : seg[p].b.x, fabsf(q ? T[p].y : T[p].x));
            }
            seg[p].r = seg[p].g = seg[p].b = f2s(0.f);
        }
    };
    int level = 0;

    bool more = n > 0 && !__all_sync(full, ended());
    unsigned id_next = 0;
    if (more)
        id_next = feed.issue(0, order, range.x, min(kStripBatch, n));
    int buf = 0;
    for (int base = 0; more; base += kStripBatch) {
        const int cnt = min(kStripBatch, n - base);
        const unsigned id = id_next;
        const int left = n - base - kStripBatch;
        if (left > 0)
            id_next = feed.issue(buf ^ 1, order, range.x + unsigned(base + kStripBatch),
                                 min(kStripBatch, left));
        if (!feed.wait(buf)) {
            if (left > 0)
                feed.wait(buf ^ 1);
            return false;
        }
        const SplatRec* rec = feed.s.rec[buf];
        unsigned mask[NP], all;
        unsigned m = strip_masks<TW, PX>(rec, cnt, x0, y0, mask, all);
        unsigned seen = 0; // Gaussians of the batch this lane blended
        int visit = 0;
        if constexpr (PX == 1) {
            // One pixel per thread (frames with few tiles, where a strip's
            // serial walk is the time): four Gaussians per step, their
            // opacities computed together, the blends in order.
            constexpr int U = 4;
            while (m) {
                int j[U];
                bool ok[U];
                float a[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    ok[u] = m != 0;
                    j[u] = ok[u] ? __ffs(int(m)) - 1 : j[u ? u - 1 : 0];
                    m &= m - 1;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float2 xy = rec[j[u]].xy;
                    const float4 co = rec[j[u]].co;
                    const float power = gaussian_power(co, xy.x - fx, xy.y + nfy[0].x);
                    a[u] = fminf(clip, co.w * expf(power));
                    if (!ok[u] || power > 0.f || a[u] < kAlphaFloor)
                        a[u] = 0.f;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if constexpr (kCount)
                        evaluated += ok[u] && T[0].x > 0.f ? 1u : 0u;
                    const float tt = T[0].x * (1.f - a[u]);
                    const bool bl = !(tt < kTransmittanceFloor);
                    const float w = (bl ? a[u] : 0.f) * T[0].x;
                    const float4 c = rec[j[u]].rgb;
                    if (w > 0.f) {
                        r[0].x += c.x * w;
                        g[0].x += c.y * w;
                        b[0].x += c.z * w;
                        if constexpr (kSeg) {
                            seg[0].r.x += c.x * w;
                            seg[0].g.x += c.y * w;
                            seg[0].b.x += c.z * w;
                        }
                    }
                    T[0].x = bl ? tt : -fabsf(T[0].x);
                    la[0] = bl ? unsigned(base + j[u] + 1) : la[0];
                    seen |= w > 0.f ? 1u << j[u] : 0u;
                }
                if (__all_sync(full, T[0].x < 0.f))
                    break;
            }
        } else {
            while (m) {
                const int j = __ffs(int(m)) - 1;
                m &= m - 1;
                const float2 xy = rec[j].xy;
                const float4 co = rec[j].co;
                const float4 c = rec[j].rgb;
                const float dx = xy.x - fx;
                const float xx = __fmul_rn(co.x, dx);
                const float nxy = -__fmul_rn(co.y, dx);
                const unsigned pos = unsigned(base + j + 1);
                if constexpr (kCount) {
#pragma unroll
                    for (int p = 0; p < NP; ++p)
                        if ((mask[p] >> j) & 1u)
                            evaluated += (T[p].x > 0.f ? 1u : 0u) + (T[p].y > 0.f ? 1u : 0u);
                }
                int bl = 0;
                if ((all >> j) & 1u) {
                    // every band: the pairs' opacities are independent
                    float2 e[NP];
#pragma unroll
                    for (int p = 0; p < NP; ++p)
                        e[p] = pair_alpha(co, dx, xx, nxy, __fadd2_rn(f2s(xy.y), nfy[p]), clip);
#pragma unroll
                    for (int p = 0; p < NP; ++p)
                        bl |= pair_blend<kSeg, kGuard>(e[p], c, pos, T[p], r[p], g[p], b[p], la[p],
                                                       lb[p], seg[p]);
                } else {
#pragma unroll
                    for (int p = 0; p < NP; ++p)
                        if ((mask[p] >> j) & 1u)
                            bl |= pair_blend<kSeg, kGuard>(
                                pair_alpha(co, dx, xx, nxy, __fadd2_rn(f2s(xy.y), nfy[p]), clip),
                                c, pos, T[p], r[p], g[p], b[p], la[p], lb[p], seg[p]);
                }
                seen |= (bl << 1) != 0 ? 1u << j : 0u;
                if ((++visit & 3) == 0 && __all_sync(full, ended()))
                    break;
            }
        }
        if (visibility) {
            const unsigned vis = __reduce_or_sync(full, seen);
            if ((vis >> lane) & 1u)
                visibility[id] = 1.f;
        }
        more = left > 0;
        if (more && __all_sync(full, ended())) {
            feed.wait(buf ^ 1); // the copy in flight lands before the CTA leaves
            more = false;
        }
        if constexpr (kSeg) {
            if (!more)
                checkpoint(level);
            else if ((base + kStripBatch) % kSegment == 0 && level + 1 < cp->levels)
                checkpoint(level++);
        }
        buf ^= 1;
    }
    if constexpr (kCount)
        warp_count_add(evaluated, pairs);
    if constexpr (kSeg) {
        unsigned wl = 0;
#pragma unroll
        for (int p = 0; p < NP; ++p)
            wl = max(wl, max(la[p], lb[p]));
        wl = __reduce_max_sync(full, wl);
        if (lane == 0 && wl)
            atomicMax(cp->tile_last + tile, wl);
    }
    if (sched.count) {
        unsigned wl = 0;
#pragma unroll
        for (int p = 0; p < NP; ++p)
            wl = max(wl, max(la[p], lb[p]));
        wl = __reduce_max_sync(full, wl);
        if (lane == 0)
            strip_order_add(sched, strip, wl);
    }
    const size_t P = size_t(o.width) * o.height;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
#pragma unroll
        for (int q = 0; q < (PX > 1 ? 2 : 1); ++q) {
            const int y = py + p * G::kBandRows + q;
            if (!(px < o.width && y < o.height))
                continue;
            const float t = fabsf(q ? T[p].y : T[p].x);
            const size_t pid = size_t(y) * o.width + px;
            o.color[pid] = (q ? r[p].y : r[p].x) + t * o.bg.x;
            o.color[P + pid] = (q ? g[p].y : g[p].x) + t * o.bg.y;
            o.color[2 * P + pid] = (q ? b[p].y : b[p].x) + t * o.bg.z;
            o.alpha[pid] = 1.f - t;
            if (o.pix_T) {
                o.pix_T[pid] = t;
                o.pix_last[pid] = q ? lb[p] : la[p];
            }
        }
    }
    return true;
}

// ---------------------------------------------------------------- adjoint --
// Gaussians whose adjoints are in flight together at one pixel per thread.
constexpr int kAdjointAhead = 2;

// Sums of one Gaussian over a lane's pixels, per element of the pairs.
template <bool kDensify> struct PairSums {
    float2 s, sy, syy; // s = o G dL/dalpha; s dy; s dy^2
    float2 refine;     // |(dL/dmx W, dL/dmy H)| / max(alpha_out, 1e-5)
    float2 cr, cg, cb; // w dL/dcolour
    float2 dn, dd;     // densify: map * w, w
};

struct PairState {
    float2 T, sdot, gx, gy, gz, rscale, dmap;
    unsigned la, lb;
};

// The adjoint of one Gaussian at a vertical pixel pair, added to `acc` (or
// stored, with kFirst). Blend decisions are the forward's (1/255 is tested on
// the unclipped opacity: with a clip below it the forward took no entry); a
// pixel that does not blend the Gaussian takes o G = alpha = 0, hence 1 / (1 - alpha) = 1,
// leaving its state unchanged and adding zero. Opacities and colours enter
// negated (nco = -o, nc = -c), so every difference is one multiply-add; the
// colour and densify sums come out negated (slot_scale). ra, rb, rc, rd: the
// mean gradient's norm is |s| |(ra + rb dy, rc + rd dy)|. kGuard: nothing of
// the Gaussian or of the pixel's gradients reaches an element that does not
// blend it (see kTame).
template <bool kRefine, bool kDensify, bool kFirst, bool kGuard = false>
__device__ __forceinline__ void pair_adjoint(PairState& p, unsigned pos, float4 co, float nco,
                                             float3 nc, float dx, float xx, float nxy, float2 dy,
                                             float clip, float ra, float rb, float rc, float rd,
                                             PairSums<kDensify>& acc) {
    const float2 power = pair_power(co, dx, xx, nxy, dy);
    const float2 og0 = __fmul2_rn(f2s(nco), f2(expf(power.x), expf(power.y)));
    const bool ha = pos < p.la && !(power.x > 0.f) && !(og0.x > -kAlphaFloor);
    const bool hb = pos < p.lb && !(power.y > 0.f) && !(og0.y > -kAlphaFloor);
    const float2 nog = f2(ha ? og0.x : 0.f, hb ? og0.y : 0.f);
    const float2 nal = f2(fmaxf(-clip, nog.x), fmaxf(-clip, nog.y));
    const float2 oma = __fadd2_rn(f2s(1.f), nal);
    const float2 inv = f2(1.f / oma.x, 1.f / oma.y);
    auto hit = [&](float2 v) { return kGuard ? f2(ha ? v.x : 0.f, hb ? v.y : 0.f) : v; };
    const float2 ncdot = hit(
        __ffma2_rn(f2s(nc.z), p.gz, __ffma2_rn(f2s(nc.y), p.gy, __fmul2_rn(f2s(nc.x), p.gx))));
    // -dL/dalpha = (S - T_behind c.g) / (1 - alpha), S the colour behind
    // (background included) along the gradient
    const float2 nda = __fmul2_rn(inv, __ffma2_rn(p.T, ncdot, p.sdot));
    p.T = __fmul2_rn(p.T, inv);
    const float2 nw = __fmul2_rn(nal, p.T);
    p.sdot = __ffma2_rn(nw, ncdot, p.sdot);
    const float2 s = hit(__fmul2_rn(nog, nda));
    const float2 sy = __fmul2_rn(s, dy);
    acc.s = kFirst ? s : __fadd2_rn(acc.s, s);
    acc.sy = kFirst ? sy : __fadd2_rn(acc.sy, sy);
    acc.syy = kFirst ? __fmul2_rn(sy, dy) : __ffma2_rn(sy, dy, acc.syy);
    if constexpr (kRefine) {
        const float2 u = __fmul2_rn(s, __ffma2_rn(f2s(rb), dy, f2s(ra)));
        const float2 v = __fmul2_rn(s, __ffma2_rn(f2s(rd), dy, f2s(rc)));
        const float2 q = __ffma2_rn(v, v, __fmul2_rn(u, u));
        const float2 nrm = f2(sqrtf(q.x), sqrtf(q.y));
        acc.refine = kFirst ? __fmul2_rn(nrm, p.rscale) : __ffma2_rn(nrm, p.rscale, acc.refine);
    }
    acc.cr = kFirst ? __fmul2_rn(nw, p.gx) : __ffma2_rn(nw, hit(p.gx), acc.cr);
    acc.cg = kFirst ? __fmul2_rn(nw, p.gy) : __ffma2_rn(nw, hit(p.gy), acc.cg);
    acc.cb = kFirst ? __fmul2_rn(nw, p.gz) : __ffma2_rn(nw, hit(p.gz), acc.cb);
    if constexpr (kDensify) {
        acc.dn = kFirst ? __fmul2_rn(p.dmap, nw) : __ffma2_rn(hit(p.dmap), nw, acc.dn);
        acc.dd = kFirst ? nw : __fadd2_rn(acc.dd, nw);
    }
}

// A lane's sums as the twelve gradient slots, up to slot_scale's factors.
template <bool kDensify>
__device__ __forceinline__ void lane_partials(const PairSums<kDensify>& a, bool refine, float4 co,
                                              float dx, float (&v)[12]) {
    const float s = a.s.x + a.s.y, sy = a.sy.x + a.sy.y, syy = a.syy.x + a.syy.y;
    const float sx = dx * s;
    v[0] = dx * sx;
    v[1] = dx * sy;
    v[2] = syy;
    v[3] = s;
    v[4] = co.x * sx + co.y * sy;
    v[5] = co.z * sy + co.y * sx;
    v[6] = refine ? a.refine.x + a.refine.y : 0.f;
    v[7] = kDensify ? a.dn.x + a.dn.y : 0.f;
    v[8] = a.cr.x + a.cr.y;
    v[9] = a.cg.x + a.cg.y;
    v[10] = a.cb.x + a.cb.y;
    v[11] = kDensify ? a.dd.x + a.dd.y : 0.f;
}

// The factor of gradient slot `slot` left out of lane_partials: -1/2 on the
// conic, -1 on the mean, the colour and the densify terms (1 / o on the
// opacity, slot 3, is the caller's).
__device__ __forceinline__ float slot_scale(int slot) {
    return slot < 3 ? -0.5f : slot == 6 ? 1.f : -1.f;
}

// Sums of twelve per-lane values over the warp: a reduce-scatter by halves of
// the values (13 shuffles); lane l ends with the sum of slot strip_slot12().
__device__ __forceinline__ float strip_reduce12(const float (&v)[12]) {
    const unsigned full = 0xffffffffu;
    const unsigned lane = lane_id();
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
    float u[6], w[4], x[2];
#pragma unroll
    for (int k = 0; k < 6; ++k)
        u[k] = (b4 ? v[k + 6] : v[k]) + __shfl_xor_sync(full, b4 ? v[k] : v[k + 6], 16);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        w[k] = (b3 ? u[k + 3] : u[k]) + __shfl_xor_sync(full, b3 ? u[k] : u[k + 3], 8);
    w[3] = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k)
        x[k] = (b2 ? w[k + 2] : w[k]) + __shfl_xor_sync(full, b2 ? w[k] : w[k + 2], 4);
    float y = (b1 ? x[1] : x[0]) + __shfl_xor_sync(full, b1 ? x[0] : x[1], 2);
    return y + __shfl_xor_sync(full, y, 1);
}

__device__ __forceinline__ int strip_slot12() {
    const unsigned lane = lane_id();
    const int idx = (lane & 4) ? ((lane & 2) ? -1 : 2) : ((lane & 2) ? 1 : 0);
    return (idx < 0 || (lane & 1)) ? -1 : ((lane & 16) ? 6 : 0) + ((lane & 8) ? 3 : 0) + idx;
}

// strip_reduce12 for the ten values that are not densify terms (slots 0-6 and
// 8-10): 12 shuffles.
__device__ __forceinline__ float strip_reduce10(const float (&v)[12]) {
    const unsigned full = 0xffffffffu;
    const unsigned lane = lane_id();
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
    const float p[10] = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[8], v[9], v[10]};
    float u[6], w[4], x[2];
#pragma unroll
    for (int k = 0; k < 5; ++k)
        u[k] = (b4 ? p[k + 5] : p[k]) + __shfl_xor_sync(full, b4 ? p[k] : p[k + 5], 16);
    u[5] = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        w[k] = (b3 ? u[k + 3] : u[k]) + __shfl_xor_sync(full, b3 ? u[k] : u[k + 3], 8);
    w[3] = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k)
        x[k] = (b2 ? w[k + 2] : w[k]) + __shfl_xor_sync(full, b2 ? w[k] : w[k + 2], 4);
    float y = (b1 ? x[1] : x[0]) + __shfl_xor_sync(full, b1 ? x[0] : x[1], 2);
    return y + __shfl_xor_sync(full, y, 1);
}

__device__ __forceinline__ int strip_slot10() {
    const unsigned lane = lane_id();
    // place in the lane's group of five: the group of three (b3) it ended in,
    // and its place there (b2, b1; the fourth place is padding)
    const int idx = (lane & 4) ? ((lane & 2) ? -1 : 2) : ((lane & 2) ? 1 : 0);
    const int e5 = idx < 0 ? -1 : ((lane & 8) ? 3 : 0) + idx;
    const int k = ((lane & 16) ? 5 : 0) + e5;
    return (e5 < 0 || e5 >= 5 || (lane & 1)) ? -1 : (k < 7 ? k : k + 1);
}

// Adjoint of the strip with origin (x0, y0): per-Gaussian gradients are added
// to rows of kGradSlots float4 at `grad`. kCount: counts into *pairs the
// (Gaussian, pixel) pairs evaluated (the pixel's recorded last entry lies at or
// behind the Gaussian) and does nothing else. kSeg: only segment `level` of
// the list, from the forward's checkpoints. False as the forward.
template <int TW, int PX, bool kRefine, bool kDensify, bool kCount = false, bool kSeg = false>
__device__ __forceinline__ bool composite_backward_strip(
    StripFeed& feed, int x0, int y0, uint2 range, const unsigned* __restrict__ order,
    const ViewGrads& o, float4* __restrict__ grad,
    unsigned long long* __restrict__ pairs = nullptr, const Checkpoints* cp = nullptr,
    int level = 0) {
    using G = StripGeom<TW, PX>;
    constexpr int NP = G::kBands;
    constexpr unsigned full = 0xffffffffu;
    const int lane = int(lane_id());
    const int px = x0 + lane % TW;
    const int py = y0 + (PX == 1 ? 1 : 2) * (lane / TW);
    const float fx = float(px);
    const float clip = o.clip;
    const size_t P = size_t(o.width) * o.height;
    const float Wf = float(o.width), Hf = float(o.height);

    PairState st[NP];
    float2 nfy[NP];
    unsigned wl = 0;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int y = py + p * G::kBandRows;
        PixBack a, c;
        const bool in_a = px < o.width && y < o.height;
        pixel_backward_init(a, in_a, in_a ? size_t(y) * o.width + px : 0, P, o.bg, o.pix_T,
                            o.pix_last, o.dL_color, o.dL_alpha, o.densify_map);
        const bool in_b = PX > 1 && px < o.width && y + 1 < o.height;
        pixel_backward_init(c, in_b, in_b ? size_t(y + 1) * o.width + px : 0, P, o.bg, o.pix_T,
                            o.pix_last, o.dL_color, o.dL_alpha, o.densify_map);
        st[p].T = f2(a.T, c.T);
        st[p].sdot = f2(a.fin_term, c.fin_term);
        st[p].gx = f2(a.gx, c.gx);
        st[p].gy = f2(a.gy, c.gy);
        st[p].gz = f2(a.gz, c.gz);
        st[p].rscale = f2(a.refine_scale, c.refine_scale);
        st[p].dmap = f2(a.dmap, c.dmap);
        st[p].la = a.last;
        st[p].lb = c.last;
        nfy[p] = f2(-float(y), -float(y + 1));
        wl = max(wl, max(a.last, c.last));
    }
    int total = int(min(__reduce_max_sync(full, wl), range.y - range.x));
    const int start = kSeg ? level * kSegment : 0; // first list position walked
    if (total <= start)
        return true;
    if constexpr (kSeg) {
        if (level + 1 < cp->levels) {
            const unsigned end = unsigned(start + kSegment);
            total = min(total, int(end));
            // a pixel blended past the segment starts from its checkpoint; the
            // colour behind it is that of the later segments
            auto resume = [&](int y, unsigned last, float& T, float& sdot, float gx, float gy,
                              float gz) {
                if (last <= end)
                    return;
                const float4* c = cp->data + size_t(level) * P + size_t(y) * o.width + px;
                T = c->w;
                for (unsigned l = unsigned(level) + 1;
                     l < unsigned(cp->levels) && l * kSegment < last; ++l) {
                    c += P;
                    sdot += c->x * gx + c->y * gy + c->z * gz;
                }
            };
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const int y = py + p * G::kBandRows;
                resume(y, st[p].la, st[p].T.x, st[p].sdot.x, st[p].gx.x, st[p].gy.x, st[p].gz.x);
                if constexpr (PX > 1)
                    resume(y + 1, st[p].lb, st[p].T.y, st[p].sdot.y, st[p].gx.y, st[p].gy.y,
                           st[p].gz.y);
            }
        }
    }
    const int slot = kDensify ? strip_slot12() : strip_slot10();
    const float scale = slot_scale(slot);
    float* const row = reinterpret_cast<float*>(grad) + max(slot, 0);
    bool calm = true;
#pragma unroll
    for (int p = 0; p < NP; ++p)
        calm = calm && tame(st[p].gx.x, st[p].gy.x, st[p].gz.x) &&
               tame(st[p].gx.y, st[p].gy.y, st[p].gz.y) &&
               tame(st[p].sdot.x, st[p].sdot.y, 0.f) && tame(st[p].dmap.x, st[p].dmap.y, 0.f);
    calm = __all_sync(full, calm);
    unsigned long long evaluated = 0;
    int base = (total - 1) / kStripBatch * kStripBatch;
    unsigned id_next = feed.issue(0, order, range.x + unsigned(base), total - base);
    int buf = 0;
    for (; base >= start; base -= kStripBatch) {
        const int cnt = min(kStripBatch, total - base);
        const unsigned id = id_next;
        if (base > start)
            id_next = feed.issue(buf ^ 1, order, range.x + unsigned(base - kStripBatch),
                                 kStripBatch);
        if (!feed.wait(buf)) {
            if (base > start)
                feed.wait(buf ^ 1);
            return false;
        }
        const SplatRec* rec = feed.s.rec[buf];
        unsigned mask[NP], all;
        unsigned m = strip_masks<TW, PX>(rec, cnt, x0, y0, mask, all);
        // Sums a Gaussian's partials over the warp and adds them to its row.
        auto reduce_add = [&](int j, const float (&v)[12], float opacity) {
            const unsigned gid = __shfl_sync(full, id, j);
            const float sum = kDensify ? strip_reduce12(v) : strip_reduce10(v);
            if (slot >= 0 && sum != 0.f)
                atomicAdd(row + size_t(gid) * (4 * kGradSlots),
                          sum * (slot == 3 ? 1.f / opacity : scale));
        };
        if constexpr (kCount) {
            for (; m; m &= m - 1) {
                const int j = __ffs(int(m)) - 1;
                const unsigned pos = unsigned(base + j);
#pragma unroll
                for (int p = 0; p < NP; ++p)
                    if ((mask[p] >> j) & 1u)
                        evaluated += (pos < st[p].la ? 1u : 0u) + (pos < st[p].lb ? 1u : 0u);
            }
        } else if constexpr (PX == 1) {
            // One pixel per thread: kAhead Gaussians per step, back to front.
            // Their opacities and reductions are independent; only T and the
            // colour behind run in order.
            constexpr int U = kAdjointAhead;
            PairState& t = st[0];
            while (m) {
                int j[U];
                bool ok[U]; // then: the pixel blends it
                float dx[U], dy[U], og[U], v[U][12];
                float4 co[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    ok[u] = m != 0;
                    j[u] = ok[u] ? 31 - __clz(int(m)) : j[u ? u - 1 : 0];
                    m &= ~(1u << j[u]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float2 xy = rec[j[u]].xy;
                    co[u] = rec[j[u]].co;
                    dx[u] = xy.x - fx;
                    dy[u] = xy.y + nfy[0].x;
                    const float power = gaussian_power(co[u], dx[u], dy[u]);
                    og[u] = co[u].w * expf(power);
                    ok[u] = ok[u] && unsigned(base + j[u]) < t.la && !(power > 0.f) &&
                            !(fminf(clip, og[u]) < kAlphaFloor);
                    og[u] = ok[u] ? og[u] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float4 c = rec[j[u]].rgb;
                    const float al = fminf(clip, og[u]);
                    const float inv = 1.f / (1.f - al);
                    // guarded at every pixel (see kTame)
                    auto hit = [&](float x) { return ok[u] ? x : 0.f; };
                    const float cdot = hit(c.x * t.gx.x + c.y * t.gy.x + c.z * t.gz.x);
                    const float da = inv * (t.T.x * cdot - hit(t.sdot.x));
                    t.T.x *= inv;
                    const float w = al * t.T.x;
                    t.sdot.x += w * cdot;
                    const float s = og[u] * da, sx = s * dx[u], sy = s * dy[u];
                    v[u][0] = dx[u] * sx;
                    v[u][1] = dx[u] * sy;
                    v[u][2] = dy[u] * sy;
                    v[u][3] = s;
                    v[u][4] = co[u].x * sx + co[u].y * sy;
                    v[u][5] = co[u].z * sy + co[u].y * sx;
                    const float rx = v[u][4] * Wf, ry = v[u][5] * Hf;
                    v[u][6] = kRefine ? sqrtf(rx * rx + ry * ry) * t.rscale.x : 0.f;
                    v[u][7] = kDensify ? -w * hit(t.dmap.x) : 0.f;
                    v[u][8] = -w * hit(t.gx.x);
                    v[u][9] = -w * hit(t.gy.x);
                    v[u][10] = -w * hit(t.gz.x);
                    v[u][11] = kDensify ? -w : 0.f;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    reduce_add(j[u], v[u], co[u].w);
            }
        } else {
            auto visits = [&]<bool kGuard>() {
                while (m) {
                    const int j = 31 - __clz(int(m));
                    m ^= 1u << j;
                    const unsigned pos = unsigned(base + j);
                    const float2 xy = rec[j].xy;
                    const float4 co = rec[j].co;
                    const float4 c = rec[j].rgb;
                    const float3 nc = make_float3(-c.x, -c.y, -c.z);
                    const float dx = xy.x - fx;
                    const float xx = __fmul_rn(co.x, dx);
                    const float nxy = -__fmul_rn(co.y, dx);
                    const float ra = xx * Wf, rb = co.y * Wf, rc = -nxy * Hf, rd = co.z * Hf;
                    PairSums<kDensify> acc;
                    if (!kGuard && ((all >> j) & 1u)) {
                        pair_adjoint<kRefine, kDensify, true>(
                            st[0], pos, co, -co.w, nc, dx, xx, nxy, __fadd2_rn(f2s(xy.y), nfy[0]),
                            clip, ra, rb, rc, rd, acc);
#pragma unroll
                        for (int p = 1; p < NP; ++p)
                            pair_adjoint<kRefine, kDensify, false>(
                                st[p], pos, co, -co.w, nc, dx, xx, nxy,
                                __fadd2_rn(f2s(xy.y), nfy[p]), clip, ra, rb, rc, rd, acc);
                    } else {
                        acc.s = acc.sy = acc.syy = acc.refine = f2s(0.f);
                        acc.cr = acc.cg = acc.cb = acc.dn = acc.dd = f2s(0.f);
#pragma unroll
                        for (int p = 0; p < NP; ++p)
                            if ((mask[p] >> j) & 1u)
                                pair_adjoint<kRefine, kDensify, false, kGuard>(
                                    st[p], pos, co, -co.w, nc, dx, xx, nxy,
                                    __fadd2_rn(f2s(xy.y), nfy[p]), clip, ra, rb, rc, rd, acc);
                    }
                    float v[12];
                    lane_partials<kDensify>(acc, kRefine, co, dx, v);
                    reduce_add(j, v, co.w);
                }
            };
            if (tame_colours(rec, cnt) && calm)
                visits.template operator()<false>();
            else
                visits.template operator()<true>();
        }
        buf ^= 1;
    }
    if constexpr (kCount)
        warp_count_add(evaluated, pairs);
    return true;
}

} // namespace gsb
