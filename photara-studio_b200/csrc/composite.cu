// Single-view compositing kernels: one warp per strip of a reference 16x16
// tile running the forward / adjoint of strip.cuh (numerics and organisation
// described there; reference: third_party/splat_drender/src/render_forward.cu
// :341-416, :508-525 and render_backward.cu:156-519).
#include <algorithm>

#include "kernels.h"
#include "strip.cuh"

namespace gsb {

// Resident warps per SM that the strip kernels are compiled for: the register
// budget of each pixels-per-thread count without spills (the guarded and the
// counting forward at eight spill 8 bytes).
template <int PX> constexpr int kForwardCtas = PX == 8 ? 20 : PX == 4 ? 28 : 32;
template <int PX> constexpr int kBackwardCtas = PX == 8 ? 16 : PX == 4 ? 20 : 24;

// One warp per strip of a reference 16x16 tile (256 / (32 PX) strips per
// tile). kCount: the same forward that also counts its evaluated pairs. kSeg:
// it stores the adjoint's checkpoints. kGuard: with the guarded blend. wild
// (may be NULL): the device word that says which of the two kernels runs.
template <int PX, bool kCount = false, bool kSeg = false, bool kGuard = false>
__global__ void __launch_bounds__(32, kForwardCtas<PX>) composite_forward_kernel(
    const __grid_constant__ CUtensorMap map, unsigned* __restrict__ err,
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order, const Camera K,
    float3 bg, float* __restrict__ out_color, float* __restrict__ out_alpha,
    float* __restrict__ pix_T, unsigned* __restrict__ pix_last, float* __restrict__ visibility,
    StripOrder sched, Checkpoints cp, const unsigned* __restrict__ wild,
    unsigned long long* __restrict__ pairs = nullptr) {
    if (wild && (*wild != 0) != kGuard)
        return;
    constexpr int kStrips = kTileH / StripGeom<kTileW, PX>::kRows;
    __shared__ StripStage s;
    StripFeed feed{s, &map, err};
    feed.init();
    const int tile = int(blockIdx.x) / kStrips, strip = int(blockIdx.x) % kStrips;
    const ViewTarget o{K.width, K.height, K.alpha_clip, bg, out_color, out_alpha, pix_T, pix_last};
    composite_forward_strip<kTileW, PX, kCount, kSeg, kGuard>(
        feed, (tile % K.grid_x) * kTileW,
        (tile / K.grid_x) * kTileH + strip * StripGeom<kTileW, PX>::kRows, ranges[tile], order, o,
        visibility, sched, blockIdx.x, pairs, &cp, tile);
}

template <int PX, bool kRefine, bool kDensify, bool kCount = false>
__global__ void __launch_bounds__(32, kBackwardCtas<PX>) composite_backward_kernel(
    const __grid_constant__ CUtensorMap map, unsigned* __restrict__ err,
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order, float4* __restrict__ grad,
    const Camera K, float3 bg, const float* __restrict__ pix_T,
    const unsigned* __restrict__ pix_last, const float* __restrict__ dL_color,
    const float* __restrict__ dL_alpha, const float* __restrict__ densify_map, StripOrder sched,
    unsigned long long* __restrict__ pairs = nullptr) {
    constexpr int kStrips = kTileH / StripGeom<kTileW, PX>::kRows;
    __shared__ StripStage s;
    StripFeed feed{s, &map, err};
    feed.init();
    // heaviest strips first where the forward listed them
    const unsigned at = sched.count ? strip_order_get(sched, blockIdx.x) : blockIdx.x;
    if (at == 0xffffffffu)
        return;
    const int tile = int(at) / kStrips, strip = int(at) % kStrips;
    const ViewGrads o{K.width, K.height, K.alpha_clip, bg, pix_T, pix_last, dL_color, dL_alpha,
                      densify_map};
    composite_backward_strip<kTileW, PX, kRefine, kDensify, kCount>(
        feed, (tile % K.grid_x) * kTileW,
        (tile / K.grid_x) * kTileH + strip * StripGeom<kTileW, PX>::kRows, ranges[tile], order, o,
        grad, pairs);
}

// The adjoint from the forward's checkpoints: one-warp CTAs take the (segment,
// strip) items of the frame in turn, segments in front first. Four pixels per
// thread whatever the forward took, since segments already give enough warps
// (256 tiles: 52 us, at eight 78 us; the whole-list adjoint 114 us at its best).
constexpr int kSegmentPx = 4;

template <bool kRefine, bool kDensify>
__global__ void __launch_bounds__(32, kBackwardCtas<kSegmentPx>) composite_backward_segment_kernel(
    const __grid_constant__ CUtensorMap map, unsigned* __restrict__ err, unsigned tiles,
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order, float4* __restrict__ grad,
    const Camera K, float3 bg, const float* __restrict__ pix_T,
    const unsigned* __restrict__ pix_last, const float* __restrict__ dL_color,
    const float* __restrict__ dL_alpha, const float* __restrict__ densify_map, Checkpoints cp) {
    constexpr int PX = kSegmentPx;
    constexpr unsigned kStrips = kTileH / StripGeom<kTileW, PX>::kRows;
    __shared__ StripStage s;
    StripFeed feed{s, &map, err};
    feed.init();
    const unsigned strips = tiles * kStrips;
    const ViewGrads o{K.width, K.height, K.alpha_clip, bg, pix_T, pix_last, dL_color, dL_alpha,
                      densify_map};
    for (unsigned item = blockIdx.x; item < strips * unsigned(cp.levels); item += gridDim.x) {
        const unsigned level = item / strips, at = item % strips;
        const int tile = int(at / kStrips), strip = int(at % kStrips);
        if (cp.tile_last[tile] <= level * kSegment)
            continue;
        if (!composite_backward_strip<kTileW, PX, kRefine, kDensify, false, true>(
                feed, (tile % K.grid_x) * kTileW,
                (tile / K.grid_x) * kTileH + strip * StripGeom<kTileW, PX>::kRows, ranges[tile],
                order, o, grad, nullptr, &cp, int(level)))
            break;
        __syncwarp();
    }
}

size_t strip_order_words(int tiles, int pixels_per_thread) {
    return kWorkClasses * (1 + size_t(tiles) * size_t(8 / pixels_per_thread));
}

static StripOrder strip_order(unsigned* words, int tiles, int pixels_per_thread) {
    if (!words)
        return {};
    return {words, words + kWorkClasses, unsigned(tiles) * unsigned(8 / pixels_per_thread)};
}

// Test hook for the staging wait: one CTA announces 256 bytes on its
// mbarrier that no copy delivers, waits at most `limit` suspended waits
// (as StripFeed::wait does), and reports the timeout as it does.
__global__ void stage_probe_kernel(unsigned limit, unsigned* __restrict__ err) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0)
        mbar_init(&bar, 1);
    __syncthreads();
    if (threadIdx.x == 0)
        mbar_arrive_expect_tx(&bar, 256u);
    const bool ok = mbar_wait_bounded(&bar, 0u, limit);
    if (__syncthreads_or(!ok) && threadIdx.x == 0)
        atomicOr(err, kDevStageTimeout);
}

void launch_stage_probe(cudaStream_t s, unsigned limit, unsigned* err) {
    stage_probe_kernel<<<1, 64, 0, s>>>(limit, err);
}

// Evaluated (Gaussian, pixel) pairs of the colour compositing forward and its
// adjoint for the last forward's draw list: pairs[0] forward, pairs[1]
// adjoint (zeroed by the caller). The forward pass re-renders into color /
// alpha (identical images); the adjoint count needs only the per-pixel last
// contributors.
void launch_composite_count_pairs(cudaStream_t s, int tiles, const uint2* ranges,
                                  const unsigned* order, const GaussianState& st,
                                  const Camera& K, float3 bg, float* color, float* alpha,
                                  const float* pix_T, const unsigned* pix_last,
                                  int pixels_per_thread, unsigned long long* pairs,
                                  const RecStaging& rs) {
    // the count run writes no per-pixel state (NULL) and no visibility
    auto count = [&]<int PX>() {
        const int blocks = tiles * (8 / PX);
        composite_forward_kernel<PX, true><<<blocks, 32, 0, s>>>(
            rs.map, rs.err, ranges, order, K, bg, color, alpha, nullptr, nullptr, nullptr, {}, {},
            nullptr, pairs);
        composite_backward_kernel<PX, false, false, true><<<blocks, 32, 0, s>>>(
            rs.map, rs.err, ranges, order, st.grad, K, bg, pix_T, pix_last, color, nullptr,
            nullptr, {}, pairs + 1);
    };
    if (pixels_per_thread == 1)
        count.template operator()<1>();
    else if (pixels_per_thread == 2)
        count.template operator()<2>();
    else if (pixels_per_thread == 4)
        count.template operator()<4>();
    else
        count.template operator()<8>();
}

// ------------------------------------------------- geometry channels ----
// Forward with the median-depth and normal channels (render_forward.cu
// :274-525, blend_tile<GEOMETRY = true>): one thread per pixel of a 16x16
// tile. Pass 1 is the colour forward (the same per-pixel arithmetic as the
// colour kernels, so colour, alpha and final transmittance are bit-identical to
// them; the last contributor is the last one blended) plus the alpha-weighted footprint normal and the
// depth seed (the ray-plane depth of the last Gaussian blended while the
// transmittance was above 0.5). Pass 2 finds the depth at which the
// transmittance along the ray crosses 0.5: each Gaussian is a 1D Gaussian
// along the ray around its plane depth, and the pixel's transmittance at a
// probe depth is the product of the Gaussians' partial opacities there; 8
// probes over a +-0.4 window around the seed, refined 5 times (the first two
// refinements walk the tile's list up to the pixel's last contributor again,
// the later ones the Gaussians kept in front of and around the bracket), then linear
// interpolation inside the final bracket.
constexpr int kDepthSplit = 8;
constexpr int kDepthRefinements = 5;
constexpr float kDepthSeedWindow = 0.4f;
constexpr float kDepthMinTransmittance = 0.45f;
constexpr int kGeoThreads = kTileW * kTileH;
// Gaussians kept per pixel in front of and around the second refinement's
// bracket (0.1 wide), in thread-local memory. Forward with depth, us, five more
// walks of the list / keeping 48, 64, 96, 128: 500,000 at 1280x720 1,755 /
// 1,185, 1,177, 1,180, 1,177; 50,000 dense at 1280x960 2,285 / 2,364, 1,981,
// 1,952-1,966, 1,977; 200,000 at 700x500 1,263 / 746, 744, 733, 733 (with too
// few, most blocks hold a pixel that has to walk its list again). The 1,152-byte
// frames are above the default stack of 1,024 and make the driver enlarge its
// local memory by 40 MB when the kernel first runs.
constexpr int kNear = 96;

__global__ void __launch_bounds__(kGeoThreads) composite_geometry_kernel(
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order, GaussianState st,
    const Camera K, float3 bg, float* __restrict__ out_color, float* __restrict__ out_alpha,
    float* __restrict__ pix_T, unsigned* __restrict__ pix_last, float* __restrict__ pix_dtdt,
    float* __restrict__ visibility, float* __restrict__ out_depth,
    float* __restrict__ out_normal) {
    __shared__ unsigned s_id[kGeoThreads];
    __shared__ float2 s_xy[kGeoThreads];
    __shared__ float4 s_co[kGeoThreads];
    __shared__ float4 s_rgb[kGeoThreads];
    __shared__ float4 s_plane[kGeoThreads];
    __shared__ float4 s_nrm[kGeoThreads];
    __shared__ unsigned s_warp[kGeoThreads / 32];
    const int tile = blockIdx.x;
    const int tx = tile % K.grid_x, ty = tile / K.grid_x;
    const int tid = threadIdx.x;
    const int px = tx * kTileW + tid % kTileW, py = ty * kTileH + tid / kTileW;
    const bool inside = px < K.width && py < K.height;
    const float fx = float(px), fy = float(py);
    const uint2 range = ranges[tile];
    const int n = int(range.y - range.x);
    const float clip = K.alpha_clip;

    // ---- pass 1: colour, alpha, normal, depth seed ----
    float T = 1.f, cr = 0.f, cg = 0.f, cb = 0.f;
    float nx = 0.f, ny = 0.f, nz = 0.f, seed = 0.f;
    unsigned last = 0;
    bool done = !inside;
    for (int base = 0; base < n; base += kGeoThreads) {
        if (__syncthreads_and(done))
            break;
        if (base + tid < n) {
            const unsigned g = order[range.x + base + tid];
            s_id[tid] = g;
            s_xy[tid] = st.rec[g].xy;
            s_co[tid] = st.rec[g].co;
            s_rgb[tid] = st.rec[g].rgb;
            s_plane[tid] = st.plane[g];
            s_nrm[tid] = st.normal[g];
        }
        __syncthreads();
        const int cnt = min(kGeoThreads, n - base);
        for (int j = 0; !done && j < cnt; ++j) {
            const float dx = s_xy[j].x - fx, dy = s_xy[j].y - fy;
            const float4 co = s_co[j];
            const float power = gaussian_power(co, dx, dy);
            if (power > 0.f)
                continue;
            const float alpha = fminf(clip, co.w * expf(power));
            if (alpha < kAlphaFloor)
                continue;
            const float test_t = T * (1.f - alpha);
            if (test_t < kTransmittanceFloor) {
                done = true;
                continue;
            }
            const float w = alpha * T;
            const float4 c = s_rgb[j];
            cr += c.x * w;
            cg += c.y * w;
            cb += c.z * w;
            const float4 rp = s_plane[j];
            const float4 nm = s_nrm[j];
            const float t = rp.x * dx + rp.y * dy + rp.z;
            nx += nm.x * w;
            ny += nm.y * w;
            nz += nm.z * w;
            seed = T > 0.5f ? t : seed;
            if (visibility)
                visibility[s_id[j]] = 1.f;
            T = test_t;
            last = unsigned(base + j + 1);
        }
    }
    // the tile's furthest last contributor bounds pass 2
    unsigned wmax = last;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        wmax = max(wmax, __shfl_xor_sync(0xffffffffu, wmax, off));
    if ((tid & 31) == 0)
        s_warp[tid >> 5] = wmax;
    __syncthreads();
    unsigned block_max = 0;
#pragma unroll
    for (int w = 0; w < kGeoThreads / 32; ++w)
        block_max = max(block_max, s_warp[w]);

    // ---- pass 2: median-depth bisection ----
    // Walks the pixel's blended Gaussians (alpha, peak distance, 1/sigma).
    auto walk = [&](bool run, auto&& f) {
        bool ldone = !run;
        unsigned seen = 0;
        for (int base = 0; base < int(block_max); base += kGeoThreads) {
            if (__syncthreads_and(ldone))
                break;
            if (base + tid < int(block_max)) {
                const unsigned g = order[range.x + base + tid];
                s_xy[tid] = st.rec[g].xy;
                s_co[tid] = st.rec[g].co;
                s_plane[tid] = st.plane[g];
            }
            __syncthreads();
            const int cnt = min(kGeoThreads, int(block_max) - base);
            for (int j = 0; !ldone && j < cnt; ++j) {
                ++seen;
                ldone = seen >= last;
                const float dx = s_xy[j].x - fx, dy = s_xy[j].y - fy;
                const float4 co = s_co[j];
                const float power = gaussian_power(co, dx, dy);
                if (power > 0.f)
                    continue;
                const float alpha = fminf(clip, co.w * expf(power));
                if (alpha < kAlphaFloor)
                    continue;
                const float4 rp = s_plane[j];
                f(alpha, rp.x * dx + rp.y * dy + rp.z, rp.w);
            }
        }
    };
    constexpr int S = kDepthSplit;
    float depth_min = fmaxf(seed - kDepthSeedWindow, 0.f);
    float depth_max = fmaxf(seed + kDepthSeedWindow, 0.f);
    bool in_range = T <= kDepthMinTransmittance;
    float Tp[S + 1];
    float interval = 0.f;
    // One Gaussian's factors on the probes (first: the window's ends too).
    // Beyond 6 sigma of the peak a probe's Gaussian factor is exactly 0 in the
    // product (alpha g < 2^-25, so 1 - alpha g rounds to 1 and its inverse
    // square root is 1): the probe takes (1 - alpha) behind the peak and 1 in
    // front of it. A Gaussian whose peak is that far behind every probe
    // changes nothing; one that far in front scales all.
    auto probe = [&](bool first, float alpha, float t_peak, float rsigma) {
        const bool ball = rsigma > 0.f;
        const int k0 = first ? 0 : 1, k1 = first ? S : S - 1;
        const float d_lo = (depth_min + interval * float(k0) - t_peak) * rsigma;
        const float d_hi = (depth_min + interval * float(k1) - t_peak) * rsigma;
        if (ball && d_hi < -6.f)
            return;
        const float oma = 1.f - alpha;
        const bool step = !ball || d_lo > 6.f;
#pragma unroll
        for (int k = 0; k <= S; ++k) {
            if (!(first || (k > 0 && k < S)))
                continue;
            const float ts = depth_min + interval * float(k);
            const float delta = (ts - t_peak) * rsigma;
            if (step || delta * delta > 36.f) {
                Tp[k] *= ts > t_peak ? oma : 1.f;
                continue;
            }
            const float gk = expf(-0.5f * delta * delta);
            const float omg = 1.f - alpha * gk;
            const float rv = rsqrtf(omg);
            Tp[k] *= (ts > t_peak ? oma : omg) * rv;
        }
    };
    auto begin = [&](bool first) {
#pragma unroll
        for (int k = 0; k <= S; ++k)
            if (first || (k > 0 && k < S))
                Tp[k] = 1.f;
        interval = (depth_max - depth_min) * (1.f / float(S));
    };
    // Keeps the bracket of the probes around transmittance 0.5.
    auto narrow = [&](bool first) {
        if (first)
            in_range = Tp[0] >= 0.5f && Tp[S] <= 0.5f && in_range;
        int start = 0;
#pragma unroll
        for (int k = 1; k < S; ++k)
            start = Tp[k] >= 0.5f ? k : start;
        // Tp indices are compile-time after unrolling: pick the bracket ends
        // with selects.
        float lo_T = Tp[0], hi_T = Tp[1];
#pragma unroll
        for (int k = 1; k < S; ++k) {
            lo_T = start == k ? Tp[k] : lo_T;
            hi_T = start == k ? Tp[k + 1] : hi_T;
        }
        depth_max = depth_min + float(start + 1) * interval;
        depth_min = depth_min + float(start + 0) * interval;
        Tp[0] = lo_T;
        Tp[S] = hi_T;
    };
    begin(true);
    walk(in_range, [&](float alpha, float t, float rs) { probe(true, alpha, t, rs); });
    narrow(true);
    // The second refinement's walk also keeps the Gaussians that its bracket,
    // which holds all later probes, does not lie 8 sigma or more in front of:
    // those behind it change nothing any more. The later refinements and dT/dt
    // then need no walk (five walks of the list before, and a sixth for dT/dt),
    // and multiply the same factors in the same order.
    float near_alpha[kNear], near_peak[kNear], near_rs[kNear];
    int near_n = 0;
    begin(false);
    walk(in_range, [&](float alpha, float t, float rs) {
        probe(false, alpha, t, rs);
        if (rs > 0.f && (depth_max - t) * rs < -8.f)
            return;
        if (near_n < kNear) {
            near_alpha[near_n] = alpha;
            near_peak[near_n] = t;
            near_rs[near_n] = rs;
        }
        ++near_n;
    });
    narrow(false);
    // a pixel with more of them than are kept walks its list again
    const bool kept = near_n <= kNear;
    const bool any_over = __syncthreads_or(in_range && !kept);
#pragma unroll 1
    for (int r = 2; r < kDepthRefinements; ++r) {
        begin(false);
        if (in_range && kept)
            for (int k = 0; k < near_n; ++k)
                probe(false, near_alpha[k], near_peak[k], near_rs[k]);
        if (any_over)
            walk(in_range && !kept,
                 [&](float alpha, float t, float rs) { probe(false, alpha, t, rs); });
        narrow(false);
    }
    const float w_max = __saturatef((Tp[0] - 0.5f) / (Tp[0] - Tp[S]));
    const float w_min = 1.f - w_max;
    const float median = in_range ? w_max * depth_max + w_min * depth_min : 0.f;
    const float rln = pixel_ray_z(fx, fy, K);
    const float depth_out = median * rln;

    // ---- pass 3 (training forward only): dT/dt at the median depth ----
    // The derivative of the ray transmittance with respect to the median
    // distance, summed over the pixel's blended Gaussians:
    // -1/4 G_t / (1 - G_t) |delta| / sigma (render_backward.cu:47-151,
    // median_scale_walk, here evaluated where the median is found, at the
    // distance the backward recovers from the written depth). The backward
    // turns it into dL/dt with the depth gradient. Gaussians beyond 8 sigma
    // of the bracket (G_t below 1.3e-14) add nothing.
    float dTdt = 0.f;
    if (pix_dtdt) {
        const float mD = depth_out / fmaxf(rln, 1.0e-8f);
        const bool run = inside && mD != 0.f && last != 0;
        auto slope = [&](float alpha, float t, float rs) {
            const float t_delta = (mD - t) * rs;
            const float g_exp = expf(-0.5f * t_delta * t_delta);
            const float gt = alpha * g_exp;
            dTdt += -0.25f * gt / (1.f - gt) * fabsf(t_delta) * rs;
        };
        if (run && kept)
            for (int k = 0; k < near_n; ++k)
                slope(near_alpha[k], near_peak[k], near_rs[k]);
        if (any_over)
            walk(run && !kept, slope);
    }

    if (inside) {
        const size_t P = size_t(K.width) * K.height;
        const size_t pid = size_t(py) * K.width + px;
        out_color[pid] = cr + T * bg.x;
        out_color[P + pid] = cg + T * bg.y;
        out_color[2 * P + pid] = cb + T * bg.z;
        out_alpha[pid] = 1.f - T;
        if (pix_T) {
            pix_T[pid] = T;
            pix_last[pid] = last;
        }
        if (pix_dtdt)
            pix_dtdt[pid] = dTdt;
        out_depth[pid] = depth_out;
        const float len = 1.f - T;
        out_normal[pid] = last ? nx / len : 0.f;
        out_normal[P + pid] = last ? ny / len : 0.f;
        out_normal[2 * P + pid] = last ? nz / len : 0.f;
    }
}

void launch_composite_geometry(cudaStream_t s, int tiles, const uint2* ranges,
                               const unsigned* order, const GaussianState& st, const Camera& K,
                               float3 bg, float* color, float* alpha, float* pix_T,
                               unsigned* pix_last, float* pix_dtdt, float* visibility,
                               float* median_depth, float* normal) {
    composite_geometry_kernel<<<tiles, kGeoThreads, 0, s>>>(ranges, order, st, K, bg, color,
                                                            alpha, pix_T, pix_last, pix_dtdt,
                                                            visibility, median_depth, normal);
}

// ------------------------------------------- geometry-channel adjoint ----
// Backward of the colour, median-depth and normal channels together
// (render_backward.cu:156-519, blend_bucket_backward<GEOMETRY = true>): one
// warp per strip walks it back to front from its pixels' last contributors,
// recovering T by T_i = T_{i+1} / (1 - a_i) as the colour adjoint does. Per
// pixel it also carries the normal-output gradient divided by the rendered
// alpha (the normal output is the alpha-normalised sum), the running sum of the
// normals blended behind the current Gaussian projected on it, the median
// distance and dL/dt (the depth gradient over -dT/dt from the forward). Per
// (Gaussian, pixel) it adds, besides the colour terms: to dL/d opacity the
// normal term and the median term, to dL/d mean2d the ray plane's screen slope
// times dL/dt, and the gradients of the footprint normal (3) and of the ray
// plane (4). The refine weight takes the colour part of the mean2d gradient
// only, as the reference's. A pixel adds the moments of its gradient (strip.cuh)
// and of dL/dt; the partials are formed per lane, reduced across the warp (two
// reduce-scatters) and added by one atomic each. Bound: instruction issue.
// 500,000 Gaussians at 1280x720 1,030 -> 723 us, against a thread per pixel,
// both reductions per 32 pixels and accumulators in shared memory.
// Reduce 8 per-lane values across the warp; returns the sum of slot `slot`
// (slot = -1 for lanes that hold a duplicate).
__device__ __forceinline__ float reduce_scatter8(const float (&v)[8], int& slot) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    float u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float send = b4 ? v[k] : v[k + 4];
        const float keep = b4 ? v[k + 4] : v[k];
        u[k] = keep + __shfl_xor_sync(full, send, 16);
    }
    float w[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float send = b3 ? u[k] : u[k + 2];
        const float keep = b3 ? u[k + 2] : u[k];
        w[k] = keep + __shfl_xor_sync(full, send, 8);
    }
    const float send = b2 ? w[0] : w[1];
    const float keep = b2 ? w[1] : w[0];
    float x = keep + __shfl_xor_sync(full, send, 4);
    x += __shfl_xor_sync(full, x, 2);
    x += __shfl_xor_sync(full, x, 1);
    slot = (lane & 3) ? -1 : (b4 ? 4 : 0) + (b3 ? 2 : 0) + (b2 ? 1 : 0);
    return x;
}

// Ray planes and normals of a strip's two batches, beside the records.
struct GeoStage {
    float4 plane[2][kStripBatch];
    float4 normal[2][kStripBatch];
};

__device__ __forceinline__ void geo_copy16(float4* dst, const float4* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}

template <int PX, bool kRefine, bool kDensify>
__global__ void __launch_bounds__(32, PX == 4 ? 16 : 20) composite_backward_geometry_kernel(
    const __grid_constant__ CUtensorMap map, unsigned* __restrict__ err,
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order, GaussianState st,
    const Camera K, float3 bg, const float* __restrict__ pix_T,
    const unsigned* __restrict__ pix_last, const float* __restrict__ pix_dtdt,
    const float* __restrict__ dL_color, const float* __restrict__ dL_alpha,
    const float* __restrict__ densify_map, const float* __restrict__ dL_depth,
    const float* __restrict__ dL_normal, const float* __restrict__ fwd_depth,
    const float* __restrict__ fwd_normal) {
    using G = StripGeom<kTileW, PX>;
    constexpr int NP = G::kBands;
    constexpr unsigned full = 0xffffffffu;
    constexpr int kStrips = kTileH / G::kRows;
    __shared__ StripStage s;
    __shared__ GeoStage geo;
    StripFeed feed{s, &map, err};
    feed.init();
    const int tile = int(blockIdx.x) / kStrips, strip = int(blockIdx.x) % kStrips;
    const int lane = int(lane_id());
    const int x0 = (tile % K.grid_x) * kTileW;
    const int y0 = (tile / K.grid_x) * kTileH + strip * G::kRows;
    const int px = x0 + lane % kTileW;
    const int py = y0 + 2 * (lane / kTileW); // pixel 2 p + q: row py + p * kBandRows + q
    const float fx = float(px);
    const uint2 range = ranges[tile];
    const float clip = K.alpha_clip;
    const size_t P = size_t(K.width) * K.height;
    const bool with_depth = dL_depth != nullptr, with_normal = dL_normal != nullptr;
    const float Wf = float(K.width), Hf = float(K.height);

    // ---- per-pixel state ----
    float T[PX], sdot[PX], ndot[PX], gx[PX], gy[PX], gz[PX], gnx[PX], gny[PX], gnz[PX];
    float fin_r[PX], fin[PX], rscale[PX], dmap[kDensify ? PX : 1], mD[PX], dmt[PX];
    unsigned last[PX], wl = 0;
#pragma unroll
    for (int k = 0; k < PX; ++k) {
        const int y = py + (k / 2) * G::kBandRows + (k & 1);
        T[k] = 1.f;
        last[k] = 0;
        sdot[k] = ndot[k] = gx[k] = gy[k] = gz[k] = gnx[k] = gny[k] = gnz[k] = 0.f;
        fin_r[k] = fin[k] = mD[k] = dmt[k] = 0.f;
        if constexpr (kDensify)
            dmap[k] = 0.f;
        if (px < K.width && y < K.height) {
            const size_t pid = size_t(y) * K.width + px;
            T[k] = pix_T[pid];
            last[k] = pix_last[pid];
            gx[k] = dL_color[pid];
            gy[k] = dL_color[P + pid];
            gz[k] = dL_color[2 * P + pid];
            const float dfin_r =
                bg.x * gx[k] + bg.y * gy[k] + bg.z * gz[k] - (dL_alpha ? dL_alpha[pid] : 0.f);
            float dfin = dfin_r;
            if (with_normal) {
                // the normal output is the blended normal sum over alpha = 1 - T
                const float wf = 1.f - T[k];
                const float inv_w = wf > 0.f ? 1.f / wf : 0.f;
                gnx[k] = dL_normal[pid] * inv_w;
                gny[k] = dL_normal[P + pid] * inv_w;
                gnz[k] = dL_normal[2 * P + pid] * inv_w;
                dfin += gnx[k] * fwd_normal[pid] + gny[k] * fwd_normal[P + pid] +
                        gnz[k] * fwd_normal[2 * P + pid];
            }
            if (with_depth) {
                const float rln = pixel_ray_z(fx, float(y), K);
                mD[k] = fwd_depth[pid] / fmaxf(rln, 1.0e-8f);
                dmt[k] = dL_depth[pid] * rln / fmaxf(-pix_dtdt[pid], 1.0e-7f);
            }
            fin_r[k] = T[k] * dfin_r;
            fin[k] = T[k] * dfin;
            if constexpr (kDensify)
                dmap[k] = densify_map ? densify_map[pid] : 0.f;
        }
        rscale[k] = 1.f / fmaxf(1.f - T[k], 1.0e-5f);
        wl = max(wl, last[k]);
    }
    const int total = int(min(__reduce_max_sync(full, wl), range.y - range.x));
    if (total == 0)
        return;
    const int slot = kDensify ? strip_slot12() : strip_slot10();
    const float scale = slot_scale(slot);
    float* const row = reinterpret_cast<float*>(st.grad) + max(slot, 0);

    auto issue = [&](int b, unsigned first, int cnt) {
        const unsigned id = feed.issue(b, order, first, cnt);
        geo_copy16(&geo.plane[b][lane], st.plane + id);
        geo_copy16(&geo.normal[b][lane], st.normal + id);
        asm volatile("cp.async.commit_group;" ::: "memory");
        return id;
    };
    int base = (total - 1) / kStripBatch * kStripBatch;
    unsigned id_next = issue(0, range.x + unsigned(base), total - base);
    int buf = 0;
    for (; base >= 0; base -= kStripBatch) {
        const int cnt = min(kStripBatch, total - base);
        const unsigned id = id_next;
        if (base > 0) {
            id_next = issue(buf ^ 1, range.x + unsigned(base - kStripBatch), kStripBatch);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        if (!feed.wait(buf)) {
            if (base > 0)
                feed.wait(buf ^ 1);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            return;
        }
        const SplatRec* rec = feed.s.rec[buf];
        unsigned mask[NP], all;
        unsigned m = strip_masks<kTileW, PX>(rec, cnt, x0, y0, mask, all);
        while (m) {
            const int j = 31 - __clz(int(m));
            m ^= 1u << j;
            const unsigned pos = unsigned(base + j);
            const float2 xy = rec[j].xy;
            const float4 co = rec[j].co;
            const float4 c = rec[j].rgb;
            const float4 rp = geo.plane[buf][j];
            const float4 n = geo.normal[buf][j];
            const float dx = xy.x - fx;
            PairSums<kDensify> acc; // .x: the lane's sums (.y unused, zero)
            acc.s = acc.sy = acc.syy = acc.refine = f2s(0.f);
            acc.cr = acc.cg = acc.cb = acc.dn = acc.dd = f2s(0.f);
            float dts = 0.f, dty = 0.f; // sums of dL/dt, dL/dt dy
            float vg[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                vg[k] = 0.f;
#pragma unroll
            for (int k = 0; k < PX; ++k) {
                if (!((mask[k / 2] >> j) & 1u))
                    continue;
                const float dy = xy.y - float(py + (k / 2) * G::kBandRows + (k & 1));
                const float power = gaussian_power(co, dx, dy);
                const float og = co.w * expf(power);
                const float alpha = fminf(clip, og);
                if (pos >= last[k] || power > 0.f || alpha < kAlphaFloor)
                    continue;
                const float inv_1ma = 1.f / (1.f - alpha);
                T[k] *= inv_1ma; // transmittance in front of this Gaussian
                const float w = alpha * T[k];
                const float cdot = c.x * gx[k] + c.y * gy[k] + c.z * gz[k];
                const float dL_da_r = T[k] * cdot - (sdot[k] + fin_r[k]) * inv_1ma;
                float dL_da = T[k] * cdot - (sdot[k] + fin[k]) * inv_1ma;
                sdot[k] += w * cdot;
                if (with_normal) {
                    const float nd = n.x * gnx[k] + n.y * gny[k] + n.z * gnz[k];
                    dL_da += T[k] * nd - ndot[k] * inv_1ma;
                    ndot[k] += w * nd;
                    vg[4] += w * gnx[k];
                    vg[5] += w * gny[k];
                    vg[6] += w * gnz[k];
                }
                if (with_depth) {
                    const float t_peak = rp.x * dx + rp.y * dy + rp.z;
                    const float rsigma = rp.w;
                    const float t_delta = (mD[k] - t_peak) * rsigma;
                    const float g_exp = expf(-0.5f * t_delta * t_delta);
                    const float gt = alpha * g_exp;
                    float dgt = dmt[k] * 0.25f / (1.f - gt);
                    dgt = mD[k] > t_peak ? dgt : -dgt;
                    dgt = rsigma > 0.f ? dgt : 0.f;
                    dL_da += dgt * g_exp - dmt[k] * (t_delta > 0.f ? 0.5f * inv_1ma : 0.f);
                    const float ddelta = -dgt * gt * t_delta;
                    const float dt = -ddelta * rsigma;
                    vg[3] += ddelta * (mD[k] - t_peak);
                    dts += dt;
                    dty += dt * dy;
                }
                const float sg = og * dL_da, sgy = sg * dy;
                acc.s.x += sg;
                acc.sy.x += sgy;
                acc.syy.x += sgy * dy;
                if constexpr (kRefine) {
                    const float sr = og * dL_da_r;
                    const float rx = sr * (co.x * dx + co.y * dy) * Wf;
                    const float ry = sr * (co.z * dy + co.y * dx) * Hf;
                    acc.refine.x += sqrtf(rx * rx + ry * ry) * rscale[k];
                }
                // the colour and densify sums enter negated (slot_scale)
                acc.cr.x -= w * gx[k];
                acc.cg.x -= w * gy[k];
                acc.cb.x -= w * gz[k];
                if constexpr (kDensify) {
                    acc.dn.x -= dmap[k] * w;
                    acc.dd.x -= w;
                }
            }
            float v[12];
            lane_partials<kDensify>(acc, kRefine, co, dx, v);
            v[4] -= rp.x * dts; // scaled by -1
            v[5] -= rp.y * dts;
            vg[0] = dx * dts;
            vg[1] = dty;
            vg[2] = dts;
            const unsigned gid = __shfl_sync(full, id, j);
            const float sum = kDensify ? strip_reduce12(v) : strip_reduce10(v);
            if (slot >= 0 && sum != 0.f)
                atomicAdd(row + size_t(gid) * (4 * kGradSlots),
                          sum * (slot == 3 ? 1.f / co.w : scale));
            int gslot;
            const float gsum = reduce_scatter8(vg, gslot);
            if (gslot >= 0 && gslot < 7 && gsum != 0.f)
                atomicAdd(reinterpret_cast<float*>(st.geo_grad) + size_t(gid) * (4 * kGeoGradSlots) +
                              gslot,
                          gsum);
        }
        buf ^= 1;
    }
}

void launch_composite_backward_geometry(cudaStream_t s, int tiles, const uint2* ranges,
                                        const unsigned* order, const GaussianState& st,
                                        const Camera& K, float3 bg, const float* pix_T,
                                        const unsigned* pix_last, const float* pix_dtdt,
                                        const float* dL_color, const float* dL_alpha,
                                        const float* densify_map, int want_refine,
                                        const float* dL_depth, const float* dL_normal,
                                        const float* fwd_depth, const float* fwd_normal,
                                        const RecStaging& rs) {
    auto bwd = [&]<int PX>() {
        auto go = [&](auto kernel) {
            kernel<<<tiles * (8 / PX), 32, 0, s>>>(rs.map, rs.err, ranges, order, st, K, bg, pix_T,
                                                   pix_last, pix_dtdt, dL_color, dL_alpha,
                                                   densify_map, dL_depth, dL_normal, fwd_depth,
                                                   fwd_normal);
        };
        if (want_refine && densify_map)
            go(composite_backward_geometry_kernel<PX, true, true>);
        else if (want_refine)
            go(composite_backward_geometry_kernel<PX, true, false>);
        else if (densify_map)
            go(composite_backward_geometry_kernel<PX, false, true>);
        else
            go(composite_backward_geometry_kernel<PX, false, false>);
    };
    // more strips where there are too few tiles to fill the GPU; us at two /
    // four pixels per thread: 256 tiles 298 / 461, 690 tiles 222 / 297, 1,200
    // tiles 458 / 439, 1,900 tiles 648 / 667, 3,600 tiles 769 / 723, 8,160 tiles
    // 1,335 / 1,203
    if (tiles <= 1000)
        bwd.template operator()<2>();
    else
        bwd.template operator()<4>();
}

void launch_composite_forward(cudaStream_t s, int tiles, const uint2* ranges,
                              const unsigned* order, const Camera& K, float3 bg, float* color,
                              float* alpha, float* pix_T, unsigned* pix_last, float* visibility,
                              int pixels_per_thread, const RecStaging& rs, ColourGuard guard,
                              unsigned* work_lists, const SegmentStore* segments) {
    const bool seg = segments && segments->levels > 0;
    const StripOrder sched = strip_order(seg ? nullptr : work_lists, tiles, pixels_per_thread);
    const Checkpoints cp = seg ? Checkpoints{segments->data, segments->tile_last, segments->levels}
                               : Checkpoints{};
    auto fwd = [&]<int PX>() {
        auto go = [&](auto kernel) {
            kernel<<<tiles * (8 / PX), 32, 0, s>>>(rs.map, rs.err, ranges, order, K, bg, color,
                                                   alpha, pix_T, pix_last, visibility, sched, cp,
                                                   PX > 1 ? guard.word : nullptr, nullptr);
        };
        auto either = [&]<bool kSeg>() {
            if constexpr (PX > 1)
                if (guard.on || guard.word)
                    go(composite_forward_kernel<PX, false, kSeg, true>);
            if (PX == 1 || !guard.on || guard.word)
                go(composite_forward_kernel<PX, false, kSeg, false>);
        };
        if constexpr (PX <= 2)
            if (seg)
                return either.template operator()<true>();
        either.template operator()<false>();
    };
    if (pixels_per_thread == 1)
        fwd.template operator()<1>();
    else if (pixels_per_thread == 2)
        fwd.template operator()<2>();
    else if (pixels_per_thread == 4)
        fwd.template operator()<4>();
    else
        fwd.template operator()<8>();
}

void launch_composite_backward(cudaStream_t s, int tiles, const uint2* ranges,
                               const unsigned* order, const GaussianState& st, const Camera& K,
                               float3 bg, const float* pix_T, const unsigned* pix_last,
                               const float* dL_color, const float* dL_alpha,
                               const float* densify_map, int want_refine, int pixels_per_thread,
                               const RecStaging& rs, unsigned* work_lists,
                               const SegmentStore* segments) {
    if (segments && segments->levels > 0) {
        const Checkpoints cp{segments->data, segments->tile_last, segments->levels};
        constexpr int PX = kSegmentPx;
        const unsigned items = unsigned(tiles) * (8 / PX) * unsigned(cp.levels);
        const unsigned blocks = std::min(items, 148u * kBackwardCtas<PX>);
        auto go = [&](auto kernel) {
            kernel<<<blocks, 32, 0, s>>>(rs.map, rs.err, unsigned(tiles), ranges, order, st.grad,
                                         K, bg, pix_T, pix_last, dL_color, dL_alpha, densify_map,
                                         cp);
        };
        if (want_refine && densify_map)
            go(composite_backward_segment_kernel<true, true>);
        else if (want_refine)
            go(composite_backward_segment_kernel<true, false>);
        else if (densify_map)
            go(composite_backward_segment_kernel<false, true>);
        else
            go(composite_backward_segment_kernel<false, false>);
        return;
    }
    const StripOrder sched = strip_order(work_lists, tiles, pixels_per_thread);
    auto bwd = [&]<int PX>() {
        auto go = [&](auto kernel) {
            kernel<<<tiles * (8 / PX), 32, 0, s>>>(rs.map, rs.err, ranges, order, st.grad, K, bg,
                                                   pix_T, pix_last, dL_color, dL_alpha,
                                                   densify_map, sched, nullptr);
        };
        if (want_refine && densify_map)
            go(composite_backward_kernel<PX, true, true>);
        else if (want_refine)
            go(composite_backward_kernel<PX, true, false>);
        else if (densify_map)
            go(composite_backward_kernel<PX, false, true>);
        else
            go(composite_backward_kernel<PX, false, false>);
    };
    if (pixels_per_thread == 1)
        bwd.template operator()<1>();
    else if (pixels_per_thread == 2)
        bwd.template operator()<2>();
    else if (pixels_per_thread == 4)
        bwd.template operator()<4>();
    else
        bwd.template operator()<8>();
}

} // namespace gsb
