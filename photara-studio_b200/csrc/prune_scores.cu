// Speedy-Splat pruning scores (photara/src/splat/rasterizer.cu:93-146,
// CudaRasterizer::pruning_scores :450-490): per Gaussian, the sum over the
// pixels it was blended into of the squared sensitivity of the pixel's
// colour sum to its opacity, d = o (T c - R / (1 - a)), with R the colour
// left behind it (the rendered colour, background included, minus what the
// Gaussians up to it added), c its colour sum; or, with gaussian_pop, the
// squared norm of the per-channel a (T c_k - R_k / (1 - a)).
//
// B200 organisation: the reference adds every (pixel, Gaussian) value to the
// Gaussian's score with a global atomic. Here one warp owns a strip of a 16x16
// tile (strip.cuh: TMA-staged records, visit masks per band), sums each
// Gaussian's values over a lane's pixels, then over the warp with shuffles, and
// issues one global atomic. The per-pixel walk follows the forward's draw order
// up to the pixel's recorded last entry (at or behind the last blended one) and repeats the reference's per-pixel
// arithmetic expression for expression. Bound: instruction issue. 500,000
// Gaussians at 1280x720 268 -> 179 us, against one pixel per thread and a warp
// reduction per 32 pixels.
#include <cuda_runtime.h>

#include "kernels.h"
#include "strip.cuh"

namespace gsb {

namespace {

// kGuard: for colours that are not finite, which reach the pixels that blend
// them only (179 us without, 185 with).
template <int PX, bool kPop, bool kGuard>
__global__ void __launch_bounds__(32, PX == 8 ? 20 : 28) pruning_scores_kernel(
    const __grid_constant__ CUtensorMap map, unsigned* __restrict__ err,
    const uint2* __restrict__ ranges, const unsigned* __restrict__ order,
    const unsigned* __restrict__ pix_last, const float* __restrict__ image, int width, int height,
    int grid_x, float alpha_clip, float* __restrict__ scores) {
    using G = StripGeom<kTileW, PX>;
    constexpr int NP = G::kBands;
    constexpr unsigned full = 0xffffffffu;
    constexpr int kStrips = kTileH / G::kRows;
    __shared__ StripStage s;
    StripFeed feed{s, &map, err};
    feed.init();
    const int tile = int(blockIdx.x) / kStrips, strip = int(blockIdx.x) % kStrips;
    const int lane = int(lane_id());
    const int x0 = (tile % grid_x) * kTileW;
    const int y0 = (tile / grid_x) * kTileH + strip * G::kRows;
    const int x = x0 + lane % kTileW;
    const int y = y0 + 2 * (lane / kTileW); // pixel 2 p + q: row y + p * kBandRows + q
    const uint2 range = ranges[tile];
    const unsigned len = range.y - range.x;
    const size_t pixels = size_t(width) * height;
    unsigned limit[PX], most = 0;
    float residual[PX], T[PX];
    float3 residual_rgb[kPop ? PX : 1];
#pragma unroll
    for (int k = 0; k < PX; ++k) {
        const int yk = y + (k / 2) * G::kBandRows + (k & 1);
        limit[k] = 0;
        residual[k] = 0.f;
        T[k] = 1.f;
        if constexpr (kPop)
            residual_rgb[k] = make_float3(0.f, 0.f, 0.f);
        if (x < width && yk < height) {
            const size_t p = size_t(yk) * width + x;
            limit[k] = min(len, pix_last[p]);
            residual[k] = image[p] + image[p + pixels] + image[p + 2 * pixels];
            if constexpr (kPop)
                residual_rgb[k] = make_float3(image[p], image[p + pixels], image[p + 2 * pixels]);
        }
        most = max(most, limit[k]);
    }
    // the walk ends at the strip's largest last entry
    const int total = int(__reduce_max_sync(full, most));
    if (total == 0)
        return;
    unsigned id_next = feed.issue(0, order, range.x, min(kStripBatch, total));
    int buf = 0;
    for (int base = 0; base < total; base += kStripBatch) {
        const int cnt = min(kStripBatch, total - base);
        const unsigned id = id_next;
        const int left = total - base - kStripBatch;
        if (left > 0)
            id_next = feed.issue(buf ^ 1, order, range.x + unsigned(base + kStripBatch),
                                 min(kStripBatch, left));
        if (!feed.wait(buf)) {
            if (left > 0)
                feed.wait(buf ^ 1);
            return;
        }
        const SplatRec* rec = feed.s.rec[buf];
        unsigned mask[NP], all;
        unsigned m = strip_masks<kTileW, PX>(rec, cnt, x0, y0, mask, all);
        while (m) {
            const int j = __ffs(int(m)) - 1;
            m &= m - 1;
            const float2 xy = rec[j].xy;
            const float4 co = rec[j].co;
            const float4 c = rec[j].rgb;
            const float colour = c.x + c.y + c.z;
            const float dx = xy.x - x;
            float value = 0.f;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                if (!((mask[p] >> j) & 1u))
                    continue;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int k = 2 * p + q;
                    const float dy = xy.y - (y + p * G::kBandRows + q);
                    const float power = -.5f * (co.x * dx * dx + co.z * dy * dy) - co.y * dx * dy;
                    const float alpha = fminf(alpha_clip, co.w * expf(power));
                    const bool blended = unsigned(base + j) < limit[k] && !(power > 0.f) &&
                                         !(alpha < kAlphaFloor);
                    // a dropped Gaussian takes alpha 0 and adds nothing
                    const float a = blended ? alpha : 0.f;
                    const float inv = 1.f / (1.f - a);
                    auto at = [&](float v) { return kGuard && !blended ? 0.f : v; };
                    residual[k] -= T[k] * a * at(colour);
                    if constexpr (kPop) {
                        float3& rgb = residual_rgb[k];
                        rgb.x -= T[k] * a * at(c.x);
                        rgb.y -= T[k] * a * at(c.y);
                        rgb.z -= T[k] * a * at(c.z);
                        const float ex = a * (T[k] * c.x - rgb.x * inv);
                        const float ey = a * (T[k] * c.y - rgb.y * inv);
                        const float ez = a * (T[k] * c.z - rgb.z * inv);
                        value += blended ? ex * ex + ey * ey + ez * ez : 0.f;
                    } else {
                        const float derivative = co.w * (T[k] * colour - residual[k] * inv);
                        value += blended ? derivative * derivative : 0.f;
                    }
                    T[k] *= 1.f - a;
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                value += __shfl_xor_sync(full, value, off);
            const unsigned gid = __shfl_sync(full, id, j);
            if (lane == 0 && value != 0.f)
                atomicAdd(scores + gid, value);
        }
        buf ^= 1;
    }
}

} // namespace

cudaError_t launch_pruning_scores(cudaStream_t s, int tiles, const uint2* ranges,
                                  const unsigned* order, const Camera& K,
                                  const unsigned* pix_last, const float* image, int gaussian_pop,
                                  float* scores, const RecStaging& rs, bool guard) {
    if (tiles <= 0)
        return cudaGetLastError();
    auto go = [&]<int PX>() {
        auto kernel = gaussian_pop ? (guard ? pruning_scores_kernel<PX, true, true>
                                            : pruning_scores_kernel<PX, true, false>)
                                   : (guard ? pruning_scores_kernel<PX, false, true>
                                            : pruning_scores_kernel<PX, false, false>);
        kernel<<<tiles * (8 / PX), 32, 0, s>>>(rs.map, rs.err, ranges, order, pix_last, image,
                                               K.width, K.height, K.grid_x, K.alpha_clip, scores);
    };
    // more strips where there are too few tiles to fill the GPU; us at two / four
    // / eight pixels per thread: 256 tiles 123 / 173 / 271, 690 tiles 75 / 93 /
    // 133, 1,200 tiles 131 / 140 / 183, 1,900 tiles 204 / 187 / 215, 3,600 tiles
    // 210 / 181 / 197, 5,700 tiles 286 / 239 / 242, 8,160 tiles 348 / 279 / 272
    if (tiles <= 1000)
        go.template operator()<2>();
    else if (tiles <= 4800)
        go.template operator()<4>();
    else
        go.template operator()<8>();
    return cudaGetLastError();
}

} // namespace gsb
