// Per-Gaussian backward (EWA projection adjoint + SH adjoint) fused with the
// Adam updates, plus the standalone Adam and L1-loss kernels of the step.
//
// Reference behaviour followed:
//   gaussian_backward        third_party/splat_drender/src/render_backward.cu:708-862
//   splat_backward (pinhole RGB chain, conic / cap / cov3D / J / mean2d)
//                            third_party/splat_drender/src/device/geometry.cuh:317-912
//   update_structure_adam_row, adam_scalar, shape regularizers
//                            third_party/splat_drender/src/render_backward.cu:525-706
//   quantized SH Adam codec  third_party/splat_drender/include/splat_drender/sh_adam_quant.cuh:23-234
//   standalone Adam / L1     photara/src/splat/cuda_ops.cu:846-891, :1336
//
// B200 organisation: 128 Gaussians per CTA. Phase 1, one thread per
// Gaussian: the CTA's SH rows (contiguous in HBM) and, with the fused SH Adam,
// their fp16 first moments, u8 codes and code bounds are staged through shared
// memory with coalesced asynchronous copies while the per-Gaussian inputs
// load; then each thread runs its Gaussian's projection and SH adjoints and
// the structure Adam from registers. The SH adjoint leaves the row's basis
// values and clamped colour gradient in shared memory (19 words instead of the
// 48 coefficient gradients: each gradient is one product of the two).
// Phase 2, the quantized SH Adam: degree-3 rows one thread per row on f32x2
// pairs (only the parameters staged; 284 bytes of shared memory per Gaussian
// and 96 registers give 5 CTAs, 20 warps, per SM); other strides and degrees
// one half-warp per row with everything staged (440 bytes: 4 CTAs).
// Bound: the latency of its loads and of the codec's chains at 20 warps per
// SM, half issue; it moves 1,208 MB for 1,116 MB of algorithmic bytes (96
// registers spill 44 bytes a thread). 1M / 1080p 306 -> 268 us,
// 8.4M / 2160p 2,364 -> 2,006 us (4.4 TB/s) against the layout with every row
// staged at 4 CTAs; 4 CTAs 275 us, 6 CTAs (80 registers, more spills) 308 us, CTAs
// of 64 and 32 rows 267 and 286 us (2,040 and 2,209 us at 8.4M).
#include <cuda_fp16.h>

#include <algorithm>

#include "adjoint.cuh"
#include "common.cuh"
#include "kernels.h"

namespace gsb {

constexpr int kGBlock = 128;
constexpr int kShStride = 49; // padded float row (odd: conflict-free per-thread walks)

// ------------------------------------------------------------------ Adam --
__device__ __forceinline__ void adam_one(float* param, size_t idx, float grad, float* first,
                                         float* second, float lr, float b1, float b2, float c1,
                                         float c2, float eps, float lo, float hi) {
    const float prev = param[idx];
    if (!isfinite(prev) || !isfinite(grad)) {
        first[idx] = 0.f;
        second[idx] = 0.f;
        param[idx] = isfinite(prev) ? fminf(fmaxf(prev, lo), hi) : fminf(fmaxf(0.f, lo), hi);
        return;
    }
    const float m = b1 * first[idx] + (1.f - b1) * grad;
    const float v = b2 * second[idx] + (1.f - b2) * grad * grad;
    if (!isfinite(m) || !isfinite(v)) {
        first[idx] = 0.f;
        second[idx] = 0.f;
        param[idx] = fminf(fmaxf(prev, lo), hi);
        return;
    }
    first[idx] = m;
    second[idx] = v;
    const float cand = prev - lr * (m / c1) / (sqrtf(v / c2) + eps);
    const float upd = isfinite(cand) ? cand : prev;
    param[idx] = fminf(fmaxf(upd, lo), hi);
}

// Adam on register values (same arithmetic as adam_one); returns the new
// parameter and updates m / v in place.
__device__ __forceinline__ float adam_reg(float prev, float grad, float& m, float& v, float lr,
                                          float b1, float b2, float c1, float c2, float eps,
                                          float lo, float hi) {
    if (!isfinite(prev) || !isfinite(grad)) {
        m = 0.f;
        v = 0.f;
        return isfinite(prev) ? fminf(fmaxf(prev, lo), hi) : fminf(fmaxf(0.f, lo), hi);
    }
    const float mm = b1 * m + (1.f - b1) * grad;
    const float vv = b2 * v + (1.f - b2) * grad * grad;
    if (!isfinite(mm) || !isfinite(vv)) {
        m = 0.f;
        v = 0.f;
        return fminf(fmaxf(prev, lo), hi);
    }
    m = mm;
    v = vv;
    const float cand = prev - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    const float upd = isfinite(cand) ? cand : prev;
    return fminf(fmaxf(upd, lo), hi);
}

// Shape priors on (log scale, quaternion) (render_backward.cu:552-648).
// Works on private copies (dynamic axis indices put them in local memory) and
// adds the result to the caller's register arrays with constant indices.
struct PriorGrad {
    float log_s[3];
    float quat[4];
};

__device__ __noinline__ PriorGrad shape_priors_delta(float ls0, float ls1, float ls2, float q0,
                                                     float q1, float q2, float q3,
                                                     const StructureAdamArgs a) {
    const float ls[3] = {ls0, ls1, ls2};
    const float q[4] = {q0, q1, q2, q3};
    PriorGrad out;
    float* g_log = out.log_s;
    float* g_quat = out.quat;
    for (int k = 0; k < 3; ++k) g_log[k] = 0.f;
    for (int k = 0; k < 4; ++k) g_quat[k] = 0.f;
    if (a.shape_quat_norm_reg > 0.f) {
        const float ns = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        if (ns > 1e-20f) {
            const float nrm = sqrtf(ns);
            const float f = a.shape_quat_norm_reg * (nrm - 1.f) / ns;
            for (int c = 0; c < 4; ++c)
                g_quat[c] += f * q[c];
        }
    }
    if (a.shape_axis_ratio_reg > 0.f) {
        int hi = 0, lo = 0;
        for (int k = 1; k < 3; ++k) {
            if (ls[k] > ls[hi]) hi = k;
            if (ls[k] < ls[lo]) lo = k;
        }
        const float excess = ls[hi] - ls[lo] - logf(a.shape_max_axis_ratio);
        if (excess > 0.f && isfinite(excess)) {
            g_log[hi] += a.shape_axis_ratio_reg * excess;
            g_log[lo] -= a.shape_axis_ratio_reg * excess;
        }
    }
    if (a.shape_erank_reg <= 0.f && a.shape_erank_s3_reg <= 0.f)
        return out;
    float l[3];
    int largest = 0;
    for (int k = 0; k < 3; ++k) {
        l[k] = ls[k];
        if (!(l[k] > -1e4f)) l[k] = -1e4f;
        if (k > 0 && l[k] > l[largest]) largest = k;
    }
    float x[3];
    for (int k = 0; k < 3; ++k)
        x[k] = expf(2.f * (l[k] - l[largest]));
    const float sum = x[0] + x[1] + x[2];
    if (!(sum > 0.f))
        return out;
    int smallest = 0;
    for (int k = 1; k < 3; ++k)
        if (x[k] < x[smallest]) smallest = k;
    const float p_large = x[largest] / sum;
    const float raw_small = x[smallest] / sum;
    const bool small_clamped = !(raw_small > 1e-30f);
    const float p_small = small_clamped ? 1e-30f : raw_small;
    const float mid_c = 1.f - p_large - p_small;
    const bool mid_clamped = !(mid_c > 1e-30f);
    const float p_mid = mid_clamped ? 1e-30f : mid_c;
    const float entropy = -(p_large * logf(p_large) + p_mid * logf(p_mid) + p_small * logf(p_small));
    const float rank = expf(entropy);
    float dshare[3] = {0.f, 0.f, 0.f};
    if (a.shape_erank_reg > 0.f && rank - 0.99999f < 1.f) {
        const float p[3] = {p_large, p_mid, p_small};
        for (int k = 0; k < 3; ++k)
            dshare[k] = a.shape_erank_reg * rank * (logf(p[k]) + 1.f) / (rank - 0.99999f);
    }
    const float d_small_total = dshare[2] + a.shape_erank_s3_reg;
    float dx[3];
    for (int k = 0; k < 3; ++k) {
        const float d_large = k == largest ? (1.f - p_large) / sum : -p_large / sum;
        float d_small = 0.f;
        if (k == smallest) {
            if (!small_clamped) d_small = (1.f - p_small) / sum;
        } else {
            d_small = -p_small / sum;
        }
        const float d_mid = mid_clamped ? 0.f : -(d_large + d_small);
        dx[k] = dshare[0] * d_large + dshare[1] * d_mid + d_small_total * d_small;
    }
    for (int k = 0; k < 3; ++k) {
        if (k == largest) {
            float pull = 0.f;
            for (int o = 0; o < 3; ++o)
                if (o != largest) pull += dx[o] * x[o];
            g_log[k] += -2.f * pull;
        } else {
            g_log[k] += dx[k] * 2.f * x[k];
        }
    }
    return out;
}

// ------------------------------------------------------- SH quant codec --
constexpr float kCodecEps = 1e-15f;

__device__ __forceinline__ float codec_prev_correction(float c, float beta) {
    return beta > 0.f ? fmaxf((c - (1.f - beta)) / beta, 0.f) : 0.f;
}
__device__ __forceinline__ float codec_to_normalized(float m, float v, float c1, float c2,
                                                     float eps) {
    if (c1 <= 0.f || c2 <= 0.f)
        return 0.f;
    return (m / c1) / (sqrtf(fmaxf(v, 0.f) / c2) + eps);
}
// The codec's expm1 / log1p pair (decode / encode of the log second moment)
// runs on the exp / log intrinsics: log values are either 0 (a coefficient
// with no second moment, exact either way) or large (sqrt(v) / 1e-15 >> 1),
// where exp(x) - 1 and log(1 + y) lose nothing; only second moments below
// ~1e-31, far under the update's epsilon, see a difference. With the
// software expm1f / log1pf the kernel took 0.627 ms at 1M Gaussians, with the
// intrinsics 0.568 ms.
__device__ __forceinline__ float codec_log_to_second(float log_s) {
    const float s = kCodecEps * (__expf(log_s) - 1.f);
    return s * s;
}

// One coefficient of one row, on registers. `first` is the stored fp16
// normalised update (as float) on entry and the new one on exit, `param` the
// coefficient before and after; returns the log-second value to re-encode.
__device__ __forceinline__ float sh_adam_column(int col, int active, float& param, float grad_in,
                                                float& first, unsigned code, float lo, float hi,
                                                const ShAdamArgs& a) {
    float log_s = lo + (hi - lo) * (float(code) * (1.f / 255.f));
    const float g2 = codec_log_to_second(log_s);
    const float stored = first;
    const float pc1 = codec_prev_correction(a.correction1, a.beta1);
    const float pc2 = codec_prev_correction(a.correction2, a.beta2);
    float g1 = 0.f;
    if (pc1 > 0.f) {
        const float sv = pc2 > 0.f ? sqrtf(fmaxf(g2, 0.f) / pc2) : 0.f;
        g1 = stored * (sv + a.epsilon) * pc1;
    }
    if (col >= active) {
        if (!isfinite(g1)) g1 = 0.f;
        if (!isfinite(log_s)) {
            log_s = 0.f;
            g1 = 0.f;
        }
        const float enc = codec_to_normalized(g1, codec_log_to_second(log_s), a.correction1,
                                              a.correction2, a.epsilon);
        first = isfinite(enc) ? enc : 0.f;
        return log_s;
    }
    float grad = grad_in;
    const float prev = param;
    if (a.regularization > 0.f && col >= 3 && isfinite(prev))
        grad += a.regularization * prev;
    if (!isfinite(prev) || !isfinite(grad)) {
        first = 0.f;
        param = isfinite(prev) ? prev : 0.f;
        return 0.f;
    }
    const float m = a.beta1 * g1 + (1.f - a.beta1) * grad;
    const float v = a.beta2 * g2 + (1.f - a.beta2) * grad * grad;
    if (!isfinite(m) || !isfinite(v)) {
        first = 0.f;
        return 0.f;
    }
    const float lr = col >= 3 ? a.rest_lr : a.lr;
    const float nrm = codec_to_normalized(m, v, a.correction1, a.correction2, a.epsilon);
    const float cand = prev - lr * nrm;
    param = isfinite(cand) ? cand : prev;
    first = nrm;
    float ls = __logf(1.f + sqrtf(fmaxf(v, 0.f)) * (1.f / kCodecEps));
    if (!isfinite(ls)) ls = 0.f;
    return ls;
}

// inv_range = 1 / max(hi - lo, eps), computed once per row and group (the
// division it replaces is the same reciprocal-multiply under fast math).
__device__ __forceinline__ uint8_t codec_encode(float value, float lo, float inv_range) {
    const float code = fminf(fmaxf(roundf(255.f * (value - lo) * inv_range), 0.f), 255.f);
    return static_cast<uint8_t>(code);
}

// ---------------------------------------------- SH Adam, degree-3 rows --
// The common case (48 coefficients per row, all active) on a shorter
// instruction path with the same arithmetic: launch constants are folded once
// per thread; sqrt(v / c2) is sqrt(v) / sqrt(c2) and sqrt(g2 / pc2) is
// |s| / sqrt(pc2), so one square root per coefficient serves the update and
// the re-encoded log value; the u8 code becomes a float and the re-encode
// rounding becomes an integer without conversion instructions (the special
// function unit was the kernel's busiest pipe); fp16 moments move as half2
// pairs and codes as 32-bit words.
struct ShAdamConsts {
    float pc1, rs_pc2;    // previous-step corrections: pc1 (0: no first moment), 1/sqrt(pc2)
    float b1, ob1, b2, ob2;
    float ic1, rs_c2;     // 1/c1, 1/sqrt(c2)
    float eps, lr, rest_lr, reg;
    bool norm_ok;         // c1 > 0 and c2 > 0
};

__device__ __forceinline__ ShAdamConsts sh_adam_consts(const ShAdamArgs& a) {
    ShAdamConsts k;
    const float pc1 = codec_prev_correction(a.correction1, a.beta1);
    const float pc2 = codec_prev_correction(a.correction2, a.beta2);
    k.pc1 = pc1;
    k.rs_pc2 = pc2 > 0.f ? 1.f / sqrtf(pc2) : 0.f;
    k.b1 = a.beta1;
    k.ob1 = 1.f - a.beta1;
    k.b2 = a.beta2;
    k.ob2 = 1.f - a.beta2;
    k.norm_ok = a.correction1 > 0.f && a.correction2 > 0.f;
    k.ic1 = k.norm_ok ? 1.f / a.correction1 : 0.f;
    k.rs_c2 = k.norm_ok ? 1.f / sqrtf(a.correction2) : 0.f;
    k.eps = a.epsilon;
    k.lr = a.lr;
    k.rest_lr = a.rest_lr;
    k.reg = fmaxf(a.regularization, 0.f); // a negative factor or a NaN is no term
    return k;
}

// One active coefficient: code (as float) -> previous moments -> Adam ->
// new parameter, new fp16 normalised first moment, returned log-second value.
__device__ __forceinline__ float sh_adam_coef(bool rest, float& param, float grad, float& first,
                                              float code, float lo, float range,
                                              const ShAdamConsts& k) {
    const float log_s = lo + range * (code * (1.f / 255.f));
    const float s = kCodecEps * (__expf(log_s) - 1.f);
    const float g2 = s * s;
    const float g1 = k.pc1 > 0.f ? first * (fabsf(s) * k.rs_pc2 + k.eps) * k.pc1 : 0.f;
    const float prev = param;
    if (rest && k.reg > 0.f && isfinite(prev))
        grad += k.reg * prev;
    if (!isfinite(prev) || !isfinite(grad)) {
        first = 0.f;
        param = isfinite(prev) ? prev : 0.f;
        return 0.f;
    }
    const float m = k.b1 * g1 + k.ob1 * grad;
    const float v = k.b2 * g2 + k.ob2 * grad * grad;
    if (!isfinite(m) || !isfinite(v)) {
        first = 0.f;
        return 0.f;
    }
    const float sv = sqrtf(fmaxf(v, 0.f));
    const float nrm = k.norm_ok ? __fdividef(m * k.ic1, sv * k.rs_c2 + k.eps) : 0.f;
    const float cand = prev - (rest ? k.rest_lr : k.lr) * nrm;
    param = isfinite(cand) ? cand : prev;
    first = nrm;
    const float ls = __logf(1.f + sv * (1.f / kCodecEps));
    return isfinite(ls) ? ls : 0.f;
}

// sh_adam_coef without its finiteness tests, for the common case: the new
// parameter, first moment and log-second value go to pn, fn and the return
// value, and chk accumulates m, v, the new parameter and the log value. Any
// non-finite input or intermediate the tests would have caught makes chk
// non-finite (inf and NaN propagate through the sums; a finite overflow only
// sends the group to the checked path), and the caller then redoes the group
// with sh_adam_coef; with finite values both give the same results.
__device__ __forceinline__ float sh_adam_coef_fast(bool rest, float prev, float grad, float first,
                                                   float code, float lo, float range,
                                                   const ShAdamConsts& k, float& pn, float& fn,
                                                   float& chk) {
    const float log_s = lo + range * (code * (1.f / 255.f));
    const float s = kCodecEps * (__expf(log_s) - 1.f);
    const float g2 = s * s;
    const float g1 = k.pc1 > 0.f ? first * (fabsf(s) * k.rs_pc2 + k.eps) * k.pc1 : 0.f;
    if (rest && k.reg > 0.f)
        grad += k.reg * prev;
    const float m = k.b1 * g1 + k.ob1 * grad;
    const float v = k.b2 * g2 + k.ob2 * grad * grad;
    const float sv = sqrtf(fmaxf(v, 0.f));
    const float nrm = k.norm_ok ? __fdividef(m * k.ic1, sv * k.rs_c2 + k.eps) : 0.f;
    pn = prev - (rest ? k.rest_lr : k.lr) * nrm;
    fn = nrm;
    const float ls = __logf(1.f + sv * (1.f / kCodecEps));
    chk += (m + v) + (pn + ls);
    return ls;
}

// u8 code (0..255) as a float, exactly, without a conversion instruction.
__device__ __forceinline__ float code_to_float(unsigned code) {
    return __uint_as_float(0x4b000000u | code) - 8388608.f;
}

// roundf(255 * (value - lo) * inv_range) clamped to [0, 255], as an integer:
// floats in [2^22, 2^23) are multiples of a half, so y + (2^22 + 1/2) rounded
// toward zero holds floor(2 y + 1) in its low mantissa bits, and half of that
// is floor(y + 1/2), which is roundf for non-negative values. Clamping before
// rounding gives the same integer (the bounds are integers).
__device__ __forceinline__ unsigned codec_encode_int(float value, float lo, float inv_range) {
    const float y = fminf(fmaxf(255.f * (value - lo) * inv_range, 0.f), 255.f);
    return (__float_as_uint(__fadd_rz(y, 4194304.5f)) >> 1) & 0xffu;
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Calls f(e, r, c) for e = threadIdx.x, + kGBlock, ... < total with
// r = e / stride and c = e % stride, stepping r and c incrementally: one
// integer division per thread instead of one per element (the staging and
// write-back loops run 84 + 48 elements per Gaussian).
template <typename F>
__device__ __forceinline__ void for_row_elements(int total, int stride, F&& f) {
    int e = threadIdx.x;
    int r = e / stride, c = e - r * stride;
    const int dr = kGBlock / stride, dc = kGBlock - dr * stride;
    for (; e < total; e += kGBlock) {
        f(e, r, c);
        r += dr;
        c += dc;
        if (c >= stride) {
            c -= stride;
            ++r;
        }
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
// Starts `bytes` (a multiple of 16) at p, 16-byte aligned, on their way to L2.
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Staging of up to kRowsBlock degree-3 rows (16-byte aligned) for the
// thread-per-row path: thread t copies the 16-byte segments e = t + kRowsBlock
// k of the contiguous block; k -> k + 3 moves on by whole rows, so every copy
// is at a fixed offset from three per-thread bases.
constexpr int kRowsBlock = 128;
constexpr int kRowStride = 52; // floats per staged row: 16-byte reads of eight rows hit every bank
__device__ __forceinline__ void stage_rows48(float* s_coef, const float* src, int rows) {
#pragma unroll
    for (int k0 = 0; k0 < 3; ++k0) {
        constexpr int kStep = kRowsBlock / 4; // rows per three k
        const int e = int(threadIdx.x) + kRowsBlock * k0;
        const int r = e / 12, c = e - 12 * r;
        float* sd = s_coef + r * kRowStride + 4 * c;
        const float* gs = src + 4 * e;
#pragma unroll
        for (int g = 0; g < 4; ++g)
            if (r + kStep * g < rows)
                cp_async16(sd + kStep * kRowStride * g, gs + 48 * kStep * g);
    }
}

// Staging of a full CTA of degree-3 rows (128 rows of 48 coefficients) and,
// with the fused SH Adam, of their fp16 first moments and u8 codes. Thread t
// copies elements e = t + 128k of the CTA's contiguous block; an element's
// padded shared-memory word is e + e / W (W words per row, rows padded by one
// word), and since 3 * 128 is a multiple of W, k -> k + 3 moves both
// addresses by constants. So every copy is one instruction at a fixed offset
// from three per-thread bases, instead of the general loop's index arithmetic
// per element.
__device__ __forceinline__ void stage_full48(float* s_coef, __half* s_first, uint8_t* s_code,
                                             const float* src, const uint32_t* fsrc,
                                             const uint32_t* csrc, bool fused) {
    const int t = threadIdx.x;
#pragma unroll
    for (int k0 = 0; k0 < 3; ++k0) {
        const int e = t + kGBlock * k0;
        float* sd = s_coef + e + e / 48;
        const float* gs = src + e;
#pragma unroll
        for (int g = 0; g < 16; ++g) // W = 48: + 384 elements, + 392 words
            cp_async4(sd + 392 * g, gs + 384 * g);
    }
    if (!fused)
        return;
    uint32_t* sf = reinterpret_cast<uint32_t*>(s_first);
    uint32_t* sc = reinterpret_cast<uint32_t*>(s_code);
#pragma unroll
    for (int k0 = 0; k0 < 3; ++k0) {
        const int e = t + kGBlock * k0;
#pragma unroll
        for (int g = 0; g < 8; ++g) // fp16 pairs, W = 24: + 384 words, + 400 padded
            cp_async4(sf + e + e / 24 + 400 * g, fsrc + e + 384 * g);
#pragma unroll
        for (int g = 0; g < 4; ++g) // code quads, W = 12: + 384 words, + 416 padded
            cp_async4(sc + e + e / 12 + 416 * g, csrc + e + 384 * g);
    }
}

// --------------------------------------------------------------- kernel --
// Fused SH Adam, phase 2 for rows other than 48 active columns: one half-warp
// per row, lanes over the columns (lane l owns columns l, l + 16, l + 32
// below the row stride), reading the row's optimiser state that phase 1
// staged in shared memory and writing the new state to HBM as coalesced row
// segments. The coefficient gradient is rebuilt
// from the row's SH basis values and clamped colour gradient (wdl, written by
// phase 1): w_k * dl.channel, the product the SH adjoint forms. DC and rest
// columns share one instruction path (their learning rate, regulariser and
// code bounds are selected per column), so the DC lanes do not diverge. The
// per-row code bounds are a min / max over the row's log-second values,
// reduced across the half-warp, so the result does not depend on the thread
// layout.
constexpr int kWdlStride = 19; // per row: SH basis values [16], clamped colour gradient [3]
constexpr int kHalfStride = 50; // padded fp16 row = 25 words
constexpr int kCodeStride = 52; // padded u8 row = 13 words

// One row (ok: the row exists; every lane of the warp calls this, the
// shuffles take the whole warp). kAll48: 48 columns, all active (degree-3
// rows) on the fast coefficient path; otherwise the general column step.
template <bool kAll48>
__device__ __forceinline__ void sh_adam_row_half(bool ok, size_t i, int stride, int active, int l,
                                                 const float* coef, const float* wdl,
                                                 const __half* first_row, const uint8_t* code_row,
                                                 float4 bnd, const ShAdamArgs& a,
                                                 const ShAdamConsts& k) {
    float b0 = bnd.x, b1 = bnd.y, b2 = bnd.z, b3 = bnd.w;
    if (!isfinite(b0) || !isfinite(b1)) b0 = b1 = 0.f;
    if (!isfinite(b2) || !isfinite(b3)) b2 = b3 = 0.f;
    const float drange = b1 - b0, rrange = b3 - b2;
    float dmin = 1e30f, dmax = -1e30f, rmin = 1e30f, rmax = -1e30f;
    float ls[3];
    float* param_out = a.parameter + i * size_t(stride);
    __half* first_out = reinterpret_cast<__half*>(a.first) + i * size_t(stride);
#pragma unroll
    for (int kk = 0; kk < 3; ++kk) {
        const int c = l + 16 * kk;
        ls[kk] = 0.f;
        if (!ok || c >= stride)
            continue;
        const int b = c / 3, ch = c - 3 * b;
        const float grad = wdl[b] * wdl[16 + ch];
        float param = coef[c];
        float first = __half2float(first_row[c]);
        const bool rest = c >= 3;
        float lv;
        if constexpr (kAll48) {
            const float cf = code_to_float(code_row[c]);
            const float lo = rest ? b2 : b0, range = rest ? rrange : drange;
            float pn, fn, chk = 0.f;
            lv = sh_adam_coef_fast(rest, param, grad, first, cf, lo, range, k, pn, fn, chk);
            if (isfinite(chk)) {
                param = pn;
                first = fn;
            } else {
                lv = sh_adam_coef(rest, param, grad, first, cf, lo, range, k);
            }
        } else {
            lv = sh_adam_column(c, active, param, grad, first, code_row[c], rest ? b2 : b0,
                                rest ? b3 : b1, a);
        }
        param_out[c] = param;
        first_out[c] = __float2half_rn(first);
        ls[kk] = lv;
        if (rest) {
            rmin = fminf(rmin, lv);
            rmax = fmaxf(rmax, lv);
        } else {
            dmin = fminf(dmin, lv);
            dmax = fmaxf(dmax, lv);
        }
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) {
        dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, off));
        dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, off));
        rmin = fminf(rmin, __shfl_xor_sync(0xffffffffu, rmin, off));
        rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, off));
    }
    if (!ok)
        return;
    if (stride <= 3) rmin = rmax = 0.f;
    if (l == 0)
        reinterpret_cast<float4*>(a.bounds)[i] = make_float4(dmin, dmax, rmin, rmax);
    const float inv_d = 1.f / fmaxf(dmax - dmin, kCodecEps);
    const float inv_r = 1.f / fmaxf(rmax - rmin, kCodecEps);
    uint8_t* code_out = a.packed + i * size_t(stride);
#pragma unroll
    for (int kk = 0; kk < 3; ++kk) {
        const int c = l + 16 * kk;
        if (c >= stride)
            continue;
        const bool rest = c >= 3;
        if constexpr (kAll48)
            code_out[c] = uint8_t(codec_encode_int(ls[kk], rest ? rmin : dmin, rest ? inv_r : inv_d));
        else
            code_out[c] = codec_encode(ls[kk], rest ? rmin : dmin, rest ? inv_r : inv_d);
    }
}

// Fused SH Adam, phase 2 for degree-3 rows (48 columns, all active), one
// thread per row. Only the parameters pass through shared memory (the SH
// adjoint reads them too): the row's fp16 first moments and codes are the
// thread's own, read and written as 16- and 8-byte segments of its row, which
// leaves 284 bytes of shared memory per Gaussian and five CTAs per SM (440
// bytes and four CTAs with every row staged). Columns go in pairs on f32x2
// instructions, element by element the arithmetic of sh_adam_coef, in two
// halves of 24 columns; the coefficient gradients come from the row's basis
// values and clamped colour gradient; the log-second values take the
// parameters' shared slots for the encode pass.

struct CheckedCoef {
    float param, first, ls;
};

__device__ __noinline__ CheckedCoef sh_adam_coef_checked(bool rest, float param, float grad,
                                                         float first, float code, float lo,
                                                         float range, const ShAdamConsts& k) {
    CheckedCoef o{param, first, 0.f};
    o.ls = sh_adam_coef(rest, o.param, grad, o.first, code, lo, range, k);
    return o;
}

// Finiteness of a group is read off chk: a NaN or infinity in m or v reaches
// the new parameter or the log value, whose sum it makes non-finite; the group
// is then redone by sh_adam_coef.
__device__ __forceinline__ void sh_adam_row48(float* prow, uint4* frow, uint2* crow,
                                              const float* wdl, float4 bnd, float* pout,
                                              float4* bout, const ShAdamConsts& k) {
    float b0 = bnd.x, b1 = bnd.y, b2 = bnd.z, b3 = bnd.w;
    if (!isfinite(b0) || !isfinite(b1)) b0 = b1 = 0.f;
    if (!isfinite(b2) || !isfinite(b3)) b2 = b3 = 0.f;
    const float drange = b1 - b0, rrange = b3 - b2;
    float dmin = 1e30f, dmax = -1e30f, rmin = 1e30f, rmax = -1e30f;
    const float d[3] = {wdl[16], wdl[17], wdl[18]};
#pragma unroll 1
    for (int h = 0; h < 2; ++h) { // columns 24 h ... 24 h + 23
        uint4 fw[3];
        uint2 cw[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            fw[j] = frow[3 * h + j];
            cw[j] = crow[3 * h + j];
        }
        // the first three columns of the first half are the DC coefficient
        const float lo0 = h ? b2 : b0, range0 = h ? rrange : drange;
        const float lr0 = h ? k.rest_lr : k.lr, reg0 = h ? k.reg : 0.f;
        unsigned* fws = reinterpret_cast<unsigned*>(fw);
        const unsigned* cws = reinterpret_cast<const unsigned*>(cw);
        float mn0 = 1e30f, mx0 = -1e30f;
#pragma unroll
        for (int g = 0; g < 6; ++g) { // four columns
            const float4 p4 = *reinterpret_cast<const float4*>(prow + 24 * h + 4 * g);
            const float pv[4] = {p4.x, p4.y, p4.z, p4.w};
            float gv[4], cf[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = 4 * g + j;
                gv[j] = wdl[8 * h + c / 3] * d[c % 3];
                cf[j] = __uint_as_float(0x4b000000u | ((cws[g] >> (8 * j)) & 0xffu));
            }
            float pn[4], fn[4], ln[4];
            float2 chk = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 2; ++q) { // a pair: columns j = 2 q, 2 q + 1
                const bool dc0 = g == 0, dc1 = g == 0 && q == 0; // may be DC columns
                const float2 lo = make_float2(dc0 ? lo0 : b2, dc1 ? lo0 : b2);
                const float2 range = make_float2(dc0 ? range0 : rrange, dc1 ? range0 : rrange);
                const float2 nlr = make_float2(dc0 ? -lr0 : -k.rest_lr, dc1 ? -lr0 : -k.rest_lr);
                const float2 reg = make_float2(dc0 ? reg0 : k.reg, dc1 ? reg0 : k.reg);
                const float2 prev = make_float2(pv[2 * q], pv[2 * q + 1]);
                const float2 code = __fadd2_rn(make_float2(cf[2 * q], cf[2 * q + 1]),
                                               make_float2(-8388608.f, -8388608.f));
                const float2 log_s = __ffma2_rn(
                    range, __fmul2_rn(code, make_float2(1.f / 255.f, 1.f / 255.f)), lo);
                const float2 s = __fmul2_rn(
                    make_float2(kCodecEps, kCodecEps),
                    __fadd2_rn(make_float2(__expf(log_s.x), __expf(log_s.y)),
                               make_float2(-1.f, -1.f)));
                const float2 g2 = __fmul2_rn(s, s);
                const float2 first =
                    __half22float2(*reinterpret_cast<const __half2*>(&fws[2 * g + q]));
                const float2 g1 = __fmul2_rn(
                    __fmul2_rn(first, __ffma2_rn(make_float2(fabsf(s.x), fabsf(s.y)),
                                                 make_float2(k.rs_pc2, k.rs_pc2),
                                                 make_float2(k.eps, k.eps))),
                    make_float2(k.pc1, k.pc1));
                const float2 grad =
                    __ffma2_rn(reg, prev, make_float2(gv[2 * q], gv[2 * q + 1]));
                const float2 m = __ffma2_rn(make_float2(k.ob1, k.ob1), grad,
                                            __fmul2_rn(make_float2(k.b1, k.b1), g1));
                const float2 v = __ffma2_rn(__fmul2_rn(make_float2(k.ob2, k.ob2), grad), grad,
                                            __fmul2_rn(make_float2(k.b2, k.b2), g2));
                const float2 sv = make_float2(sqrtf(fmaxf(v.x, 0.f)), sqrtf(fmaxf(v.y, 0.f)));
                const float2 num = __fmul2_rn(m, make_float2(k.ic1, k.ic1));
                const float2 den = __ffma2_rn(sv, make_float2(k.rs_c2, k.rs_c2),
                                              make_float2(k.eps, k.eps));
                const float2 nrm =
                    make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
                const float2 np = __ffma2_rn(nlr, nrm, prev);
                const float2 one_sv = __ffma2_rn(
                    sv, make_float2(1.f / kCodecEps, 1.f / kCodecEps), make_float2(1.f, 1.f));
                const float2 ls = make_float2(__logf(one_sv.x), __logf(one_sv.y));
                chk = __fadd2_rn(chk, __fadd2_rn(np, ls));
                pn[2 * q] = np.x;
                pn[2 * q + 1] = np.y;
                fn[2 * q] = nrm.x;
                fn[2 * q + 1] = nrm.y;
                ln[2 * q] = ls.x;
                ln[2 * q + 1] = ls.y;
            }
            if (!k.norm_ok || !isfinite(chk.x + chk.y)) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool dc = g == 0 && j < 3 && h == 0;
                    const __half2 fp = *reinterpret_cast<const __half2*>(&fws[2 * g + j / 2]);
                    const CheckedCoef o = sh_adam_coef_checked(
                        !dc, pv[j], gv[j], j & 1 ? __high2float(fp) : __low2float(fp),
                        cf[j] - 8388608.f, dc ? b0 : b2, dc ? drange : rrange, k);
                    pn[j] = o.param;
                    fn[j] = o.first;
                    ln[j] = o.ls;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (g == 0 && j < 3) {
                    mn0 = fminf(mn0, ln[j]);
                    mx0 = fmaxf(mx0, ln[j]);
                } else {
                    rmin = fminf(rmin, ln[j]);
                    rmax = fmaxf(rmax, ln[j]);
                }
            }
            *reinterpret_cast<float4*>(pout + 24 * h + 4 * g) =
                make_float4(pn[0], pn[1], pn[2], pn[3]);
            *reinterpret_cast<float4*>(prow + 24 * h + 4 * g) =
                make_float4(ln[0], ln[1], ln[2], ln[3]);
            const __half2 f01 = __floats2half2_rn(fn[0], fn[1]);
            const __half2 f23 = __floats2half2_rn(fn[2], fn[3]);
            fws[2 * g] = *reinterpret_cast<const unsigned*>(&f01);
            fws[2 * g + 1] = *reinterpret_cast<const unsigned*>(&f23);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
            frow[3 * h + j] = fw[j];
        if (h == 0) {
            dmin = mn0;
            dmax = mx0;
        } else {
            rmin = fminf(rmin, mn0);
            rmax = fmaxf(rmax, mx0);
        }
    }
    *bout = make_float4(dmin, dmax, rmin, rmax);
    const float inv_d = 1.f / fmaxf(dmax - dmin, kCodecEps);
    const float inv_r = 1.f / fmaxf(rmax - rmin, kCodecEps);
#pragma unroll 1
    for (int h = 0; h < 6; ++h) { // eight columns
        unsigned w[2];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const float4 l4 = *reinterpret_cast<const float4*>(prow + 8 * h + 4 * g);
            const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
            w[g] = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool dc = g == 0 && j < 3 && h == 0;
                w[g] |= codec_encode_int(lv[j], dc ? dmin : rmin, dc ? inv_d : inv_r) << (8 * j);
            }
        }
        crow[h] = make_uint2(w[0], w[1]);
    }
}

// kRows48: the fused SH Adam on degree-3 rows with all columns active and
// 16-byte aligned state (sh_adam_row48); the other layouts and degrees take
// the half-warp rows.
template <bool kFusedStruct, bool kFusedSH, bool kGeo, bool kRows48>
__global__ void __launch_bounds__(kRows48 ? kRowsBlock : kGBlock,
                                  kRows48 && !kGeo ? 5 : 4) gaussian_backward_kernel(
    int n, const float* __restrict__ means, const float* __restrict__ log_scales,
    const float* __restrict__ quats, const float* __restrict__ logits,
    const float* __restrict__ filter_3d, const float* __restrict__ sh, int sh_degree,
    int sh_bases, const Camera K, GaussianState st, const int* __restrict__ radii,
    GradOutArgs out, StructureAdamArgs sa, ShAdamArgs sha) {
    extern __shared__ float smem[];
    // Shared memory: SH rows [kGBlock][kShStride] floats, then with the fused
    // SH Adam the basis / colour-gradient rows [kGBlock][kWdlStride], fp16
    // first moments [kGBlock][kHalfStride], u8 codes [kGBlock][kCodeStride]
    // and code bounds [kGBlock] float4; without it the coefficient gradients
    // [kGBlock][kShStride].
    // kRows48: SH rows [kGBlock][kRowStride] and basis rows [kGBlock][kWdlStride].
    constexpr int kCoefStride = kRows48 ? kRowStride : kShStride;
    float* s_coef = smem;
    constexpr int kRows = kRows48 ? kRowsBlock : kGBlock;
    float* s_aux = smem + kRows * kCoefStride;
    __half* s_first = reinterpret_cast<__half*>(s_aux + kGBlock * kWdlStride);
    uint8_t* s_code = reinterpret_cast<uint8_t*>(s_first + kGBlock * kHalfStride);
    float4* s_bnd = reinterpret_cast<float4*>(s_code + kGBlock * kCodeStride);
    const int tid = threadIdx.x;
    const int row0 = blockIdx.x * kRows;
    const int rows = min(kRows, n - row0);
    const int stride = sh ? sh_bases * 3 : 0;
    // 1. Asynchronous, coalesced staging of this CTA's SH rows (contiguous),
    //    and with fused SH Adam of their fp16 first moments, u8 codes and code
    //    bounds.
    if constexpr (kRows48) {
        stage_rows48(s_coef, sh + size_t(row0) * 48, rows);
        // the rows that the Adam reads later start their way from HBM
        if (tid == 0) {
            prefetch_l2(reinterpret_cast<const __half*>(sha.first) + size_t(row0) * 48,
                        unsigned(rows) * 96u);
            prefetch_l2(sha.packed + size_t(row0) * 48, unsigned(rows) * 48u);
        }
    } else if (stride == 48 && rows == kGBlock &&
               (!kFusedSH || ((reinterpret_cast<uintptr_t>(sha.first) |
                               reinterpret_cast<uintptr_t>(sha.packed)) & 3) == 0)) {
        // (moments and codes that are not 4-byte aligned go element by element)
        stage_full48(s_coef, s_first, s_code, sh + size_t(row0) * 48,
                     kFusedSH ? reinterpret_cast<const uint32_t*>(
                                    reinterpret_cast<const __half*>(sha.first) + size_t(row0) * 48)
                              : nullptr,
                     kFusedSH ? reinterpret_cast<const uint32_t*>(sha.packed + size_t(row0) * 48)
                              : nullptr,
                     kFusedSH);
    } else if (sh) {
        const float* src = sh + size_t(row0) * stride;
        const int total = rows * stride;
        for_row_elements(total, stride, [&](int e, int r, int c) {
            cp_async4(s_coef + r * kShStride + c, src + e);
        });
        if constexpr (kFusedSH) {
            const __half* fsrc = reinterpret_cast<const __half*>(sha.first) + size_t(row0) * stride;
            const uint8_t* csrc = sha.packed + size_t(row0) * stride;
            for_row_elements(total, stride, [&](int e, int r, int c) {
                s_first[r * kHalfStride + c] = fsrc[e];
                s_code[r * kCodeStride + c] = csrc[e];
            });
        }
    }
    if constexpr (kFusedSH && !kRows48)
        if (sh && tid < rows)
            s_bnd[tid] = reinterpret_cast<const float4*>(sha.bounds)[row0 + tid];
    // 2. Meanwhile every per-Gaussian input of this thread is loaded up front.
    const int i = row0 + tid;
    const bool valid = tid < rows;
    const bool visible = valid && radii[i] > 0;
    float3 mean = make_float3(0.f, 0.f, 0.f);
    float4 g0 = make_float4(0.f, 0.f, 0.f, 0.f), g1 = g0, g2 = g0;
    unsigned clamp_bits = 0;
    Activated act{};
    if (valid) {
        mean = make_float3(means[3 * i], means[3 * i + 1], means[3 * i + 2]);
        act = activate(log_scales, quats, logits, filter_3d, i);
    }
    float4 gplane = make_float4(0.f, 0.f, 0.f, 0.f), gnorm = gplane;
    if (visible) {
        const float4* gslot = st.grad + size_t(i) * kGradSlots;
        g0 = gslot[0];
        g1 = gslot[1];
        g2 = gslot[2];
        clamp_bits = __float_as_uint(st.rec[i].rgb.w);
        if constexpr (kGeo) {
            gplane = st.geo_grad[size_t(i) * kGeoGradSlots];
            gnorm = st.geo_grad[size_t(i) * kGeoGradSlots + 1];
        }
    }
    // Structure Adam state, loaded before any arithmetic so all requests are
    // in flight together: parameters p*, first moments m*, second moments v*.
    float pm[3], mm_[3], vm[3], pl[3], ml[3], vl[3], pq[4], mq[4], vq[4], po = 0.f, mo = 0.f,
        vo = 0.f;
    if constexpr (kFusedStruct) {
        if (valid) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                pm[k] = sa.means[3 * i + k];
                mm_[k] = sa.means_first[3 * i + k];
                vm[k] = sa.means_second[3 * i + k];
                pl[k] = sa.log_scales[3 * i + k];
                ml[k] = sa.scales_first[3 * i + k];
                vl[k] = sa.scales_second[3 * i + k];
            }
            const float4 q4 = reinterpret_cast<const float4*>(sa.quaternions)[i];
            const float4 mq4 = reinterpret_cast<const float4*>(sa.rotations_first)[i];
            const float4 vq4 = reinterpret_cast<const float4*>(sa.rotations_second)[i];
            pq[0] = q4.x; pq[1] = q4.y; pq[2] = q4.z; pq[3] = q4.w;
            mq[0] = mq4.x; mq[1] = mq4.y; mq[2] = mq4.z; mq[3] = mq4.w;
            vq[0] = vq4.x; vq[1] = vq4.y; vq[2] = vq4.z; vq[3] = vq4.w;
            po = sa.opacity_logits[i];
            mo = sa.opacity_first[i];
            vo = sa.opacity_second[i];
        }
    }
    // Rows of visible Gaussians are written whole by the SH adjoint below.
    float* wdl = s_aux + tid * kWdlStride;
    float* grow = s_aux + tid * kShStride;
    if (!visible) {
        if constexpr (kFusedSH)
            for (int c = 0; c < kWdlStride; ++c)
                wdl[c] = 0.f;
        else
            for (int c = 0; c < stride; ++c)
                grow[c] = 0.f;
    }
    if (sh)
        cp_async_wait_all();
    __syncthreads();

    // 3. Adjoints.
    ProjGrad pg;
    pg.d_mean = make_float3(0.f, 0.f, 0.f);
    pg.d_scale = make_float3(0.f, 0.f, 0.f);
    pg.d_rot = make_float4(0.f, 0.f, 0.f, 0.f);
    pg.d_opac = 0.f;
    if (visible) {
        float4* gslot = st.grad + size_t(i) * kGradSlots;
        gslot[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        gslot[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        gslot[2] = make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (kGeo) {
            st.geo_grad[size_t(i) * kGeoGradSlots] = make_float4(0.f, 0.f, 0.f, 0.f);
            st.geo_grad[size_t(i) * kGeoGradSlots + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
            pg = projection_backward<true>(mean, K, act.scale, act.rot, g0,
                                           make_float2(g1.x, g1.y), gplane,
                                           make_float3(gnorm.x, gnorm.y, gnorm.z));
        } else {
            pg = projection_backward(mean, K, act.scale, act.rot, g0, make_float2(g1.x, g1.y));
        }
        const float3 dcol = make_float3(g2.x, g2.y, g2.z);
        if (sh) {
            const float3 campos = make_float3(K.center[0], K.center[1], K.center[2]);
            float3 dm;
            const float3* crow = reinterpret_cast<const float3*>(s_coef + tid * kCoefStride);
            if constexpr (kRows48) {
                float4 q[12];
#pragma unroll
                for (int k = 0; k < 12; ++k)
                    q[k] = reinterpret_cast<const float4*>(crow)[k];
                const float* f = reinterpret_cast<const float*>(q);
                float3 c[16];
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    c[k] = make_float3(f[3 * k], f[3 * k + 1], f[3 * k + 2]);
                dm = sh_color_backward<true>(c, 3, 16, mean, campos, clamp_bits, dcol, nullptr,
                                             wdl);
            } else if constexpr (kFusedSH)
                dm = sh_color_backward<true>(crow, sh_degree, sh_bases, mean, campos, clamp_bits,
                                             dcol, nullptr, wdl);
            else
                dm = sh_color_backward(crow, sh_degree, sh_bases, mean, campos, clamp_bits, dcol,
                                       reinterpret_cast<float3*>(grow));
            pg.d_mean.x += dm.x;
            pg.d_mean.y += dm.y;
            pg.d_mean.z += dm.z;
        } else if (out.colors) {
            out.colors[3 * i + 0] += dcol.x;
            out.colors[3 * i + 1] += dcol.y;
            out.colors[3 * i + 2] += dcol.z;
        }
        if (out.refine_weight) out.refine_weight[i] += g1.z;
        if (out.densify_weight) out.densify_weight[i] += g1.w;
        if (out.densify_weight_den) out.densify_weight_den[i] += g2.w;
    }

    // 4. Structure: fused Adam or gradient outputs.
    if (valid) {
        if constexpr (kFusedStruct) {
            // Chain to raw parameters (update_structure_adam_row), priors, Adam.
            RawGrad rg;
            {
                const float f2 = sa.filter_3d ? sa.filter_3d[i] * sa.filter_3d[i] : 0.f;
                const float ds[3] = {pg.d_scale.x, pg.d_scale.y, pg.d_scale.z};
    #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float raw = (&act.raw_scale.x)[k];
                    const float sc = (&act.scale.x)[k];
                    rg.log_s[k] = ds[k] * raw * raw / sc + pg.d_opac * act.opacity * f2 / (sc * sc);
                }
                const float inv = rsqrtf(fmaxf(pq[0] * pq[0] + pq[1] * pq[1] + pq[2] * pq[2] +
                                                   pq[3] * pq[3], 1e-20f));
                const float q[4] = {pq[0] * inv, pq[1] * inv, pq[2] * inv, pq[3] * inv};
                const float dr[4] = {pg.d_rot.x, pg.d_rot.y, pg.d_rot.z, pg.d_rot.w};
                const float qdot = q[0] * dr[0] + q[1] * dr[1] + q[2] * dr[2] + q[3] * dr[3];
    #pragma unroll
                for (int k = 0; k < 4; ++k)
                    rg.quat[k] = inv * (dr[k] - q[k] * qdot);
            }
            const float sig = 1.f / (1.f + expf(-po));
            float g_log[3] = {rg.log_s[0], rg.log_s[1], rg.log_s[2]};
            float g_quat[4] = {rg.quat[0], rg.quat[1], rg.quat[2], rg.quat[3]};
            float g_logit = pg.d_opac * act.opacity * (1.f - sig);
            if (isfinite(po) && sa.opacity_reg > 0.f)
                g_logit += sa.opacity_reg * sig * (1.f - sig);
            if (sa.scale_reg > 0.f)
    #pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (isfinite(pl[k]) && pl[k] > -40.f) g_log[k] += sa.scale_reg * expf(pl[k]);
            if (sa.shape_quat_norm_reg > 0.f || sa.shape_axis_ratio_reg > 0.f ||
                sa.shape_erank_reg > 0.f || sa.shape_erank_s3_reg > 0.f) {
                const PriorGrad pr =
                    shape_priors_delta(pl[0], pl[1], pl[2], pq[0], pq[1], pq[2], pq[3], sa);
    #pragma unroll
                for (int k = 0; k < 3; ++k) g_log[k] += pr.log_s[k];
    #pragma unroll
                for (int k = 0; k < 4; ++k) g_quat[k] += pr.quat[k];
            }
            if (sa.opacity_gradient) sa.opacity_gradient[i] = g_logit;
            const float inf = 1.e30f;
            const float gm[3] = {pg.d_mean.x, pg.d_mean.y, pg.d_mean.z};
            float nm[3], nl[3], nq[4];
    #pragma unroll
            for (int c = 0; c < 3; ++c) {
                nm[c] = adam_reg(pm[c], gm[c], mm_[c], vm[c], sa.means_lr, sa.beta1, sa.beta2,
                                 sa.correction1, sa.correction2, sa.epsilon, -inf, inf);
                nl[c] = adam_reg(pl[c], g_log[c], ml[c], vl[c], sa.scales_lr, sa.beta1, sa.beta2,
                                 sa.correction1, sa.correction2, sa.epsilon, sa.minimum_log_scale,
                                 sa.maximum_log_scale);
            }
    #pragma unroll
            for (int c = 0; c < 4; ++c)
                nq[c] = adam_reg(pq[c], g_quat[c], mq[c], vq[c], sa.quaternions_lr, sa.beta1,
                                 sa.beta2, sa.correction1, sa.correction2, sa.epsilon, -inf, inf);
            const float no = adam_reg(po, g_logit, mo, vo, sa.opacities_lr, sa.beta1, sa.beta2,
                                      sa.correction1, sa.correction2, sa.epsilon, -12.f, 12.f);
    #pragma unroll
            for (int c = 0; c < 3; ++c) {
                sa.means[3 * i + c] = nm[c];
                sa.means_first[3 * i + c] = mm_[c];
                sa.means_second[3 * i + c] = vm[c];
                sa.log_scales[3 * i + c] = nl[c];
                sa.scales_first[3 * i + c] = ml[c];
                sa.scales_second[3 * i + c] = vl[c];
            }
            reinterpret_cast<float4*>(sa.quaternions)[i] = make_float4(nq[0], nq[1], nq[2], nq[3]);
            reinterpret_cast<float4*>(sa.rotations_first)[i] = make_float4(mq[0], mq[1], mq[2], mq[3]);
            reinterpret_cast<float4*>(sa.rotations_second)[i] = make_float4(vq[0], vq[1], vq[2], vq[3]);
            sa.opacity_logits[i] = no;
            sa.opacity_first[i] = mo;
            sa.opacity_second[i] = vo;
        } else if (visible) {
            if (out.means) {
                out.means[3 * i + 0] += pg.d_mean.x;
                out.means[3 * i + 1] += pg.d_mean.y;
                out.means[3 * i + 2] += pg.d_mean.z;
            }
            if (out.activated) {
                if (out.scales) {
                    out.scales[3 * i + 0] += pg.d_scale.x;
                    out.scales[3 * i + 1] += pg.d_scale.y;
                    out.scales[3 * i + 2] += pg.d_scale.z;
                }
                if (out.rotations) {
                    out.rotations[4 * i + 0] += pg.d_rot.x;
                    out.rotations[4 * i + 1] += pg.d_rot.y;
                    out.rotations[4 * i + 2] += pg.d_rot.z;
                    out.rotations[4 * i + 3] += pg.d_rot.w;
                }
                if (out.opacities) out.opacities[i] += pg.d_opac;
            } else {
                const RawGrad rg = chain_to_raw(pg, act, quats, logits, filter_3d, i);
                if (out.scales)
                    for (int k = 0; k < 3; ++k) out.scales[3 * i + k] += rg.log_s[k];
                if (out.rotations)
                    for (int k = 0; k < 4; ++k) out.rotations[4 * i + k] += rg.quat[k];
                if (out.opacities) out.opacities[i] += rg.logit;
            }
        }
    }

    // 5. SH: the fused quantized Adam (phase 2, one half-warp per row) or the
    //    coalesced accumulation of the coefficient gradients.
    if constexpr (kRows48) {
        if (valid)
            sh_adam_row48(s_coef + tid * kRowStride,
                          reinterpret_cast<uint4*>(reinterpret_cast<__half*>(sha.first) +
                                                   size_t(i) * 48),
                          reinterpret_cast<uint2*>(sha.packed + size_t(i) * 48), wdl,
                          reinterpret_cast<const float4*>(sha.bounds)[i],
                          sha.parameter + size_t(i) * 48,
                          reinterpret_cast<float4*>(sha.bounds) + i, sh_adam_consts(sha));
    } else if constexpr (kFusedSH) {
        if (!sh)
            return;
        __syncthreads();
        const int active = (sh_degree + 1) * (sh_degree + 1) * 3;
        const ShAdamConsts kc = sh_adam_consts(sha);
        // other strides and degrees: one half-warp per row
        const int l = tid & 15, hw = tid >> 4;
        constexpr int kHalves = kGBlock / 16;       // half-warps per CTA
        constexpr int kPerHalf = kGBlock / kHalves; // rows per half-warp
        for (int k = 0; k < kPerHalf; ++k) {
            const int r = hw + kHalves * k;
            const bool ok = r < rows;
            const float* coef = s_coef + r * kShStride;
            const float* w = s_aux + r * kWdlStride;
            const __half* fr = s_first + r * kHalfStride;
            const uint8_t* cr = s_code + r * kCodeStride;
            const float4 bnd = ok ? s_bnd[r] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (stride == 48 && active == 48)
                sh_adam_row_half<true>(ok, size_t(row0 + r), stride, active, l, coef, w, fr, cr,
                                       bnd, sha, kc);
            else
                sh_adam_row_half<false>(ok, size_t(row0 + r), stride, active, l, coef, w, fr, cr,
                                        bnd, sha, kc);
        }
    } else {
        __syncthreads();
        if (sh && out.sh) {
            float* dst = out.sh + size_t(row0) * stride;
            for_row_elements(rows * stride, stride, [&](int e, int r, int c) {
                dst[e] += s_aux[r * kShStride + c];
            });
        }
    }
}

static size_t gaussian_backward_smem(bool fused_sh, bool rows48) {
    if (rows48)
        return size_t(kRowsBlock) * (kRowStride + kWdlStride) * sizeof(float);
    if (!fused_sh)
        return size_t(kGBlock) * 2 * kShStride * sizeof(float);
    return size_t(kGBlock) * ((kShStride + kWdlStride) * sizeof(float) +
                              kHalfStride * sizeof(__half) + kCodeStride + sizeof(float4));
}

void launch_gaussian_backward(cudaStream_t s, int n, const float* means, const float* log_scales,
                              const float* quats, const float* logits, const float* filter_3d,
                              const float* sh, int sh_degree, int sh_bases, const Camera& K,
                              const GaussianState& st, const int* radii, const GradOutArgs& out,
                              const StructureAdamArgs* sa, const ShAdamArgs* sha, bool geometry) {
    StructureAdamArgs sa0{};
    ShAdamArgs sha0{};
    const bool fs = sa != nullptr, fh = sha != nullptr && sh != nullptr;
    const bool rows48 = fh && sh_bases == 16 && sh_degree == 3 &&
                        ((reinterpret_cast<uintptr_t>(sh) | reinterpret_cast<uintptr_t>(sha->parameter) |
                          reinterpret_cast<uintptr_t>(sha->first) |
                          reinterpret_cast<uintptr_t>(sha->packed)) & 15) == 0;
    const size_t smem = gaussian_backward_smem(fh, rows48);
    const int threads = rows48 ? kRowsBlock : kGBlock;
    const int blocks = (n + threads - 1) / threads;
#define GSB_LAUNCH(FS, FH, GEO, R48)                                                             \
    do {                                                                                         \
        auto kfn = gaussian_backward_kernel<FS, FH, GEO, R48>;                                        \
        static bool attr_set = false;                                                            \
        if (!attr_set) {                                                                         \
            cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));   \
            attr_set = true;                                                                     \
        }                                                                                        \
        kfn<<<blocks, threads, smem, s>>>(n, means, log_scales, quats, logits, filter_3d, sh,    \
                                          sh_degree, sh_bases, K, st, radii, out,                \
                                          sa ? *sa : sa0, sha ? *sha : sha0);                    \
    } while (0)
    if (geometry) {
        if (fs && rows48) GSB_LAUNCH(true, true, true, true);
        else if (rows48) GSB_LAUNCH(false, true, true, true);
        else if (fs && fh) GSB_LAUNCH(true, true, true, false);
        else if (fs) GSB_LAUNCH(true, false, true, false);
        else if (fh) GSB_LAUNCH(false, true, true, false);
        else GSB_LAUNCH(false, false, true, false);
    } else {
        if (fs && rows48) GSB_LAUNCH(true, true, false, true);
        else if (rows48) GSB_LAUNCH(false, true, false, true);
        else if (fs && fh) GSB_LAUNCH(true, true, false, false);
        else if (fs) GSB_LAUNCH(true, false, false, false);
        else if (fh) GSB_LAUNCH(false, true, false, false);
        else GSB_LAUNCH(false, false, false, false);
    }
#undef GSB_LAUNCH
}

// ------------------------------------------------------ standalone kernels --
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, size_t n, float lr,
                            float b1, float b2, float c1, float c2, float eps, float lo, float hi) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n;
         i += size_t(gridDim.x) * blockDim.x)
        adam_one(p, i, g[i], m, v, lr, b1, b2, c1, c2, eps, lo, hi);
}

void launch_adam(cudaStream_t s, float* p, const float* g, float* m, float* v, size_t n, float lr,
                 float b1, float b2, float c1, float c2, float eps, float lo, float hi) {
    if (n == 0) return;
    const int blocks = int(std::min<size_t>((n + kBlock - 1) / kBlock, size_t(148) * 16));
    adam_kernel<<<blocks, kBlock, 0, s>>>(p, g, m, v, n, lr, b1, b2, c1, c2, eps, lo, hi);
}

// L1 over [3,P] images: grad = w/(3P) sign(d), loss += w/(3P) sum |d|.
__device__ __forceinline__ float l1_grad(float d, float scale) {
    return d > 0.f ? scale : (d < 0.f ? -scale : 0.f);
}

// Four elements per thread and step with 16-byte accesses (the images are
// streamed once: HBM-bound), then a scalar tail; one atomic per warp.
__global__ void __launch_bounds__(kBlock) l1_kernel(const float* __restrict__ img,
                                                    const float* __restrict__ tgt, size_t n,
                                                    float scale, float* __restrict__ grad,
                                                    float* __restrict__ loss, bool vec) {
    float acc = 0.f;
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    const size_t first = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    size_t done = 0;
    if (vec) {
        const size_t n4 = n / 4;
        const float4* a4 = reinterpret_cast<const float4*>(img);
        const float4* b4 = reinterpret_cast<const float4*>(tgt);
        float4* g4 = reinterpret_cast<float4*>(grad);
#pragma unroll 2
        for (size_t i = first; i < n4; i += stride) {
            const float4 a = __ldcs(a4 + i), b = __ldcs(b4 + i);
            const float4 d = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
            __stcs(g4 + i, make_float4(l1_grad(d.x, scale), l1_grad(d.y, scale),
                                       l1_grad(d.z, scale), l1_grad(d.w, scale)));
            acc += (fabsf(d.x) + fabsf(d.y)) + (fabsf(d.z) + fabsf(d.w));
        }
        done = n4 * 4;
    }
    for (size_t i = done + first; i < n; i += stride) {
        const float d = img[i] - tgt[i];
        grad[i] = l1_grad(d, scale);
        acc += fabsf(d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    // One global atomic per block (per-warp atomics on one address serialise).
    __shared__ float s_warp[kBlock / 32];
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (loss && threadIdx.x == 0) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kBlock / 32; ++w) sum += s_warp[w];
        atomicAdd(loss, sum * scale);
    }
}

void launch_l1(cudaStream_t s, const float* img, const float* tgt, size_t n, float scale,
               float* grad, float* loss) {
    if (n == 0) return;
    const bool vec = ((reinterpret_cast<uintptr_t>(img) | reinterpret_cast<uintptr_t>(tgt) |
                       reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
    const size_t work = vec ? (n + 3) / 4 : n;
    const int blocks = int(std::min<size_t>((work + kBlock - 1) / kBlock, size_t(148) * 8));
    l1_kernel<<<blocks, kBlock, 0, s>>>(img, tgt, n, scale, grad, loss, vec);
}

} // namespace gsb
