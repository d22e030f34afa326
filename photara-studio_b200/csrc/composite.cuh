// Pieces shared by the compositing kernels: mbarrier waits and TMA gathers of
// Gaussian records, a view's buffers, the per-pixel adjoint state.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace gsb {

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
// One wait for the phase of `parity`: the thread is suspended until the phase
// completes or about `suspend_ns` pass (a hint, in nanoseconds), instead of
// spinning on issue slots the working warps need. True if it completed.
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity,
                                              unsigned suspend_ns) {
    unsigned done;
    asm volatile("{\n\t.reg .pred P1;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
                 "selp.b32 %0, 1, 0, P1;\n\t}"
                 : "=r"(done)
                 : "r"(smem_u32(bar)), "r"(parity), "r"(suspend_ns)
                 : "memory");
    return done != 0;
}
// Waits for the phase of `parity`, at most `limit` suspended waits of about a
// microsecond each; false if the phase did not complete.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity,
                                                  unsigned limit) {
    for (unsigned k = 0; k < limit; ++k)
        if (mbar_try_wait(bar, parity, 1000u))
            return true;
    return false;
}
constexpr unsigned kStageWaitLimit = 1u << 18; // ~0.26 s at most

// Four 64-byte rows (Gaussian ids r0..r3) of the record tensor into dst
// (256 contiguous bytes), completing on bar. The column coordinate is 0, so
// the copy's innermost offset is 16-byte aligned by construction.
__device__ __forceinline__ void tma_gather4(void* dst, const CUtensorMap* map, int r0, int r1,
                                            int r2, int r3, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(bar)), "r"(0), "r"(r0),
        "r"(r1), "r"(r2), "r"(r3)
        : "memory");
}

// One view's image constants and buffers, already offset to that view.
struct ViewTarget {
    int width, height;
    float clip;
    float3 bg;
    float* color;        // [3][H][W]
    float* alpha;        // [H][W]
    float* pix_T;        // [H][W] final transmittance (NULL: inference only)
    unsigned* pix_last;  // [H][W] 1 + position of the last instance taken while the pixel
                         // was open: at or behind the last blended one, 0 if none was taken
};

struct ViewGrads {
    int width, height;
    float clip;
    float3 bg;
    const float* pix_T;
    const unsigned* pix_last;
    const float* dL_color;
    const float* dL_alpha;    // may be NULL
    const float* densify_map; // may be NULL
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2s(float a) { return make_float2(a, a); }

// Adds a per-lane count to *out with one atomic per warp.
__device__ __forceinline__ void warp_count_add(unsigned long long v, unsigned long long* out) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v)
        atomicAdd(out, v);
}

// Per-pixel backward state.
struct PixBack {
    float T, sdot, gx, gy, gz, fin_term, refine_scale, dmap;
    unsigned last;
};

__device__ __forceinline__ void pixel_backward_init(PixBack& p, bool inside, size_t pid, size_t P,
                                                    float3 bg, const float* __restrict__ pix_T,
                                                    const unsigned* __restrict__ pix_last,
                                                    const float* __restrict__ dL_color,
                                                    const float* __restrict__ dL_alpha,
                                                    const float* __restrict__ densify_map) {
    float T_final = 1.f;
    p.gx = p.gy = p.gz = 0.f;
    p.dmap = 0.f;
    p.last = 0;
    float dfin = 0.f;
    if (inside) {
        T_final = pix_T[pid];
        p.last = pix_last[pid];
        p.gx = dL_color[pid];
        p.gy = dL_color[P + pid];
        p.gz = dL_color[2 * P + pid];
        dfin = bg.x * p.gx + bg.y * p.gy + bg.z * p.gz - (dL_alpha ? dL_alpha[pid] : 0.f);
        p.dmap = densify_map ? densify_map[pid] : 0.f;
    }
    p.refine_scale = 1.f / fmaxf(1.f - T_final, 1.0e-5f);
    p.fin_term = T_final * dfin;
    p.T = T_final;
    p.sdot = 0.f;
}

} // namespace gsb
