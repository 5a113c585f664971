// pm_sweep_device.cuh -- device helpers of the half-sweep kernels.  Shared by
// pm_slots.cu and pm_sweep.cu: bulk-copy staging and patch windows.  Of the
// warp-per-pixel kernel (pm_sweep.cu) only: the texture unit's blend from quads,
// cross-view proposals and refinement candidates, whole ones per thread (pm_slots.cu
// spreads its own over a half warp's lanes).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "pm_device.cuh"
#include "pm_kernels.h"

namespace pfd {

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ float4 lds_f4(uint32_t addr)
{
    float4 v;
    asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// Linear-filter fetch of the measured texture unit (see Tiles in pm_device.cuh)
// from a quad entry: 256 s = 256 T00 + a (T10 - T00) + b (T01 - T00) + w11 (T11 - T01 - T10 + T00)
// with w11 = (a b + 128) >> 8, regrouped per texel as
// 256 s = T00 w00 + T10 w10 + T01 w01 + T11 w11, w10 = a - w11, w01 = b - w11,
// w00 = 256 - w10 - b: all four weights lie in [0, 256], so two 16-bit pairs of
// weights against the quad's four bytes make the sum with two dp2a, exactly.
struct QuadWeights {
    uint32_t lo;             // w00 | w10 << 16, against T00, T10 (the quad's low bytes)
    uint32_t hi;             // w01 | w11 << 16, against T01, T11
};

// hi = w01 + 65536 w11 = b + 65535 w11, and lo + hi = 256 + 65535 a (w00 + w01 =
// 256 - a, w10 + w11 = a), so lo = 256 + 65535 a - hi: no weight is negative, so
// no half borrows from the other.
__device__ __forceinline__ QuadWeights quad_weights(int tbx, int tby)
{
    const uint32_t a = (uint32_t)tbx & 0xFFu, b = (uint32_t)tby & 0xFFu;
    const uint32_t w11 = (a * b + 128u) >> 8;
    QuadWeights q;
    q.hi = w11 * 65535u + b;
    q.lo = a * 65535u + 256u - q.hi;
    return q;
}

__device__ __forceinline__ float quad_blend(const QuadWeights& w, uint32_t q)
{
    const uint32_t s256 = __dp2a_lo(w.lo, q, __dp2a_hi(w.hi, q, 0u));
    return __fsub_rn(__uint_as_float(s256 | 0x47000000u), 32768.0f);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
// Bounded wait (about 2^22 polls): records PFD_DEVERR_TMA_TIMEOUT and gives up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* err)
{
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (it > 64) __nanosleep(128);
    }
    if (err) atomicOr(err, PFD_DEVERR_TMA_TIMEOUT);
    return false;
}

// The pixel's patch window: the patch's taps (x offset i, y offset j, step inc)
// that fall inside the micro-image, as a rectangle of nX x nY taps.
struct PixWin {
    int x0, y0, nX, nY;      // first tap position and tap counts
    int ii0, jj0;            // offset index of the first tap ((x0 - px + r) / inc)
};

__device__ __forceinline__ PixWin pixel_window(const PmParams& P, int px, int py)
{
    PixWin w;
    const int r = P.radius, inc = P.inc;
    const int sx = max(0, (r - px + inc - 1) / inc), sy = max(0, (r - py + inc - 1) / inc);
    w.ii0 = sx;
    w.jj0 = sy;
    w.x0 = px - r + sx * inc;
    w.y0 = py - r + sy * inc;
    const int ex = min(P.ntap - 1, (P.W - 1 - px + r) / inc), ey = min(P.ntap - 1, (P.H - 1 - py + r) / inc);
    w.nX = max(0, ex - sx + 1);
    w.nY = max(0, ey - sy + 1);
    return w;
}

__device__ __forceinline__ int nth_set_bit(uint32_t m, int n)
{
    for (int i = 0; i < n && m; ++i) m &= m - 1;
    return m ? __ffs(m) - 1 : -1;
}

// BuildCrossViewPlaneProposal (AdaptMIPMFrame.cu:350-398): the sample position
// q (local index) of pixel (x, y) under `cur` in neighbour k, or -1.  This and
// proposal_plane are called from three places each and kept out of line: less
// code between the NCC passes (1.5% of the half-sweep's time, measured).
__device__ __noinline__ int proposal_pos(const NbGeo& gk, int x, int y, int W, int H, float4 cur)
{
    const float dcur = to_disparity(x, y, disparity_plane(x, y, cur));
    const float2 qf = geo_anchor(gk, x, y, dcur);
    const float fqx = floorf(__fadd_rn(qf.x, 0.5f)), fqy = floorf(__fadd_rn(qf.y, 0.5f));
    if (!(fqx >= 0.0f && fqx < (float)W && fqy >= 0.0f && fqy < (float)H)) return -1;
    return (int)fqy * W + (int)fqx;
}

__device__ __noinline__ float4 proposal_plane(const NbGeo& gk, const float4* nb_plane, int q, int x, int y, int W)
{
    const int qx = q % W, qy = q / W;
    const float4 hn = nb_plane[q];
    const float3 dpn = disparity_plane(qx, qy, hn);
    float denom = __fmaf_rn(dpn.y, gk.by, __fmaf_rn(dpn.x, gk.bx, 1.0f));
    denom = safe_denom(denom);
    return encode_plane(x, y, __fdiv_rn(dpn.x, denom), __fdiv_rn(dpn.y, denom), __fdiv_rn(dpn.z, denom));
}

// The five candidates of PlaneHypothesisRefinement_Frame (AdaptMIPMFrame.cu:
// 400-471) for the best plane `best`, from the draws already taken (c0: the
// random plane, rn: the random normal, u1-u3: the perturbation, u4: the depth
// perturbation).
__device__ __noinline__ void refine_candidates(int x, int y, float4 best, float4 c0, float4 rn, float u1, float u2,
                                               float u3, float u4, float pert, float4 (&cand)[5])
{
    const float depth_now = best.w;
    const float4 pn = perturbed_normal_u(x, y, best, u1, u2, u3, pert);
    const float dmin_p = __fmul_rn(__fsub_rn(1.0f, 0.02f), depth_now);
    const float dmax_p = __fmul_rn(__fadd_rn(1.0f, 0.02f), depth_now);
    const float depth_perturbed = __fmaf_rn(u4, __fsub_rn(dmax_p, dmin_p), dmin_p);
    cand[0] = c0;
    cand[1] = rn;
    cand[2] = pn;
    cand[3] = best;
    cand[4] = best;
    cand[4].w = depth_perturbed;
    for (int i = 1; i < 5; ++i) cand[i].w = to_disparity(x, y, disparity_plane(x, y, cand[i]));
}

}  // namespace

}  // namespace pfd
