// fuse_kernels.cu -- LFRefocus::FuseVirtualDepth_BackProject (FocalStack/
// LFRefocus.cpp:1553-1794) on the device.
//
// The reference visits the reference micro-images in map order and their
// pixels row by row; a pixel that finds at least two consistent neighbour
// pixels becomes a fused point and masks the neighbour pixels it used, which
// everything after it then skips.  Which neighbour pixels are consistent does not
// depend on the masks, so:
//   pm_fuse_pairs_kernel    per (pixel, list entry) the consistent neighbour pixel,
//                           or none.
//   pm_fuse_resolve_kernel  the walk itself, on bits only: one warp per micro-image
//                           goes through its pixels in order with the masks that the
//                           micro-images before it leave, and publishes the pixels it
//                           masks.  All micro-images run side by side; those whose
//                           predecessors changed run again until nothing changes.  A
//                           micro-image depends on earlier ones only, so this ends at
//                           the one solution, the sequential walk's.  A cooperative
//                           launch; the grid barrier's waits are bounded.
//   pm_fuse_fold_kernel     between bands (below), what a band masks for the next ones.
//   pm_fuse_points_kernel   the fused points, one thread per pixel, their neighbours
//                           summed in list order, so every float is the reference's.
// The tests take two bytes per pixel and list entry, so a frame with long lists is walked
// in bands of micro-images, one after the other in map order: a band's walk starts from
// the masks of the bands before it, which are final.
// Points that land on the same raw pixel overwrite each other in map order in
// the reference; here each records its sequence number (micro-image, pixel)
// with atomicMax and the maps are written from the last one afterwards.
//
// A wavefront over the micro-images, one warp each with the tests in its chain of
// loads (0.5 ms per step), took 553 ms on the 4080x3068 frame and 99 ms on the
// 1024x768 one; this form 10 and 1.3 ms (12 list entries), bound by the gathers of
// the pairs kernel and the rounds' walks of 256 dependent steps.
#include <climits>
#include <algorithm>
#include <cstdint>
#include "fuse_kernels.h"
#include "grid_barrier.cuh"
#include "smem_limit.h"

namespace pfd {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr float kInvalidImage = -9999.0f;         // g_Invalid_image, Common/Common.cpp:53

// x86 conversions of the reference's host code: (int) truncates, cvRound
// rounds half to even; NaN and out-of-range values give INT_MIN.
__device__ __forceinline__ int trunc_x86(float x) { return fabsf(x) < 2147483648.0f ? __float2int_rz(x) : INT_MIN; }
__device__ __forceinline__ int round_x86(float x) { return fabsf(x) < 2147483648.0f ? __float2int_rn(x) : INT_MIN; }
__device__ __forceinline__ uint8_t sat_u8(float v)
{
    const int i = round_x86(v);
    return (uint8_t)(i < 0 ? 0 : (i > 255 ? 255 : i));
}

// ComputeVirtualDepth (:2087-2098): a float base over a double disparity.
__device__ __forceinline__ float virtual_depth(float mla_base, float disp)
{
    const double d = (double)disp;
    if (d <= 0.0) return kInvalidImage;
    return __double2float_rn(__ddiv_rn((double)mla_base, d));
}

// ComputeVirtual3D (:2100-2117)
__device__ __forceinline__ float3 virtual_3d(float vd, int col, int row, float cm, float2 c)
{
    return make_float3(__fadd_rn(__fmul_rn(__fsub_rn((float)col, cm), vd), c.x),
                       __fadd_rn(__fmul_rn(__fsub_rn((float)row, cm), vd), c.y), vd);
}

// BackProject2MI (:2119-2125)
__device__ __forceinline__ float2 back_project(float3 P, float2 c, float cm)
{
    return make_float2(__fadd_rn(__fdiv_rn(__fsub_rn(P.x, c.x), P.z), cm),
                       __fadd_rn(__fdiv_rn(__fsub_rn(P.y, c.y), P.z), cm));
}

__device__ __forceinline__ float3 colour(const FuseFrame& F, int v, int idx)
{
    if (F.bgr) {
        const uint8_t* p = F.bgr + ((size_t)v * F.ppv + idx) * 3;
        return make_float3((float)p[0], (float)p[1], (float)p[2]);
    }
    const float g = (float)F.gray[(size_t)v * F.tile_stride + idx];
    return make_float3(g, g, g);
}

__device__ __forceinline__ bool valid_vd(float vd)
{
    return !(fabsf(__fsub_rn(vd, kInvalidImage)) < 1.0e-6f) && isfinite(vd);
}

}  // namespace

// The fused point's neighbour test (:1660-1720): the pixel of list entry u that
// reference pixel (r, c) of view centre cr at virtual depth vdr projects to, when it
// is consistent; -1 otherwise.
__device__ __forceinline__ int consistent_pixel(const FuseFrame& F, float3 P, float vdr, int r, int c, float2 cr, int u,
                                                float2 cu, float cm)
{
    const float2 q = back_project(P, cu, cm);
    const int src_r = trunc_x86(__fadd_rn(q.y, 0.5f)), src_c = trunc_x86(__fadd_rn(q.x, 0.5f));
    if (!(src_c >= 0 && src_c < F.m && src_r >= 0 && src_r < F.m)) return -1;
    const int si = src_r * F.m + src_c;
    const float w = F.plane[(size_t)u * F.ppv + si].w;
    if (w <= 0.0f) return -1;
    const float vds = virtual_depth(F.mla_base, w);
    if (!valid_vd(vds)) return -1;
    const float3 Ps = virtual_3d(vds, src_c, src_r, cm, cu);
    const float2 rq = back_project(Ps, cr, cm);
    const float ex = __fsub_rn((float)c, rq.x), ey = __fsub_rn((float)r, rq.y);
    const float err = __fsqrt_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)));
    const float den = vdr < 1.0e-6f ? 1.0e-6f : vdr;
    const float rel = __fdiv_rn(fabsf(__fsub_rn(vds, vdr)), den);
    return (err < F.max_reproj_px && rel < F.max_rel_vd) ? si : -1;
}

// One CTA per micro-image: pair_si[(v, idx)][j] of its list entries, and the mask of
// the pixels that can become points (a valid depth and enough consistent entries).
__global__ void __launch_bounds__(256) pm_fuse_pairs_kernel(FuseFrame F, FuseWork X)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int b = blockIdx.x, v = X.v0 + b;
    if (!X.is_ref[v]) return;
    const int m = F.m, N = F.ppv;
    const int nl = min(F.list_counts[v], F.max_list);
    int* ids = (int*)smem;                               // [max_list]
    float2* cen = (float2*)(ids + ((F.max_list + 1) & ~1));
    for (int j = threadIdx.x; j < nl; j += blockDim.x) {
        const int u = F.lists[(size_t)v * F.max_list + j];
        ids[j] = u;
        cen[j] = u >= 0 ? F.centers[u] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const float cm = __fadd_rn(__fmul_rn((float)(m - 1), 0.5f), 1.0f);
    const float2 cr = F.centers[v];
    const int n32 = (N + 31) & ~31;
    for (int idx = threadIdx.x; idx < n32; idx += blockDim.x) {
        int num = -1;
        if (idx < N) {
            const float w = F.plane[(size_t)v * N + idx].w;
            const float vdr = virtual_depth(F.mla_base, w);
            const bool own = !(w < F.min_ref_disp) && valid_vd(vdr);
            const int r = idx / m, c = idx - r * m;
            const float3 P = virtual_3d(vdr, c, r, cm, cr);
            uint16_t* row = X.pair_si + ((size_t)b * N + idx) * F.max_list;
            if (own) num = 0;
            for (int j = 0; j < nl; ++j) {
                int si = -1;
                if (own && ids[j] >= 0) si = consistent_pixel(F, P, vdr, r, c, cr, ids[j], cen[j], cm);
                row[j] = si >= 0 ? (uint16_t)si : kFuseNone;
                num += si >= 0;
            }
        }
        const unsigned bits = __ballot_sync(kFull, num >= 0 && num >= F.min_consistent);
        if ((threadIdx.x & 31) == 0) X.maybe[(size_t)b * X.mask_words + (idx >> 5)] = bits;
    }
}

// Who masks pixels of a micro-image: the band's (reference micro-image, list entry)
// pairs that name it, as lists in X.rev.
__global__ void pm_fuse_rev_count_kernel(FuseFrame F, FuseWork X)
{
    const size_t n = (size_t)(X.v1 - X.v0) * F.max_list, e0 = (size_t)X.v0 * F.max_list;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(e / F.max_list), w = X.v0 + b, j = (int)(e - (size_t)b * F.max_list);
        if (!X.is_ref[w] || j >= F.list_counts[w]) continue;
        const int u = F.lists[e0 + e];
        if (u >= 0) atomicAdd(X.rev_start + u + 1, 1);
    }
}

__global__ void __launch_bounds__(1024) pm_fuse_rev_scan_kernel(FuseFrame F, FuseWork X)
{
    __shared__ int warp_sum[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < F.V; b += 1024) {
        const int i = b + threadIdx.x;
        int x = i < F.V ? X.rev_start[i + 1] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += t;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int s = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(kFull, s, o);
                if (lane >= o) s += t;
            }
            warp_sum[lane] = s;
        }
        __syncthreads();
        const int base = carry + (warp ? warp_sum[warp - 1] : 0);
        if (i < F.V) { X.rev_start[i + 1] = base + x; X.rev_fill[i + 1] = base + x; }
        __syncthreads();
        if (threadIdx.x == 1023) carry = base + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) { X.rev_start[0] = 0; X.rev_fill[0] = 0; }
}

__global__ void pm_fuse_rev_fill_kernel(FuseFrame F, FuseWork X)
{
    const size_t n = (size_t)(X.v1 - X.v0) * F.max_list, e0 = (size_t)X.v0 * F.max_list;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(e / F.max_list), w = X.v0 + b, j = (int)(e - (size_t)b * F.max_list);
        if (!X.is_ref[w] || j >= F.list_counts[w]) continue;
        const int u = F.lists[e0 + e];
        if (u >= 0) X.rev[atomicAdd(X.rev_fill + u, 1)] = make_int2(w, j);
    }
}

namespace {

// One micro-image's walk by one warp.  taken: [1 + nl][mw] masks of the micro-image
// itself and of its list entries (entries naming the same micro-image share the
// first one's), fresh: [nl][mw] what this walk masks.  Publishes the difference.
// LATER: the band is not the frame's first (a kernel of its own, since the places in the
// band cost the registers that keep the first band's walk from spilling, 2% of it).
template <bool LATER>
__device__ __forceinline__ void walk_view(const FuseFrame& F, const FuseWork& X, int v, uint32_t* taken, uint32_t* fresh,
                                          int* changed_at)
{
    const int v0 = LATER ? X.v0 : 0;
    const size_t vb = (size_t)(v - v0);                  // place in the band
    const int lane = threadIdx.x & 31, N = F.ppv, mw = X.mask_words;
    const int nl = min(F.list_counts[v], F.max_list);
    const int nch = (nl + 31) >> 5;
    const int* list = F.lists + (size_t)v * F.max_list;
    for (int e = lane; e < (1 + nl) * mw; e += 32) taken[e] = 0u;
    for (int e = lane; e < nl * mw; e += 32) fresh[e] = 0u;
    const uint16_t* rows = X.pair_si + vb * N * F.max_list;
    for (int b = lane * 128; b < N * F.max_list * 2; b += 32 * 128)
        asm volatile("prefetch.global.L1 [%0];" :: "l"((const char*)rows + b));
    // slot of each list entry: 0 for the micro-image itself, else 1 + the first entry
    // that names it
    int uj[kFuseMaxList / 32], slot[kFuseMaxList / 32];
#pragma unroll
    for (int ch = 0; ch < kFuseMaxList / 32; ++ch) {
        uj[ch] = -1;
        slot[ch] = 0;
        const int j = ch * 32 + lane;
        if (ch < nch && j < nl) {
            uj[ch] = list[j];
            slot[ch] = 1 + j;
            if (uj[ch] == v) slot[ch] = 0;
            else
                for (int i = 0; i < j; ++i)
                    if (list[i] == uj[ch]) { slot[ch] = 1 + i; break; }
        }
    }
    __syncwarp();
    // the masks that the micro-images before this one leave
    for (int t = 0; t <= nl; ++t) {
        int u = v;
        if (t) {
            const int ch = (t - 1) >> 5, src = (t - 1) & 31;
            int a = -1, b = 0;
#pragma unroll
            for (int c = 0; c < kFuseMaxList / 32; ++c)
                if (c == ch) { a = uj[c]; b = slot[c]; }
            u = __shfl_sync(kFull, a, src);
            if (u < 0 || __shfl_sync(kFull, b, src) != t) continue;
        }
        if (LATER)
            for (int word = lane; word < mw; word += 32) {
                const uint32_t bits = X.base[(size_t)u * mw + word];
                if (bits) atomicOr(taken + t * mw + word, bits);
            }
        const int r0 = X.rev_start[u], r1 = X.rev_start[u + 1];
        for (int e = r0 * mw + lane; e < r1 * mw; e += 32) {
            const int2 wj = X.rev[e / mw];
            if (wj.x >= v) continue;
            const int word = e % mw;
            const uint32_t bits = __ldcg(X.marks + ((size_t)(wj.x - v0) * F.max_list + wj.y) * mw + word);
            if (bits) atomicOr(taken + t * mw + word, bits);
        }
    }
    __syncwarp();
    const uint32_t* maybe = X.maybe + vb * mw;
    for (int wd = 0; wd < mw; ++wd) {
        uint32_t todo = maybe[wd], accepted = 0u;
        while (todo) {
            const int b = __ffs(todo) - 1, idx = wd * 32 + b;
            todo &= todo - 1;
            if ((taken[wd] >> b) & 1u) continue;         // used by an earlier point
            int si[kFuseMaxList / 32];
            uint32_t bits[kFuseMaxList / 32];
            int num = 0;
#pragma unroll
            for (int ch = 0; ch < kFuseMaxList / 32; ++ch) {
                bits[ch] = 0u;
                if (ch >= nch) continue;
                const int j = ch * 32 + lane;
                si[ch] = j < nl ? rows[(size_t)idx * F.max_list + j] : kFuseNone;
                const bool ok = si[ch] != kFuseNone && !((taken[slot[ch] * mw + (si[ch] >> 5)] >> (si[ch] & 31)) & 1u);
                bits[ch] = __ballot_sync(kFull, ok);
                num += __popc(bits[ch]);
            }
            if (num < F.min_consistent) continue;
            accepted |= 1u << b;
            __syncwarp();
#pragma unroll
            for (int ch = 0; ch < kFuseMaxList / 32; ++ch) {
                if (ch >= nch) continue;
                if ((bits[ch] >> lane) & 1u) {
                    atomicOr(taken + slot[ch] * mw + (si[ch] >> 5), 1u << (si[ch] & 31));
                    atomicOr(fresh + (ch * 32 + lane) * mw + (si[ch] >> 5), 1u << (si[ch] & 31));
                }
                if (lane == 0) X.chosen[(vb * N + idx) * X.chosen_words + ch] = bits[ch];
            }
            __syncwarp();
        }
        if (lane == 0) X.accepted[vb * mw + wd] = accepted;
    }
    __syncwarp();
    for (int e = lane; e < nl * mw; e += 32) {
        uint32_t* g = X.marks + vb * F.max_list * mw + e;
        if (__ldcg(g) != fresh[e]) {
            __stcg(g, fresh[e]);
            atomicMin(changed_at + list[e / mw], v);
        }
    }
    __syncwarp();
}

}  // namespace

template <bool LATER>
__global__ void __launch_bounds__(256) pm_fuse_resolve_kernel(FuseFrame F, FuseWork X, int* err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, mw = X.mask_words;
    uint32_t* taken = (uint32_t*)smem + (size_t)warp * (1 + 2 * F.max_list) * mw;
    uint32_t* fresh = taken + (1 + F.max_list) * mw;
    unsigned int arrived = 0;
    // X.ctl: 0 barrier; 1, 2, 3 list lengths of rounds 1, 2, 3 mod 3.  X.changed + (round
    // mod 3) V: the first micro-image that changed what it masks in each, per round.
    for (int round = 1; round <= F.V + 2; ++round) {
        if (blockIdx.x == 0 && threadIdx.x == 0) X.ctl[1 + (round + 1) % 3] = 0u;
        const int* last = X.changed + (size_t)((round + 2) % 3) * F.V;
        int* next = X.changed + (size_t)((round + 1) % 3) * F.V;
        for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < F.V; v += gridDim.x * blockDim.x) {
            __stcg(next + v, 0x7fffffff);
            if (v < X.v0 || v >= X.v1 || !X.is_ref[v]) continue;
            bool dirty = round == 1;
            if (!dirty) {
                dirty = __ldcg(last + v) < v;
                const int nl = min(F.list_counts[v], F.max_list);
                for (int j = 0; j < nl && !dirty; ++j) {
                    const int u = F.lists[(size_t)v * F.max_list + j];
                    dirty = u >= 0 && __ldcg(last + u) < v;
                }
            }
            if (dirty) X.list[atomicAdd(X.ctl + 1 + round % 3, 1u)] = v;
        }
        if (!grid_barrier(X.ctl, ++arrived * gridDim.x, err)) return;
        const int n_list = (int)__ldcg(X.ctl + 1 + round % 3);
        if (n_list == 0) return;
        for (int i = blockIdx.x * warps + warp; i < n_list; i += gridDim.x * warps)
            walk_view<LATER>(F, X, __ldcg(X.list + i), taken, fresh, X.changed + (size_t)(round % 3) * F.V);
        if (!grid_barrier(X.ctl, ++arrived * gridDim.x, err)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, PFD_DEVERR_TMA_TIMEOUT);       // map order has no cycles: not reached
}

__global__ void __launch_bounds__(256) pm_fuse_points_kernel(FuseFrame F, FuseWork X)
{
    const size_t n = (size_t)(X.v1 - X.v0) * F.ppv, first = (size_t)X.v0 * F.ppv;
    const int m = F.m;
    const float cm = __fadd_rn(__fmul_rn((float)(m - 1), 0.5f), 1.0f);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        const size_t seq = first + q;
        const int b = (int)(q / F.ppv), v = X.v0 + b, idx = (int)(q - (size_t)b * F.ppv);
        if (!X.is_ref[v] || !((X.accepted[(size_t)b * X.mask_words + (idx >> 5)] >> (idx & 31)) & 1u)) continue;
        const float4 pl = F.plane[seq];
        const float vdr = virtual_depth(F.mla_base, pl.w);
        const int r = idx / m, c = idx - r * m;
        float3 sp = virtual_3d(vdr, c, r, cm, F.centers[v]);
        float3 sn = make_float3(pl.x, pl.y, pl.z), sc = colour(F, v, idx);
        int num = 0;
        const int nch = (min(F.list_counts[v], F.max_list) + 31) >> 5;
        for (int ch = 0; ch < nch; ++ch) {
            uint32_t bits = X.chosen[q * X.chosen_words + ch];
            num += __popc(bits);
            while (bits) {
                const int j = ch * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                const int u = F.lists[(size_t)v * F.max_list + j], si = X.pair_si[q * F.max_list + j];
                const float4 ps = F.plane[(size_t)u * F.ppv + si];
                const int sr = si / m, scol = si - sr * m;
                const float3 Ps = virtual_3d(virtual_depth(F.mla_base, ps.w), scol, sr, cm, F.centers[u]);
                const float3 Cs = colour(F, u, si);
                sp.x = __fadd_rn(sp.x, Ps.x); sp.y = __fadd_rn(sp.y, Ps.y); sp.z = __fadd_rn(sp.z, Ps.z);
                sn.x = __fadd_rn(sn.x, ps.x); sn.y = __fadd_rn(sn.y, ps.y); sn.z = __fadd_rn(sn.z, ps.z);
                sc.x = __fadd_rn(sc.x, Cs.x); sc.y = __fadd_rn(sc.y, Cs.y); sc.z = __fadd_rn(sc.z, Cs.z);
            }
        }
        // cv::Vec3f /= float multiplies by the float reciprocal
        const float ia = __fdiv_rn(1.0f, __fadd_rn((float)num, 1.0f));
        sp = make_float3(__fmul_rn(sp.x, ia), __fmul_rn(sp.y, ia), __fmul_rn(sp.z, ia));
        sn = make_float3(__fmul_rn(sn.x, ia), __fmul_rn(sn.y, ia), __fmul_rn(sn.z, ia));
        sc = make_float3(__fmul_rn(sc.x, ia), __fmul_rn(sc.y, ia), __fmul_rn(sc.z, ia));
        const int vx = round_x86(sp.x), vy = round_x86(sp.y);
        if (vy >= 0 && vy < F.raw_h && vx >= 0 && vx < F.raw_w) {
            float* rec = F.rec + seq * 10;
            rec[0] = sp.x; rec[1] = sp.y; rec[2] = sp.z;
            rec[3] = sn.x; rec[4] = sn.y; rec[5] = sn.z;
            rec[6] = sc.x; rec[7] = sc.y; rec[8] = sc.z;
            rec[9] = (float)num;
            F.has_rec[seq] = 1u;
            atomicMax(&F.winner[(size_t)vy * F.raw_w + vx], (unsigned int)seq + 1u);
        }
    }
}

__global__ void pm_fuse_maps_kernel(FuseFrame F, float* __restrict__ vd_map, uint8_t* __restrict__ conf,
                                    uint8_t* __restrict__ aif)
{
    const size_t n = (size_t)F.raw_w * F.raw_h;
    for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x) {
        const unsigned s = F.winner[o];
        float z = 0.0f;
        uint8_t cf = 0, b = 0, g = 0, rr = 0;
        if (s) {
            const float* rec = F.rec + (size_t)(s - 1u) * 10;
            z = rec[2];
            const int k = ((int)rec[9] + 1) * 60;
            cf = (uint8_t)(k < 255 ? k : 255);
            b = sat_u8(rec[6]);
            g = sat_u8(rec[7]);
            rr = sat_u8(rec[8]);
        }
        vd_map[o] = z;
        conf[o] = cf;
        aif[3 * o + 0] = b;
        aif[3 * o + 1] = g;
        aif[3 * o + 2] = rr;
    }
}

__global__ void __launch_bounds__(kFuseScanBlock) pm_fuse_count_kernel(FuseFrame F, unsigned int* block_counts)
{
    const size_t n = (size_t)F.V * F.ppv;
    const size_t s = (size_t)blockIdx.x * kFuseScanBlock + threadIdx.x;
    const unsigned f = (s < n) ? F.has_rec[s] : 0u;
    const unsigned c = __syncthreads_count(f != 0u);
    if (threadIdx.x == 0) block_counts[blockIdx.x] = c;
}

__global__ void __launch_bounds__(kFuseScanBlock) pm_fuse_compact_kernel(FuseFrame F, const unsigned int* block_offsets,
                                                                          float* points)
{
    __shared__ unsigned warp_base[kFuseScanBlock / 32];
    const size_t n = (size_t)F.V * F.ppv;
    const size_t s = (size_t)blockIdx.x * kFuseScanBlock + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool f = (s < n) && F.has_rec[s] != 0u;
    const unsigned bits = __ballot_sync(kFull, f);
    if (lane == 0) warp_base[w] = __popc(bits);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned acc = 0;
        for (int i = 0; i < kFuseScanBlock / 32; ++i) { const unsigned t = warp_base[i]; warp_base[i] = acc; acc += t; }
    }
    __syncthreads();
    if (f) {
        const size_t o = (size_t)block_offsets[blockIdx.x] + warp_base[w] + __popc(bits & ((1u << lane) - 1u));
        const float* rec = F.rec + s * 10;
        for (int i = 0; i < 9; ++i) points[o * 9 + i] = rec[i];
    }
}

// What the band's micro-images mask, for the bands after it.
__global__ void __launch_bounds__(256) pm_fuse_fold_kernel(FuseFrame F, FuseWork X)
{
    const int mw = X.mask_words;
    const size_t n = (size_t)(X.v1 - X.v0) * F.max_list * mw;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t bits = X.marks[i];
        if (!bits) continue;
        const size_t e = i / mw;
        atomicOr(X.base + (size_t)F.lists[(size_t)X.v0 * F.max_list + e] * mw + (i - e * mw), bits);
    }
}

size_t fuse_work(const FuseFrame& F, int n, unsigned char* buf, FuseWork& X)
{
    size_t o = 0;
    auto take = [&](size_t bytes) { const size_t at = o; o += (bytes + 255) & ~(size_t)255; return buf + at; };
    const size_t V = (size_t)F.V, B = (size_t)n, px = B * F.ppv, L = (size_t)F.max_list;
    X.mask_words = (F.ppv + 31) / 32;
    X.chosen_words = (F.max_list + 31) / 32;
    X.zeroed = buf;
    X.ctl = (unsigned int*)take(16);
    X.rev_start = (int*)take(sizeof(int) * (V + 1));
    X.marks = (uint32_t*)take(sizeof(uint32_t) * B * L * X.mask_words);
    X.zeroed_bytes = o;
    X.changed = (int*)take(sizeof(int) * 3 * V);
    X.rev_fill = (int*)take(sizeof(int) * (V + 1));
    X.base = (uint32_t*)take(sizeof(uint32_t) * V * X.mask_words);
    X.rev = (int2*)take(sizeof(int2) * B * L);
    X.list = (int*)take(sizeof(int) * B);
    X.maybe = (uint32_t*)take(sizeof(uint32_t) * B * X.mask_words);
    X.accepted = (uint32_t*)take(sizeof(uint32_t) * B * X.mask_words);
    X.chosen = (uint32_t*)take(sizeof(uint32_t) * px * X.chosen_words);
    X.pair_si = (uint16_t*)take(sizeof(uint16_t) * px * L);
    return o;
}

int fuse_band(const FuseFrame& F, size_t limit)
{
    FuseWork X;
    const size_t all = fuse_work(F, F.V, nullptr, X), fixed = fuse_work(F, 0, nullptr, X);
    if (all <= limit) return F.V;
    const size_t per = (all - fixed + F.V - 1) / F.V;
    const int most = limit > fixed ? (int)std::min<size_t>(std::max<size_t>((limit - fixed) / per, 1), F.V) : 1;
    const int bands = (F.V + most - 1) / most;
    return (F.V + bands - 1) / bands;                    // equal bands
}

cudaError_t launch_fuse(const FuseFrame& F, FuseWork X, int band, int* err, cudaStream_t st, unsigned long long* launches)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t per_warp = (size_t)(1 + 2 * F.max_list) * X.mask_words * 4;
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)96 * 1024 / per_warp));
    const int smem = (int)(per_warp * warps);
    cudaError_t e = cudaSuccess;
    if (band < F.V) e = cudaMemsetAsync(X.base, 0, sizeof(uint32_t) * (size_t)F.V * X.mask_words, st);
    for (X.v0 = 0; e == cudaSuccess && X.v0 < F.V; X.v0 = X.v1) {
        X.v1 = std::min(F.V, X.v0 + band);
        const int n = X.v1 - X.v0;
        e = cudaMemsetAsync(X.zeroed, 0, X.zeroed_bytes, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(X.changed, 0x7f, sizeof(int) * 3 * (size_t)F.V, st);
        if (e != cudaSuccess) return e;
        const auto resolve = X.v0 ? pm_fuse_resolve_kernel<true> : pm_fuse_resolve_kernel<false>;
        e = allow_dynamic_smem((const void*)resolve, smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, resolve, 32 * warps, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
        const int flat = (int)std::min<size_t>(((size_t)n * F.max_list + 255) / 256, (size_t)sms * 8);
        pm_fuse_pairs_kernel<<<n, std::min(256, (F.ppv + 31) & ~31), (F.max_list + 1) * 12 + 16, st>>>(F, X);
        pm_fuse_rev_count_kernel<<<flat, 256, 0, st>>>(F, X);
        pm_fuse_rev_scan_kernel<<<1, 1024, 0, st>>>(F, X);
        pm_fuse_rev_fill_kernel<<<flat, 256, 0, st>>>(F, X);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)std::max(1, std::min((n + warps - 1) / warps, sms * std::min(per_sm, 4))));
        lc.blockDim = dim3((unsigned)(32 * warps));
        lc.dynamicSmemBytes = (size_t)smem;
        lc.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        lc.attrs = at;
        lc.numAttrs = 1;
        if ((e = cudaLaunchKernelEx(&lc, resolve, F, X, err)) != cudaSuccess) return e;
        const size_t px = (size_t)n * F.ppv;
        pm_fuse_points_kernel<<<(int)std::min<size_t>((px + 255) / 256, (size_t)sms * 16), 256, 0, st>>>(F, X);
        *launches += 6;
        if (X.v1 < F.V) {
            pm_fuse_fold_kernel<<<flat, 256, 0, st>>>(F, X);
            *launches += 1;
        }
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_fuse_maps(const FuseFrame& F, float* vd_map, uint8_t* conf, uint8_t* aif, cudaStream_t st)
{
    const size_t n = (size_t)F.raw_w * F.raw_h;
    const int grid = (int)((n + 255) / 256 < (size_t)148 * 16 ? (n + 255) / 256 : (size_t)148 * 16);
    pm_fuse_maps_kernel<<<grid > 0 ? grid : 1, 256, 0, st>>>(F, vd_map, conf, aif);
    return cudaGetLastError();
}

cudaError_t launch_fuse_count(const FuseFrame& F, unsigned int* block_counts, cudaStream_t st)
{
    const size_t n = (size_t)F.V * F.ppv;
    const int nb = (int)((n + kFuseScanBlock - 1) / kFuseScanBlock);
    pm_fuse_count_kernel<<<nb, kFuseScanBlock, 0, st>>>(F, block_counts);
    return cudaGetLastError();
}

cudaError_t launch_fuse_compact(const FuseFrame& F, const unsigned int* block_offsets, float* points, cudaStream_t st)
{
    const size_t n = (size_t)F.V * F.ppv;
    const int nb = (int)((n + kFuseScanBlock - 1) / kFuseScanBlock);
    pm_fuse_compact_kernel<<<nb, kFuseScanBlock, 0, st>>>(F, block_offsets, points);
    return cudaGetLastError();
}

}  // namespace pfd
