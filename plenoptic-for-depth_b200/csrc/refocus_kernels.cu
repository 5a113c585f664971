// refocus_kernels.cu -- focal-stack render on the device.
//
// The reference has no multi-slice render; this one is defined from its
// back-projection LFRefocus::BackProject2MI (FocalStack/LFRefocus.cpp:2119-2125):
// output pixel (ox, oy) of slice s lies at raw coordinates
// X = (ox + 0.5) * (W / out_w) - 0.5, and micro-image i sees it at
// u = (X - c_i) / vd_s + ((m-1)/2 + 1)  (the centre of FuseVirtualDepth_BackProject,
// :1635-1636).  Every micro-image whose u falls in [0, m-1]^2 contributes its
// bilinear gray sample; the output is the mean, summed in ascending view index.
//
// One CTA renders a 64 x 16 output tile of one slice.  The lenses that can reach
// the tile are gathered from a bucket grid of lens centres and sorted by view
// index (so the sum order is the oracle's).  A warp owns 32 columns x 8 rows, one
// column per lane: it takes the lenses that can reach its own pixels, works out
// the row coordinates of 4 lenses x 8 rows side by side on its lanes and the column
// coordinate once per lens, and reads a sample's four texels as one packed word
// (pm_refocus_quads_kernel lays the micro-images out so, 4 bytes per texel).
//
// Bound by instruction issue, about 20 instructions per sample and lane; texels
// become floats by their position in the mantissa of 2^23 and indices by a
// round-down addition of 2^23, because conversions run at an eighth of the rate.
// 16 slices of 2040x1534 from the 4080x3068 frame: 2.62 ms, against 5.19 ms with one
// conversion per texel, two rows x two columns per lane and staged 8-bit tiles.
#include <cstdint>
#include <cuda_runtime.h>
#include "refocus_kernels.h"

namespace pfd {

namespace {

// A warp's 32 x 8 pixels: 2.62 ms for the 16 slices above, 32 x 4 2.65, 16 x 16 2.83
// (rows no lens reaches are skipped by the whole warp only where a row is a warp's);
// all rows' texels loaded before their blends 2.96.
constexpr int kTileW = 64, kTileH = 16, kWarpRows = 8;
constexpr int kThreads = (kTileW / 32) * (kTileH / kWarpRows) * 32;
constexpr int kLensStep = 32 / kWarpRows;       // lenses whose rows a warp works out side by side
constexpr float kBig = 8388608.0f;       // 2^23

// a / v, correctly rounded, with y = 1 / v correctly rounded: two corrections of
// a * y (Markstein); for |a| 0 or normal and v within [2^-60, 2^60].
__device__ __forceinline__ float div_by(float a, float v, float y)
{
    float q = __fmul_rn(a, y);
    q = __fmaf_rn(__fmaf_rn(-q, v, a), y, q);
    return __fmaf_rn(__fmaf_rn(-q, v, a), y, q);
}

// Byte b of q as 2^23 + value.
template <int B>
__device__ __forceinline__ float big_byte(uint32_t q)
{
    return __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7650 + B));
}

}  // namespace

// quads[v][y][x] = T(y, x), T(y, x1), T(y1, x), T(y1, x1), x1 = min(x + 1, m - 1), y1 likewise.
__global__ void __launch_bounds__(256) pm_refocus_quads_kernel(const uint8_t* __restrict__ gray, int tile_stride, int m,
                                                               int mh, int V, uint32_t* __restrict__ quads)
{
    const int N = m * mh;
    const size_t total = (size_t)V * N;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int v = (int)(t / N), e = (int)(t - (size_t)v * N);
        const int y = e / m, x = e - y * m;
        const int x1 = min(x + 1, m - 1), y1 = min(y + 1, mh - 1);
        const uint8_t* T = gray + (size_t)v * tile_stride;
        quads[t] = (uint32_t)T[y * m + x] | ((uint32_t)T[y * m + x1] << 8) | ((uint32_t)T[y1 * m + x] << 16) |
                   ((uint32_t)T[y1 * m + x1] << 24);
    }
}

__global__ void __launch_bounds__(kThreads) pm_refocus_kernel(RefocusFrame F, const uint32_t* __restrict__ quads,
                                                              const float* slice_vd, int out_w, int out_h, float sx,
                                                              float sy, float* out, int* err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float2* sc = (float2*)smem;                              // [kMaxRefocusCand] centres, ascending view
    int* sid = (int*)(sc + kMaxRefocusCand);                 // [kMaxRefocusCand] views
    int* cand = sid + kMaxRefocusCand;                       // [kMaxRefocusCand] gathered
    __shared__ int n_cand;
    __shared__ uint8_t s_hits[kThreads / 32][32];

    const int s = blockIdx.z;
    const float v = slice_vd[s];
    const int ox0 = blockIdx.x * kTileW, oy0 = blockIdx.y * kTileH;
    const int m = F.m, mh = F.mh;
    const float cmx = (float)(m - 1) * 0.5f + 1.0f, cmy = (float)(mh - 1) * 0.5f + 1.0f;
    const float umax = (float)(m - 1), wmax = (float)(mh - 1);

    // ---- lenses that can reach the tile ------------------------------------
    const int ex = min(ox0 + kTileW, out_w) - 1, ey = min(oy0 + kTileH, out_h) - 1;
    const float X0 = ((float)ox0 + 0.5f) * sx - 0.5f, X1 = ((float)ex + 0.5f) * sx - 0.5f;
    const float Y0 = ((float)oy0 + 0.5f) * sy - 0.5f, Y1 = ((float)ey + 0.5f) * sy - 0.5f;
    const float bx0 = X0 - (umax - cmx) * v - 1.0f, bx1 = X1 + cmx * v + 1.0f;
    const float by0 = Y0 - (wmax - cmy) * v - 1.0f, by1 = Y1 + cmy * v + 1.0f;
    const float inv_cell = 1.0f / F.cell;
    const int gx0 = max(0, (int)floorf((bx0 - F.grid_x0) * inv_cell));
    const int gx1 = min(F.grid_w - 1, (int)floorf((bx1 - F.grid_x0) * inv_cell));
    const int gy0 = max(0, (int)floorf((by0 - F.grid_y0) * inv_cell));
    const int gy1 = min(F.grid_h - 1, (int)floorf((by1 - F.grid_y0) * inv_cell));
    if (threadIdx.x == 0) n_cand = 0;
    __syncthreads();
    if (gx1 >= gx0 && gy1 >= gy0) {
        const int gw = gx1 - gx0 + 1, ncell = gw * (gy1 - gy0 + 1);
        for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
            const int cell = (gy0 + c / gw) * F.grid_w + gx0 + c % gw;
            for (int k = F.cell_start[cell]; k < F.cell_start[cell + 1]; ++k) {
                const int id = F.cell_ids[k];
                const float2 p = F.centers[id];
                if (p.x < bx0 || p.x > bx1 || p.y < by0 || p.y > by1) continue;
                const int slot = atomicAdd(&n_cand, 1);
                if (slot < kMaxRefocusCand) cand[slot] = id;
            }
        }
    }
    __syncthreads();
    int n = n_cand;
    if (n > kMaxRefocusCand) {
        if (threadIdx.x == 0) atomicOr(err, PFD_DEVERR_REFOCUS_LENSES);
        n = kMaxRefocusCand;
    }
    // rank sort: ids are distinct
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int id = cand[i];
        int r = 0;
        for (int j = 0; j < n; ++j) r += cand[j] < id;
        sid[r] = id;
        sc[r] = F.centers[id];
    }
    __syncthreads();

    // ---- accumulate ----------------------------------------------------------
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ox = ox0 + (warp & 1) * 32 + lane, oyw = oy0 + (warp >> 1) * kWarpRows;
    const float X = ((float)ox + 0.5f) * sx - 0.5f;
    const float Yr = ((float)(oyw + lane % kWarpRows) + 0.5f) * sy - 0.5f;       // row of this lane's (lens, row) pair
    // box of the centres that can reach the warp's pixels; the slack covers the rounding
    // of the coordinates u and w
    const float slack = 1.0f + 1e-5f * v * (float)max(m, mh);
    const float wx0 = ((float)(ox0 + (warp & 1) * 32) + 0.5f) * sx - 0.5f - (umax - cmx) * v - slack;
    const float wx1 = ((float)(ox0 + (warp & 1) * 32 + 31) + 0.5f) * sx - 0.5f + cmx * v + slack;
    const float wy0 = ((float)oyw + 0.5f) * sy - 0.5f - (wmax - cmy) * v - slack;
    const float wy1 = ((float)(oyw + kWarpRows - 1) + 0.5f) * sy - 0.5f + cmy * v + slack;
    const bool fast = v >= 0x1p-60f && v <= 0x1p60f;
    const float y = __fdiv_rn(1.0f, v);
    float sum[kWarpRows];
    int cnt[kWarpRows];
#pragma unroll
    for (int r = 0; r < kWarpRows; ++r) { sum[r] = 0.0f; cnt[r] = 0; }
    uint8_t* hits = s_hits[warp];
    const int row_bytes = m * 4;
    const size_t N = (size_t)m * mh;
    for (int base = 0; base < n; base += 32) {
        const int k = base + lane;
        const float2 c = k < n ? sc[k] : make_float2(0.f, 0.f);
        const int id = k < n ? sid[k] : 0;
        const bool near = k < n && !(c.x < wx0 || c.x > wx1 || c.y < wy0 || c.y > wy1);
        const unsigned hm = __ballot_sync(0xffffffffu, near);
        const int nh = __popc(hm);
        if (near) hits[__popc(hm & ((1u << lane) - 1u))] = (uint8_t)lane;
        __syncwarp();
        for (int j0 = 0; j0 < nh; j0 += kLensStep) {
            // lane = (lens j0 + lane / rows, row lane % rows): the row's texel row (byte
            // offset, -1 outside) and fraction
            const int jl = j0 + lane / kWarpRows;
            const int src = hits[jl < nh ? jl : 0];
            const float cy = __shfl_sync(0xffffffffu, c.y, src);
            const float ny = __fsub_rn(Yr, cy);
            const float w = __fadd_rn(fast ? div_by(ny, v, y) : __fdiv_rn(ny, v), cmy);
            int yoff = -1;
            float ay = 0.0f;
            if (w >= 0.0f && w <= wmax) {
                const float t = __fadd_rd(w, kBig);
                yoff = (__float_as_int(t) - 0x4B000000) * row_bytes;
                ay = __fsub_rn(w, __fsub_rn(t, kBig));
            }
            const int nj = min(kLensStep, nh - j0);
            for (int l = 0; l < nj; ++l) {
                const int sl = hits[j0 + l];
                const float cx = __shfl_sync(0xffffffffu, c.x, sl);
                const int view = __shfl_sync(0xffffffffu, id, sl);
                const float nx = __fsub_rn(X, cx);
                const float u = __fadd_rn(fast ? div_by(nx, v, y) : __fdiv_rn(nx, v), cmx);
                const bool in = u >= 0.0f && u <= umax;
                const float t = __fadd_rd(u, kBig);
                const float ax = __fsub_rn(u, __fsub_rn(t, kBig));
                const char* tile = (const char*)(quads + (size_t)view * N) + (__float_as_int(t) - 0x4B000000) * 4;
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r) {
                    const int yo = __shfl_sync(0xffffffffu, yoff, l * kWarpRows + r);
                    const float fy = __shfl_sync(0xffffffffu, ay, l * kWarpRows + r);
                    if (yo < 0 || !in) continue;
                    const uint32_t q = __ldg((const uint32_t*)(tile + yo));
                    const float f00 = big_byte<0>(q), f01 = big_byte<1>(q), f10 = big_byte<2>(q), f11 = big_byte<3>(q);
                    const float top = __fmaf_rn(ax, __fsub_rn(f01, f00), __fsub_rn(f00, kBig));
                    const float bot = __fmaf_rn(ax, __fsub_rn(f11, f10), __fsub_rn(f10, kBig));
                    sum[r] = __fadd_rn(sum[r], __fmaf_rn(fy, __fsub_rn(bot, top), top));
                    cnt[r] += 1;
                }
            }
        }
        __syncwarp();
    }
    if (ox >= out_w) return;
    float* o = out + (size_t)s * out_h * out_w + ox;
#pragma unroll
    for (int r = 0; r < kWarpRows; ++r) {
        const int oy = oyw + r;
        if (oy < out_h) o[(size_t)oy * out_w] = cnt[r] ? __fdiv_rn(sum[r], (float)cnt[r]) : 0.0f;
    }
}

cudaError_t launch_refocus_quads(const RefocusFrame& F, uint32_t* quads, cudaStream_t st)
{
    const size_t px = (size_t)F.V * F.m * F.mh;
    pm_refocus_quads_kernel<<<(unsigned)((px + 1023) / 1024), 256, 0, st>>>(F.gray, F.tile_stride, F.m, F.mh, F.V, quads);
    return cudaGetLastError();
}

cudaError_t launch_refocus(const RefocusFrame& F, const uint32_t* quads, const float* slice_vd, int n_slices, int raw_w,
                           int raw_h, int out_w, int out_h, float* out, int* err, cudaStream_t st)
{
    if (n_slices <= 0) return cudaSuccess;
    const int smem = kMaxRefocusCand * 16;
    const float sx = (float)raw_w / (float)out_w, sy = (float)raw_h / (float)out_h;
    const dim3 grid((out_w + kTileW - 1) / kTileW, (out_h + kTileH - 1) / kTileH, n_slices);
    pm_refocus_kernel<<<grid, kThreads, smem, st>>>(F, quads, slice_vd, out_w, out_h, sx, sy, out, err);
    return cudaGetLastError();
}

}  // namespace pfd
