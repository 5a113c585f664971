// check_kernels.cu -- the consistency pass after PatchMatch, on the device:
//   pm_filter_kernel   MIDisparityFilterCPU::FilterTile (CheckModule/MIDisparityFilter.cpp:423-693)
//   pm_reproj_kernel   ComputeTileReprojectionErrorMap (MIDisparityFilter.cpp:695-842)
//   pm_cycle_kernel    MICycleCheckerCPU::CheckTile (CheckModule/MICycleCheck.cpp:282-725)
//
// The filter invalidates rejected pixels in place and walks the micro-images
// in key order, so a later micro-image reads the already filtered state of
// earlier neighbours (FilterGlobal, :962-986).  The device keeps exactly that
// dependency, in three launches:
//   pm_filter_pairs_kernel    every (pixel, view) test on the unfiltered state.
//                             What an earlier neighbour's filtering can change is
//                             only whether one of the four pixels a test reads has
//                             been rejected (then the view gives no support), so a
//                             test against an earlier neighbour is kept as (view,
//                             pixel, passed) and one against a later neighbour is
//                             final.
//   pm_filter_resolve_kernel  the rejected pixels of every micro-image as a bit
//                             mask, from its earlier neighbours' masks, repeated
//                             for the micro-images whose earlier neighbours changed
//                             until nothing changes: key order has no cycles, so
//                             this ends at the one solution, the sequential walk's.
//                             A cooperative launch; the grid barrier's waits are
//                             bounded.
//   pm_filter_apply_kernel    reasons, counters and the rejected pixels' state; nothing
//                             when the masks did not settle (a wait gave up), so that a
//                             reported timeout leaves the state as it was.
// A rejected pixel gets disparity -1; where the configuration accepts such a
// disparity (min_valid_disp < -1) it is not an unusable one, and the filter runs as
// a wavefront instead (pm_filter_kernel): micro-image (col, row) in step
// col + c * row, with c chosen on the host so that every neighbour earlier in key
// order falls in an earlier step and every later one in a later step.
//
// The wavefront was bound by the latency of its steps (779 launches of 22 us on the
// 4080x3068 frame, 34 micro-images each): 17.5 ms, now 1.7 ms (1024x768: 2.74 and
// 0.18 ms), bound by the gathers of the pairs kernel.
//
// Arithmetic is the reference's expressions evaluated as written, one
// rounding per operation (the library is built with -fmad=false), matching the
// CPU oracle (oracle/checks.c).
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include <math_constants.h>
#include "check_kernels.h"
#include "grid_barrier.cuh"
#include "smem_limit.h"

namespace pfd {

namespace {

__device__ __forceinline__ float hypot_canon(float x, float y)
{
    const double dx = (double)x, dy = (double)y;
    return (float)sqrt(dx * dx + dy * dy);
}

__device__ __forceinline__ bool bilinear_f32(const float* img, int W, int H, float x, float y, float& v)
{
    if (x < 0 || y < 0 || x > W - 1 || y > H - 1) return false;
    const int x0 = (int)floorf(x), y0 = (int)floorf(y);
    const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
    const float ax = x - (float)x0, ay = y - (float)y0;
    const float v00 = img[y0 * W + x0], v01 = img[y1 * W + x0], v10 = img[y0 * W + x1], v11 = img[y1 * W + x1];
    float s = ((1.0f - ax) * (1.0f - ay)) * v00;
    s = s + ((1.0f - ax) * ay) * v01;
    s = s + (ax * (1.0f - ay)) * v10;
    s = s + (ax * ay) * v11;
    v = s;
    return true;
}

// cv::meanStdDev of a 3x3 window (top-left x0, y0): double sums, row-major.
__device__ __forceinline__ void mean_std_3x3(const float* img, int W, int x0, int y0, float& mean, float& stdv)
{
    double s = 0.0, sq = 0.0;
    for (int y = y0; y < y0 + 3; ++y)
        for (int x = x0; x < x0 + 3; ++x) {
            const double v = (double)img[y * W + x];
            s += v;
            sq += v * v;
        }
    const double scale = 1.0 / 9.0;
    s *= scale;
    double var = sq * scale - s * s;
    if (var < 0.0) var = 0.0;
    mean = (float)s;
    stdv = (float)sqrt(var);
}

__device__ __forceinline__ bool patch_mean_std_centred(const float* img, int W, int H, float fx, float fy, float& m,
                                                       float& s)
{
    const int cx = (int)roundf(fx), cy = (int)roundf(fy);
    if (cx < 1 || cy < 1 || cx >= W - 1 || cy >= H - 1) return false;
    mean_std_3x3(img, W, cx - 1, cy - 1, m, s);
    return isfinite(m) && isfinite(s) && s > 1.0e-3f;
}

// ComputePhotoResidual, MIDisparityFilter.cpp:138-156
__device__ __forceinline__ float photo_residual(const float* ref, const float* nei, int W, int H, float px, float py,
                                               float qx, float qy)
{
    float Ir = 0.0f, In = 0.0f;
    if (!bilinear_f32(ref, W, H, px, py, Ir)) return CUDART_NAN_F;
    if (!bilinear_f32(nei, W, H, qx, qy, In)) return CUDART_NAN_F;
    float mr, sr, mn, sn;
    if (patch_mean_std_centred(ref, W, H, px, py, mr, sr) && patch_mean_std_centred(nei, W, H, qx, qy, mn, sn)) {
        const float Irn = (Ir - mr) / sr;
        const float Inn = (In - mn) / sn;
        return fabsf(Irn - Inn);
    }
    return fabsf(In - Ir);
}

// BilinearDisparity (MIDisparityFilter.cpp:80-118) over a neighbour's state.
__device__ __forceinline__ float bilinear_disp(const float4* plane, int W, int H, float x, float y, float min_valid)
{
    if (x < 0 || y < 0 || x > W - 1 || y > H - 1) return CUDART_NAN_F;
    const int x0 = (int)floorf(x), y0 = (int)floorf(y);
    const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
    const float ax = x - (float)x0, ay = y - (float)y0;
    const float d00 = plane[y0 * W + x0].w, d01 = plane[y1 * W + x0].w;
    const float d10 = plane[y0 * W + x1].w, d11 = plane[y1 * W + x1].w;
    if (!isfinite(d00) || d00 <= min_valid || !isfinite(d01) || d01 <= min_valid ||
        !isfinite(d10) || d10 <= min_valid || !isfinite(d11) || d11 <= min_valid)
        return CUDART_NAN_F;
    float r = ((1.0f - ax) * (1.0f - ay)) * d00;
    r = r + ((1.0f - ax) * ay) * d01;
    r = r + (ax * (1.0f - ay)) * d10;
    r = r + (ax * ay) * d11;
    return r;
}

__device__ __forceinline__ float bilinear_cost(const float* cost, int W, int H, float x, float y)
{
    if (x < 0 || y < 0 || x > W - 1 || y > H - 1) return CUDART_NAN_F;
    const int x0 = (int)floorf(x), y0 = (int)floorf(y);
    const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
    const float ax = x - (float)x0, ay = y - (float)y0;
    const float c00 = cost[y0 * W + x0], c01 = cost[y1 * W + x0], c10 = cost[y0 * W + x1], c11 = cost[y1 * W + x1];
    if (!isfinite(c00) || !isfinite(c01) || !isfinite(c10) || !isfinite(c11)) return CUDART_NAN_F;
    float r = ((1.0f - ax) * (1.0f - ay)) * c00;
    r = r + ((1.0f - ax) * ay) * c01;
    r = r + (ax * (1.0f - ay)) * c10;
    r = r + (ax * ay) * c11;
    return r;
}

struct NbDir { float dx, dy, scale; bool ok; };

__device__ __forceinline__ NbDir neighbour_dir(float2 c0, float2 c1, float unit)
{
    NbDir r{ 0.f, 0.f, 0.f, false };
    const float Bx = c0.x - c1.x, By = c0.y - c1.y;
    const float baseline = hypot_canon(Bx, By);
    if (baseline < 1.0e-6f) return r;
    r.dx = Bx / baseline;
    r.dy = By / baseline;
    r.scale = baseline / unit;
    r.ok = true;
    return r;
}

__device__ __forceinline__ int set_bits(uint32_t mask, int* out, int max_needed)
{
    int n = 0;
    for (int b = 0; mask && n < max_needed; ++b) {
        if (mask & 1u) out[n++] = b;
        mask >>= 1u;
    }
    return n;
}

// Stage 1 of FilterTile for one pixel; returns the reject reason (0 = keep).
// Also used, with geometry only, by the reprojection-error map.
__device__ __forceinline__ bool cost_ok(float c, const FilterCfg& cfg)
{
    if (!cfg.enable_cost_filter) return true;
    return !((!isfinite(c) || c < 0.0f) || (isfinite(c) && c > cfg.max_cost));
}

}  // namespace

// Gray micro-images are read as floats from the 8-bit tiles.
__global__ void pm_filter_kernel(CheckFrame F, FilterCfg cfg, StateDev st, const int* step_views, int n_step,
                                 uint8_t* reason, unsigned long long* stats)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int W = F.W, H = F.H, N = W * H;
    float* ref = (float*)smem;                        // [N]
    float* nei = ref + N;                              // [K][N] neighbour grays
    unsigned char* keep1 = (unsigned char*)(nei + (size_t)F.K * N);
    unsigned char* keepf = keep1 + N;
    __shared__ unsigned long long cnt[8];
    for (int item = blockIdx.x; item < n_step; item += gridDim.x) {
        const int v = step_views[item];
        const int nc = min(F.nb_counts[v], F.K);
        const size_t base = (size_t)v * N;
        if (threadIdx.x < 8) cnt[threadIdx.x] = 0;
        for (int e = threadIdx.x; e < N; e += blockDim.x) ref[e] = (float)F.gray[(size_t)v * F.tile_stride + e];
        for (int e = threadIdx.x; e < nc * N; e += blockDim.x) {
            const int k = e / N, r = e % N;
            const int nv = F.nb_ids[v * F.K + k];
            nei[e] = nv >= 0 ? (float)F.gray[(size_t)nv * F.tile_stride + r] : 0.0f;
        }
        __syncthreads();
        const float2 c0 = F.centers[v];
        for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
            const int x = idx % W, y = idx / W;
            keep1[idx] = 0;
            uint8_t why = kPrKeep;
            atomicAdd(&cnt[kFsTotal], 1ull);
            const float d = st.plane[base + idx].w;
            if (isfinite(d) && d > cfg.min_valid_disp) {
                atomicAdd(&cnt[kFsValidIn], 1ull);
                const float cost = st.cost[base + idx];
                if (!cost_ok(cost, cfg)) {
                    why = kPrCost;
                } else {
                    int vids[32];
                    int nv;
                    if (cfg.use_selected_views_only) nv = set_bits(st.sel[base + idx], vids, cfg.max_triplet);
                    else { nv = min(nc, cfg.max_triplet); for (int i = 0; i < nv; ++i) vids[i] = i; }
                    if (nv == 0) {
                        why = kPrNoSupport;
                    } else {
                        const float px = (float)x, py = (float)y;
                        int support = 0, good = 0;
                        for (int vi = 0; vi < nv; ++vi) {
                            const int b = vids[vi];
                            if (b < 0 || b >= nc) continue;
                            const int nvid = F.nb_ids[v * F.K + b];
                            if (nvid < 0) continue;
                            const NbDir g = neighbour_dir(c0, F.centers[nvid], F.baseline_unit);
                            if (!g.ok) continue;
                            const float qx = px + (g.dx * d) * g.scale;
                            const float qy = py + (g.dy * d) * g.scale;
                            if (qx < 0 || qy < 0 || qx > W - 1 || qy > H - 1) continue;
                            const size_t nbase = (size_t)nvid * N;
                            const float d_nei = bilinear_disp(st.plane + nbase, W, H, qx, qy, cfg.min_valid_disp);
                            if (!isfinite(d_nei)) continue;
                            if (cfg.enable_cost_filter && !cost_ok(bilinear_cost(st.cost + nbase, W, H, qx, qy), cfg)) continue;
                            ++support;
                            bool pass_geo = true, pass_photo = true;
                            if (cfg.enable_cycle_geo_filter) {
                                const float phx = qx - (g.dx * d_nei) * g.scale;
                                const float phy = qy - (g.dy * d_nei) * g.scale;
                                const float ge = hypot_canon(phx - px, phy - py);
                                pass_geo = isfinite(ge) && ge <= cfg.max_geo_err_px;
                            }
                            if (cfg.enable_cycle_photo_filter) {
                                const float pe = photo_residual(ref, nei + (size_t)b * N, W, H, px, py, qx, qy);
                                pass_photo = isfinite(pe) && pe <= cfg.max_photo_err_u;
                            }
                            if (pass_geo && pass_photo) ++good;
                        }
                        if (support < cfg.min_good_neighbors) why = kPrNoSupport;
                        else if (good < cfg.min_good_neighbors) why = kPrCycle;
                        else keep1[idx] = 1;
                    }
                }
                if (why == kPrCost) atomicAdd(&cnt[kFsCost], 1ull);
                if (why == kPrNoSupport) atomicAdd(&cnt[kFsNoSupport], 1ull);
                if (why == kPrCycle) atomicAdd(&cnt[kFsCycle], 1ull);
            }
            if (reason) reason[base + idx] = why;
        }
        __syncthreads();
        // spike pass (MIDisparityFilter.cpp:644-676): reads before any write
        for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
            keepf[idx] = keep1[idx];
            if (!cfg.enable_spike_filter || !keep1[idx]) continue;
            const int x = idx % W, y = idx / W;
            float nvals[8];
            int n = 0;
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    if (dx == 0 && dy == 0) continue;
                    const int xn = x + dx, yn = y + dy;
                    if (xn < 0 || yn < 0 || xn >= W || yn >= H) continue;
                    const int ni = yn * W + xn;
                    if (!keep1[ni]) continue;
                    const float dv = st.plane[base + ni].w;
                    if (!isfinite(dv) || dv <= cfg.min_valid_disp) continue;
                    nvals[n++] = dv;
                }
            if (n < cfg.spike_min_neighbors) continue;
            for (int a = 1; a < n; ++a) {
                const float t = nvals[a];
                int b = a - 1;
                while (b >= 0 && nvals[b] > t) { nvals[b + 1] = nvals[b]; --b; }
                nvals[b + 1] = t;
            }
            const float med = nvals[n / 2];
            const float cur = st.plane[base + idx].w;
            if (!isfinite(cur)) continue;
            if (fabsf(cur - med) > cfg.spike_abs_diff) {
                keepf[idx] = 0;
                if (reason) reason[base + idx] = kPrSpike;
                atomicAdd(&cnt[kFsSpike], 1ull);
            }
        }
        __syncthreads();
        // InvalidatePixel (MIDisparityFilter.cpp:158-174) for every rejected valid pixel
        for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
            const float d = st.plane[base + idx].w;
            if (!isfinite(d) || d <= cfg.min_valid_disp) continue;
            if (keepf[idx]) { atomicAdd(&cnt[kFsKept], 1ull); continue; }
            atomicAdd(&cnt[kFsRemoved], 1ull);
            st.plane[base + idx] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
            st.cost[base + idx] = 2.0f;
            st.disp[base + idx] = make_float4(-1.0f, -1.0f, 0.0f, 0.0f);
            if (cfg.clear_selected_views_when_invalid) st.sel[base + idx] = 0u;
        }
        __syncthreads();
        if (threadIdx.x < 8 && stats) atomicAdd(&stats[threadIdx.x], cnt[threadIdx.x]);
        __syncthreads();
    }
}

// ---- the filter in three launches -----------------------------------------------
namespace {

// FilterWork::head of a pixel: what its own state decides, and the counts that are final.
constexpr uint32_t kHeadInvalid = 0u, kHeadCost = 1u, kHeadNoViews = 2u, kHeadOpen = 3u;
__device__ __forceinline__ uint32_t make_head(uint32_t cls, int support, int good, int n)
{
    return cls | ((uint32_t)support << 2) | ((uint32_t)good << 8) | ((uint32_t)n << 14);
}

// Bytes -> floats of the view's tile and of its neighbours' tiles (as bytes).
__device__ __forceinline__ float bilinear_u8(const uint8_t* img, int W, int H, float x, float y)
{
    const int x0 = (int)floorf(x), y0 = (int)floorf(y);
    const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
    const float ax = x - (float)x0, ay = y - (float)y0;
    const float v00 = (float)img[y0 * W + x0], v01 = (float)img[y1 * W + x0];
    const float v10 = (float)img[y0 * W + x1], v11 = (float)img[y1 * W + x1];
    float s = ((1.0f - ax) * (1.0f - ay)) * v00;
    s = s + ((1.0f - ax) * ay) * v01;
    s = s + (ax * (1.0f - ay)) * v10;
    s = s + (ax * ay) * v11;
    return s;
}

// cv::meanStdDev of the 3x3 window centred on (cx, cy): the sums are integers, so
// they are the double sums exactly.
__device__ __forceinline__ bool patch_mean_std_u8(const uint8_t* img, int W, int H, int cx, int cy, float& m, float& s)
{
    if (cx < 1 || cy < 1 || cx >= W - 1 || cy >= H - 1) return false;
    int sum = 0, sq = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int v = img[(cy + dy) * W + cx + dx];
            sum += v;
            sq += v * v;
        }
    const double scale = 1.0 / 9.0;
    const double ds = (double)sum * scale;
    double var = (double)sq * scale - ds * ds;
    if (var < 0.0) var = 0.0;
    m = (float)ds;
    s = (float)sqrt(var);
    return isfinite(m) && isfinite(s) && s > 1.0e-3f;
}

__device__ __forceinline__ bool key_before(int2 a, int2 b) { return a.y < b.y || (a.y == b.y && a.x < b.x); }

}  // namespace

__global__ void __launch_bounds__(256) pm_filter_pairs_kernel(CheckFrame F, FilterCfg cfg, StateDev st, FilterWork X)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int W = F.W, H = F.H, N = W * H, v = blockIdx.x;
    const int nc = min(F.nb_counts[v], F.K);
    uint8_t* tiles = smem;                               // [1 + K][tile_stride]: the view, its neighbours
    NbDir* dir = (NbDir*)(smem + (size_t)(1 + F.K) * F.tile_stride);     // [K]
    int* ids = (int*)(dir + F.K);                        // [K] neighbour, -1 unusable; bit 30: earlier in key order
    const int words = F.tile_stride >> 4;
    for (int e = threadIdx.x; e < (1 + nc) * words; e += blockDim.x) {
        const int t = e / words;
        const int u = t == 0 ? v : F.nb_ids[v * F.K + t - 1];
        if (u >= 0) ((uint4*)tiles)[e] = ((const uint4*)(F.gray + (size_t)u * F.tile_stride))[e - t * words];
    }
    for (int k = threadIdx.x; k < nc; k += blockDim.x) {
        const int u = F.nb_ids[v * F.K + k];
        int id = -1;
        if (u >= 0) {
            dir[k] = neighbour_dir(F.centers[v], F.centers[u], F.baseline_unit);
            if (dir[k].ok) id = u | (key_before(F.keys[u], F.keys[v]) ? 1 << 30 : 0);
        }
        ids[k] = id;
    }
    __syncthreads();
    const size_t base = (size_t)v * N;
    for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
        const int x = idx % W, y = idx / W;
        const float d = st.plane[base + idx].w;
        uint32_t cls = kHeadInvalid;
        int support = 0, good = 0, n = 0;
        if (isfinite(d) && d > cfg.min_valid_disp) {
            uint32_t mask = cfg.use_selected_views_only ? st.sel[base + idx] : (nc < 32 ? (1u << nc) - 1u : ~0u);
            if (!cost_ok(st.cost[base + idx], cfg)) {
                cls = kHeadCost;
            } else if (mask == 0u || cfg.max_triplet <= 0) {
                cls = kHeadNoViews;
            } else {
                cls = kHeadOpen;
                const float px = (float)x, py = (float)y;
                const float Ir = (float)tiles[idx];
                float mr = 0.0f, sr = 0.0f;
                const bool ref_ok = cfg.enable_cycle_photo_filter && patch_mean_std_u8(tiles, W, H, x, y, mr, sr);
                for (int t = 0; mask && t < cfg.max_triplet; ++t) {
                    const int b = __ffs(mask) - 1;
                    mask &= mask - 1;
                    if (b >= nc) continue;
                    const int id = ids[b];
                    if (id < 0) continue;
                    const NbDir g = dir[b];
                    const float qx = px + (g.dx * d) * g.scale;
                    const float qy = py + (g.dy * d) * g.scale;
                    if (qx < 0 || qy < 0 || qx > W - 1 || qy > H - 1) continue;
                    const size_t nbase = (size_t)(id & ~(1 << 30)) * N;
                    const float d_nei = bilinear_disp(st.plane + nbase, W, H, qx, qy, cfg.min_valid_disp);
                    if (!isfinite(d_nei)) continue;
                    if (cfg.enable_cost_filter && !cost_ok(bilinear_cost(st.cost + nbase, W, H, qx, qy), cfg)) continue;
                    bool pass = true;
                    if (cfg.enable_cycle_geo_filter) {
                        const float phx = qx - (g.dx * d_nei) * g.scale;
                        const float phy = qy - (g.dy * d_nei) * g.scale;
                        const float ge = hypot_canon(phx - px, phy - py);
                        pass = isfinite(ge) && ge <= cfg.max_geo_err_px;
                    }
                    if (pass && cfg.enable_cycle_photo_filter) {
                        // ComputePhotoResidual, MIDisparityFilter.cpp:138-156 (the pixel is on the grid)
                        const uint8_t* nei = tiles + (size_t)(1 + b) * F.tile_stride;
                        const float In = bilinear_u8(nei, W, H, qx, qy);
                        float mn, sn, pe;
                        if (ref_ok && patch_mean_std_u8(nei, W, H, (int)roundf(qx), (int)roundf(qy), mn, sn))
                            pe = fabsf((Ir - mr) / sr - (In - mn) / sn);
                        else
                            pe = fabsf(In - Ir);
                        pass = isfinite(pe) && pe <= cfg.max_photo_err_u;
                    }
                    if (id & (1 << 30)) {
                        X.ent[(size_t)n * X.total + base + idx] =
                            (uint16_t)(b | ((int)floorf(qx) << 5) | ((int)floorf(qy) << 10) | (pass ? 1 << 15 : 0));
                        ++n;
                    } else {
                        ++support;
                        good += pass;
                    }
                }
            }
        }
        X.head[base + idx] = make_head(cls, support, good, n);
        X.disp[base + idx] = d;
    }
}

namespace {

// One view's tests under the masks of its earlier neighbours: per pixel the reject
// reason (smem why[N]; kPrKeep for a pixel that stays or was never valid).  Ends
// with a barrier.
__device__ __forceinline__ void eval_view(const CheckFrame& F, const FilterCfg& cfg, const FilterWork& X, int v,
                                          uint32_t* nmask, float* dv, uint8_t* keep, uint8_t* why)
{
    const int W = F.W, H = F.H, N = W * H, mw = X.mask_words;
    const int nc = min(F.nb_counts[v], F.K);
    const size_t base = (size_t)v * N;
    for (int e = threadIdx.x; e < nc * mw; e += blockDim.x) {
        const int k = e / mw, u = F.nb_ids[v * F.K + k];
        nmask[e] = u >= 0 ? __ldcg(X.mask + (size_t)u * mw + (e - k * mw)) : 0u;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
        const uint32_t head = X.head[base + idx];
        const uint32_t cls = head & 3u;
        dv[idx] = X.disp[base + idx];
        uint8_t r = kPrKeep;
        bool k1 = false;
        if (cls == kHeadCost) r = kPrCost;
        else if (cls == kHeadNoViews) r = kPrNoSupport;
        else if (cls == kHeadOpen) {
            int support = (int)((head >> 2) & 63u), good = (int)((head >> 8) & 63u);
            const int n = (int)(head >> 14);
            for (int j = 0; j < n; ++j) {
                const uint32_t e = X.ent[(size_t)j * X.total + base + idx];
                const uint32_t* m = nmask + (e & 31u) * mw;
                const int x0 = (int)((e >> 5) & 31u), y0 = (int)((e >> 10) & 31u);
                const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
                auto out = [&](int b) { return (m[b >> 5] >> (b & 31)) & 1u; };
                if (out(y0 * W + x0) | out(y0 * W + x1) | out(y1 * W + x0) | out(y1 * W + x1)) continue;
                ++support;
                good += (int)(e >> 15);
            }
            if (support < cfg.min_good_neighbors) r = kPrNoSupport;
            else if (good < cfg.min_good_neighbors) r = kPrCycle;
            else k1 = true;
        }
        keep[idx] = k1;
        why[idx] = r;
    }
    __syncthreads();
    if (cfg.enable_spike_filter)
        // spike pass (MIDisparityFilter.cpp:644-676): the disparity against the median
        // (element n / 2 in ascending order) of the kept neighbours'.  The median is too
        // low or too high exactly when the values too low, or too high, reach its place.
        for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
            if (!keep[idx]) continue;
            const int x = idx % W, y = idx / W;
            const float cur = dv[idx];
            int n = 0, lo = 0, hi = 0;
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                if (q == 4) continue;
                const int xn = x + q % 3 - 1, yn = y + q / 3 - 1;
                if (xn < 0 || yn < 0 || xn >= W || yn >= H) continue;
                const int ni = yn * W + xn;
                if (!keep[ni]) continue;
                const float val = dv[ni];
                ++n;
                if (fabsf(cur - val) > cfg.spike_abs_diff) { if (val < cur) ++lo; else ++hi; }
            }
            if (n < cfg.spike_min_neighbors || n == 0) continue;
            if (lo > n / 2 || n - hi <= n / 2) why[idx] = kPrSpike;
        }
    __syncthreads();
}

}  // namespace

__global__ void __launch_bounds__(256) pm_filter_resolve_kernel(CheckFrame F, FilterCfg cfg, FilterWork X, int* err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int N = F.W * F.H, mw = X.mask_words;
    uint32_t* nmask = (uint32_t*)smem;                   // [K][mw]
    float* dv = (float*)(nmask + F.K * mw);              // [N]
    uint8_t* keep = (uint8_t*)(dv + N);                  // [N]
    uint8_t* why = keep + N;                             // [N]
    unsigned int arrived = 0;
    // X.ctl: 0 barrier; 1, 2, 3 list lengths of rounds 1, 2, 3 mod 3; 4 settled; 5 a wait gave up
    auto barrier = [&]() {
        const bool ok = grid_barrier(X.ctl, ++arrived * gridDim.x, err);
        if (!ok && threadIdx.x == 0) X.ctl[kFilterGaveUp] = 1u;
        return ok;
    };
    for (int round = 1; round <= F.V + 2; ++round) {
        // views with an earlier neighbour that changed in the last round (or already in
        // this one); all of them in the first round
        int n_list = F.V;
        if (round > 1) {
            if (blockIdx.x == 0 && threadIdx.x == 0) X.ctl[1 + (round + 1) % 3] = 0u;
            for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < F.V; v += gridDim.x * blockDim.x) {
                const int nc = min(F.nb_counts[v], F.K);
                const int2 key = F.keys[v];
                bool dirty = false;
                for (int k = 0; k < nc && !dirty; ++k) {
                    const int u = F.nb_ids[v * F.K + k];
                    if (u >= 0 && __ldcg(X.changed + u) >= round - 1 && key_before(F.keys[u], key)) dirty = true;
                }
                if (dirty) X.list[atomicAdd(X.ctl + 1 + round % 3, 1u)] = v;
            }
            if (!barrier()) return;
            n_list = (int)__ldcg(X.ctl + 1 + round % 3);
            if (n_list == 0) {
                if (blockIdx.x == 0 && threadIdx.x == 0) X.ctl[kFilterSettled] = 1u;
                return;
            }
        }
        for (int i = blockIdx.x; i < n_list; i += gridDim.x) {
            const int v = round > 1 ? __ldcg(X.list + i) : i;
            eval_view(F, cfg, X, v, nmask, dv, keep, why);
            int diff = 0;
            for (int b0 = 0; b0 < mw * 32; b0 += blockDim.x) {
                const int b = b0 + threadIdx.x;
                const uint32_t bits = __ballot_sync(0xffffffffu, b < N && why[b < N ? b : 0] != kPrKeep);
                if ((threadIdx.x & 31) == 0 && b < mw * 32) {
                    uint32_t* m = X.mask + (size_t)v * mw + (b >> 5);
                    if (__ldcg(m) != bits) { __stcg(m, bits); diff = 1; }
                }
            }
            if (__syncthreads_or(diff) && threadIdx.x == 0) __stcg(X.changed + v, round);
        }
        if (!barrier()) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, PFD_DEVERR_TMA_TIMEOUT);       // key order has no cycles: not reached
}

__global__ void __launch_bounds__(256) pm_filter_apply_kernel(CheckFrame F, FilterCfg cfg, StateDev st, FilterWork X,
                                                              uint8_t* reason, unsigned long long* stats)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if (!X.ctl[kFilterSettled] || X.ctl[kFilterGaveUp]) return;
    const int N = F.W * F.H, v = blockIdx.x;
    uint32_t* nmask = (uint32_t*)smem;
    float* dv = (float*)(nmask + F.K * X.mask_words);
    uint8_t* keep = (uint8_t*)(dv + N);
    uint8_t* why = keep + N;
    __shared__ unsigned int cnt[8];
    if (threadIdx.x < 8) cnt[threadIdx.x] = 0;
    eval_view(F, cfg, X, v, nmask, dv, keep, why);
    const size_t base = (size_t)v * N;
    unsigned int valid = 0, cost = 0, support = 0, cycle = 0, spike = 0;
    for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
        const uint8_t r = why[idx];
        if (reason) reason[base + idx] = r;
        if ((X.head[base + idx] & 3u) == kHeadInvalid) continue;
        ++valid;
        cost += r == kPrCost;
        support += r == kPrNoSupport;
        cycle += r == kPrCycle;
        spike += r == kPrSpike;
        if (r == kPrKeep) continue;
        // InvalidatePixel (MIDisparityFilter.cpp:158-174)
        st.plane[base + idx] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        st.cost[base + idx] = 2.0f;
        st.disp[base + idx] = make_float4(-1.0f, -1.0f, 0.0f, 0.0f);
        if (cfg.clear_selected_views_when_invalid) st.sel[base + idx] = 0u;
    }
    const unsigned int part[5] = { valid, cost, support, cycle, spike };
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const unsigned int t = __reduce_add_sync(0xffffffffu, part[i]);
        if ((threadIdx.x & 31) == 0 && t) atomicAdd(&cnt[i], t);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int gone = cnt[1] + cnt[2] + cnt[3] + cnt[4];
        atomicAdd(stats + kFsTotal, (unsigned long long)N);
        if (cnt[0]) atomicAdd(stats + kFsValidIn, (unsigned long long)cnt[0]);
        if (cnt[0] - gone) atomicAdd(stats + kFsKept, (unsigned long long)(cnt[0] - gone));
        if (gone) atomicAdd(stats + kFsRemoved, (unsigned long long)gone);
        if (cnt[1]) atomicAdd(stats + kFsCost, (unsigned long long)cnt[1]);
        if (cnt[2]) atomicAdd(stats + kFsNoSupport, (unsigned long long)cnt[2]);
        if (cnt[3]) atomicAdd(stats + kFsCycle, (unsigned long long)cnt[3]);
        if (cnt[4]) atomicAdd(stats + kFsSpike, (unsigned long long)cnt[4]);
    }
}

// ComputeTileReprojectionErrorMap for every pixel of every view (read-only).
__global__ void pm_reproj_kernel(CheckFrame F, FilterCfg cfg, StateDev st, float* err)
{
    const int N = F.W * F.H;
    const size_t total = (size_t)F.V * N;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int v = (int)(t / N), idx = (int)(t % N);
        const int W = F.W, H = F.H, x = idx % W, y = idx / W;
        const int nc = min(F.nb_counts[v], F.K);
        float out = -1.0f;
        const float d = st.plane[t].w;
        if (isfinite(d) && d > cfg.min_valid_disp && cost_ok(st.cost[t], cfg)) {
            int vids[32];
            int nv;
            if (cfg.use_selected_views_only) nv = set_bits(st.sel[t], vids, cfg.max_triplet);
            else { nv = min(nc, cfg.max_triplet); for (int i = 0; i < nv; ++i) vids[i] = i; }
            const float px = (float)x, py = (float)y;
            float ge[32];
            int ng = 0;
            const float2 c0 = F.centers[v];
            for (int vi = 0; vi < nv; ++vi) {
                const int b = vids[vi];
                if (b < 0 || b >= nc) continue;
                const int nvid = F.nb_ids[v * F.K + b];
                if (nvid < 0) continue;
                const NbDir g = neighbour_dir(c0, F.centers[nvid], F.baseline_unit);
                if (!g.ok) continue;
                const float qx = px + (g.dx * d) * g.scale;
                const float qy = py + (g.dy * d) * g.scale;
                if (qx < 0 || qy < 0 || qx > W - 1 || qy > H - 1) continue;
                const size_t nbase = (size_t)nvid * N;
                const float d_nei = bilinear_disp(st.plane + nbase, W, H, qx, qy, cfg.min_valid_disp);
                if (!isfinite(d_nei)) continue;
                if (cfg.enable_cost_filter && !cost_ok(bilinear_cost(st.cost + nbase, W, H, qx, qy), cfg)) continue;
                const float phx = qx - (g.dx * d_nei) * g.scale;
                const float phy = qy - (g.dy * d_nei) * g.scale;
                const float e = hypot_canon(phx - px, phy - py);
                if (isfinite(e)) ge[ng++] = e;
            }
            if (ng >= cfg.min_good_neighbors) {
                for (int a = 1; a < ng; ++a) {
                    const float tv = ge[a];
                    int b = a - 1;
                    while (b >= 0 && ge[b] > tv) { ge[b + 1] = ge[b]; --b; }
                    ge[b + 1] = tv;
                }
                // QuantileFromSorted(v, 0.5), MIDisparityFilter.cpp:36-51
                const float pos = 0.5f * (float)(ng - 1);
                const int lo = (int)floorf(pos), hi = (int)ceilf(pos);
                const float tq = pos - (float)lo;
                out = (lo == hi) ? ge[lo] : ge[lo] * (1.0f - tq) + ge[hi] * tq;
            }
        }
        err[t] = out;
    }
}

namespace {

// cv::BORDER_REFLECT_101 (borderInterpolate)
__device__ __forceinline__ int reflect101(int i, int n)
{
    if (n == 1) return 0;
    while (i < 0 || i >= n) i = i < 0 ? -i : 2 * n - 2 - i;
    return i;
}

// bilinear_disp lambda (MICycleCheck.cpp:306-325): non-finite corners replaced
__device__ __forceinline__ float bilinear_disp_cycle(const float4* plane, int W, int H, float fx, float fy)
{
    if (fx < 0 || fy < 0 || fx > W - 1 || fy > H - 1) return CUDART_NAN_F;
    const int x0 = (int)floorf(fx), y0 = (int)floorf(fy);
    const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, H - 1);
    const float ax = fx - (float)x0, ay = fy - (float)y0;
    float d00 = plane[y0 * W + x0].w, d01 = plane[y1 * W + x0].w;
    float d10 = plane[y0 * W + x1].w, d11 = plane[y1 * W + x1].w;
    if (!isfinite(d00)) d00 = 0.0f;
    if (!isfinite(d01)) d01 = d00;
    if (!isfinite(d10)) d10 = d00;
    if (!isfinite(d11)) d11 = d00;
    float r = ((1.0f - ax) * (1.0f - ay)) * d00;
    r = r + ((1.0f - ax) * ay) * d01;
    r = r + (ax * (1.0f - ay)) * d10;
    r = r + (ax * ay) * d11;
    return r;
}

__device__ __forceinline__ float min_std(float a, float b) { return (b < a) ? b : a; }   // std::min
__device__ __forceinline__ float max_std(float a, float b) { return (a < b) ? b : a; }   // std::max

}  // namespace

// One CTA per micro-image: BuildTextureMaskAndViz on the reference gray, the
// per-pixel cycle errors, then the tile's sums in pixel order (one lane per
// sum, so each double sum keeps the reference's order; a pixel outside a sum
// adds +0).  The gray values are integers, so every window sum is an exact
// integer sum and only the final products are doubles.
// Bound by the gathers of the neighbours' state and the four-neighbour loop.  With
// the window sums in doubles, 49 and 9 terms per pixel, the tiles as floats and the
// histogram counted pixel by pixel in global memory:
// 4.36 -> 0.79 ms on the 4080x3068 frame.
__global__ void __launch_bounds__(256) pm_cycle_kernel(CheckFrame F, CycleCfg cfg, StateDev st, float* geo_err,
                                                       float* pho_err, uint8_t* texmask, CycleTileRec* recs,
                                                       unsigned int* hist)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int W = F.W, H = F.H, N = W * H, v = blockIdx.x, lane = threadIdx.x & 31;
    uint8_t* tiles = smem;                               // [1 + K][tile_stride]: the view, its neighbours
    NbDir* dir = (NbDir*)(smem + (size_t)(1 + F.K) * F.tile_stride);     // [K]
    int* ids = (int*)(dir + F.K);                        // [K] neighbour, -1 unusable
    int* h1 = ids + F.K;                                 // [N] 7-sums along rows, and of squares
    int* h2 = h1 + N;
    float* gavg = (float*)h1;                            // [N] per-pixel mean errors (after the mask is made)
    float* pavg = (float*)h2;
    uint8_t* flag = (uint8_t*)(h2 + N);                  // [N] bit 0 sample, bit 1 textured
    uint8_t* tm = flag + N;                              // [N] texture mask
    __shared__ int comp[6];
    __shared__ unsigned int mnmx[2], bins[kCycleHistBins];
    const int nc = min(F.nb_counts[v], F.K);
    const size_t base = (size_t)v * N;
    if (threadIdx.x < 6) comp[threadIdx.x] = 0;
    if (threadIdx.x == 0) { mnmx[0] = 0x7f800000u; mnmx[1] = 0u; }
    for (int i = threadIdx.x; i < kCycleHistBins; i += blockDim.x) bins[i] = 0u;
    const int words = F.tile_stride >> 4;
    for (int e = threadIdx.x; e < (1 + nc) * words; e += blockDim.x) {
        const int t = e / words;
        const int u = t == 0 ? v : F.nb_ids[v * F.K + t - 1];
        if (u >= 0) ((uint4*)tiles)[e] = ((const uint4*)(F.gray + (size_t)u * F.tile_stride))[e - t * words];
    }
    for (int k = threadIdx.x; k < nc; k += blockDim.x) {
        const int u = F.nb_ids[v * F.K + k];
        ids[k] = -1;                                     // no gray image: the sample fails
        if (u >= 0) {
            dir[k] = neighbour_dir(F.centers[v], F.centers[u], F.baseline_unit);
            if (dir[k].ok) ids[k] = u;
        }
    }
    __syncthreads();
    // ---- texture mask: Sobel magnitude and 7x7 variance
    for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
        const int y = idx / W, x = idx - y * W;
        int s1 = 0, s2 = 0;
#pragma unroll
        for (int dx = -3; dx <= 3; ++dx) {
            const int t = tiles[y * W + reflect101(x + dx, W)];
            s1 += t;
            s2 += t * t;
        }
        h1[idx] = s1;
        h2[idx] = s2;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < N; idx += blockDim.x) {
        const int y = idx / W, x = idx - y * W;
        const int xm = reflect101(x - 1, W), xp = reflect101(x + 1, W);
        const int ym = reflect101(y - 1, H) * W, yp = reflect101(y + 1, H) * W, yc = y * W;
        const int mm = tiles[ym + xm], mp = tiles[ym + xp], pm = tiles[yp + xm], pp = tiles[yp + xp];
        const float gx = (float)((mp - mm) + 2 * ((int)tiles[yc + xp] - (int)tiles[yc + xm]) + (pp - pm));
        const float gy = (float)((pm - mm) + 2 * ((int)tiles[yp + x] - (int)tiles[ym + x]) + (pp - mp));
        const float mag = sqrtf(gx * gx + gy * gy);
        int s1 = 0, s2 = 0;
#pragma unroll
        for (int dy = -3; dy <= 3; ++dy) {
            const int r = reflect101(y + dy, H) * W + x;
            s1 += h1[r];
            s2 += h2[r];
        }
        const float mean = (float)((double)s1 * (1.0 / 49.0)), mean2 = (float)((double)s2 * (1.0 / 49.0));
        const float var = mean2 - mean * mean;
        const bool m1 = mag > cfg.sobel_thresh, m2 = var > cfg.var_thresh;
        tm[idx] = (cfg.use_and ? (m1 && m2) : (m1 || m2)) ? 255 : 0;
    }
    __syncthreads();
    // ---- per-pixel cycle errors
    int total = 0, good = 0, good_geo = 0, good_photo = 0, n_all = 0, n_masked = 0;
    uint32_t mn = 0x7f800000u, mx = 0u;
    const int n32 = (N + 31) & ~31;
    for (int idx = threadIdx.x; idx < n32; idx += blockDim.x) {
        const int y = idx / W, x = idx - y * W;
        float gcell = 0.0f, pcell = 0.0f, ga = 0.0f, pa = 0.0f;
        uint8_t fl = 0;
        int bin = -1;
        if (idx < N) {
            const float d = st.plane[base + idx].w;
            uint32_t mask = isfinite(d) ? st.sel[base + idx] : 0u;
            if (mask && cfg.max_triplet > 0) {
                const float px = (float)x, py = (float)y;
                float gsum = 0.0f, psum = 0.0f, mr = 0.0f, sr = 0.0f;
                int cnt = 0, gate = 0, gate_geo = 0, gate_photo = 0;
                const float Ir = (float)tiles[idx];
                // patch_mean_std lambda (MICycleCheck.cpp:327-339): 3x3 window, top-left round(p) - 2
                const bool ref_ok = x >= 2 && y >= 2 && x < W - 2 && y < H - 2 && patch_mean_std_u8(tiles, W, H, x - 1, y - 1, mr, sr);
                for (int t = 0; mask && t < cfg.max_triplet; ++t) {
                    const int b = __ffs(mask) - 1;
                    mask &= mask - 1;
                    if (b >= nc || ids[b] < 0) continue;
                    const NbDir g = dir[b];
                    const float qx = px + (g.dx * d) * g.scale;
                    const float qy = py + (g.dy * d) * g.scale;
                    if (qx < 0 || qy < 0 || qx > W - 1 || qy > H - 1) continue;
                    const float d_nei = bilinear_disp_cycle(st.plane + (size_t)ids[b] * N, W, H, qx, qy);
                    const float phx = qx - (g.dx * d_nei) * g.scale;
                    const float phy = qy - (g.dy * d_nei) * g.scale;
                    const float geo_e = hypot_canon(phx - px, phy - py);
                    if (!(geo_e < (float)(W * 2))) continue;
                    const uint8_t* nimg = tiles + (size_t)(1 + b) * F.tile_stride;
                    const float In = bilinear_u8(nimg, W, H, qx, qy);
                    float mn, sn, phe;
                    const int cx = (int)roundf(qx), cy = (int)roundf(qy);
                    if (ref_ok && cx >= 2 && cy >= 2 && cx < W - 2 && cy < H - 2 &&
                        patch_mean_std_u8(nimg, W, H, cx - 1, cy - 1, mn, sn)) {
                        const float Irn = (Ir - mr) / sr, Inn = (In - mn) / sn;
                        phe = fabsf(Irn - Inn);
                    } else {
                        phe = fabsf(In - Ir);
                    }
                    const float phe_raw = phe;
                    if (isfinite(phe)) phe = min_std(phe, 3.0f);
                    const float geo_used = cfg.clamp_geo ? min_std(geo_e, cfg.geo_u_px) : geo_e;
                    const float phe_used = cfg.clamp_photo ? min_std(phe, cfg.photo_u) : phe;
                    const bool pg = cfg.gate_use_clamped ? (geo_used <= cfg.gate_geo_px) : (geo_e <= cfg.gate_geo_px);
                    const bool pp = cfg.gate_use_clamped ? (phe_used <= cfg.gate_photo_u) : (phe_raw <= cfg.gate_photo_u);
                    gate += (pg && pp);
                    gate_geo += pg;
                    gate_photo += pp;
                    const bool ok = cfg.pixel_gate_enabled ? (pg && pp) : true;
                    if (ok) { gsum = gsum + geo_used; psum = psum + phe_used; ++cnt; }
                    if (cnt > 0) { gcell = max_std(gcell, geo_used); pcell = max_std(pcell, phe_used); }
                }
                if (ref_ok) {
                    ++total;
                    good += gate >= cfg.gate_min_good_neighbors;
                    good_geo += gate_geo >= cfg.gate_min_good_neighbors;
                    good_photo += gate_photo >= cfg.gate_min_good_neighbors;
                }
                if ((!cfg.pixel_gate_enabled && cnt > 0) || (cfg.pixel_gate_enabled && cnt >= cfg.gate_min_good_neighbors)) {
                    ga = cnt > 0 ? gsum / (float)cnt : 0.0f;
                    pa = cnt > 0 ? psum / (float)cnt : 0.0f;
                    fl = 1 | (tm[idx] ? 2 : 0);
                    ++n_all;
                    if (tm[idx]) {
                        ++n_masked;
                        // doubling is exact: floor(ga / 0.5)
                        if (isfinite(ga) && !(ga < 0.0f)) bin = (int)fminf(2.0f * ga, (float)(kCycleHistBins - 1));
                    }
                }
            }
        }
        // histogram and range of the masked samples: one addition per bin that the warp
        // meets (most errors fall into a few bins, whose global counters would be the
        // bottleneck); finite values >= 0 order as their bits do (-0 counts as 0)
        const uint32_t bits = __float_as_uint(ga + 0.0f);
        mn = min(mn, bin >= 0 ? bits : 0x7f800000u);
        mx = max(mx, bin >= 0 ? bits : 0u);
        for (uint32_t todo = __ballot_sync(0xffffffffu, bin >= 0); todo;) {
            const int lead = __shfl_sync(0xffffffffu, bin, __ffs(todo) - 1);
            const uint32_t same = __ballot_sync(0xffffffffu, bin == lead);
            if (lane == __ffs(same) - 1) atomicAdd(&bins[lead], (unsigned int)__popc(same));
            todo &= ~same;
        }
        if (idx >= N) continue;
        flag[idx] = fl;
        gavg[idx] = ga;
        pavg[idx] = pa;
        if (geo_err) geo_err[base + idx] = gcell;
        if (pho_err) pho_err[base + idx] = pcell;
        if (texmask) texmask[base + idx] = tm[idx];
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) { atomicMin(&mnmx[0], mn); atomicMax(&mnmx[1], mx); }
    const int part[6] = { total, good, good_geo, good_photo, n_all, n_masked };
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int t = __reduce_add_sync(0xffffffffu, part[i]);
        if (lane == 0 && t) atomicAdd(&comp[i], t);
    }
    __syncthreads();
    if (hist)
        for (int i = threadIdx.x; i < kCycleHistBins; i += blockDim.x)
            if (bins[i]) atomicAdd(&hist[i], bins[i]);
    // ---- tile sums, each by one lane in pixel order
    const int t = threadIdx.x;
    if (t < 8) {
        const bool sq = (t & 1) != 0;
        const uint8_t need = (t & 4) ? 3 : 1;
        const float* a = (t & 2) ? pavg : gavg;
        double acc = 0.0;
#pragma unroll 8
        for (int i = 0; i < N; ++i) {
            const float x = a[i];
            const float s = sq ? x * x : x;
            acc += (flag[i] & need) == need ? (double)s : 0.0;
        }
        CycleTileRec& r = recs[v];
        switch (t) {
            case 0: r.sum_geo = acc; break;
            case 1: r.sq_geo = acc; break;
            case 2: r.sum_photo = acc; break;
            case 3: r.sq_photo = acc; break;
            case 4: r.sum_geo_m = acc; break;
            case 5: r.sq_geo_m = acc; break;
            case 6: r.sum_photo_m = acc; break;
            default: r.sq_photo_m = acc; break;
        }
    } else if (t == 8) {
        recs[v].n = comp[4];
        recs[v].n_masked = comp[5];
        recs[v].min_geo_m = __uint_as_float(mnmx[0]);
        recs[v].max_geo_m = __uint_as_float(mnmx[1]);
        recs[v].comp_total = comp[0];
        recs[v].comp_good = comp[1];
        recs[v].comp_good_geo = comp[2];
        recs[v].comp_good_photo = comp[3];
    }
}

int cycle_smem_bytes(const CheckFrame& F)
{
    const int N = F.W * F.H;
    return (3 + F.K) * N * 4 + 2 * N;                    // of the plan that decides what is refused
}

cudaError_t launch_cycle(const CheckFrame& F, const CycleCfg& cfg, const StateDev& st, float* geo_err, float* pho_err,
                         uint8_t* texmask, CycleTileRec* recs, unsigned int* hist, cudaStream_t s)
{
    if (F.V <= 0) return cudaSuccess;
    const int N = F.W * F.H;
    const int smem = (1 + F.K) * F.tile_stride + F.K * (int)(sizeof(NbDir) + sizeof(int)) + N * 10;
    cudaError_t e = allow_dynamic_smem((const void*)pm_cycle_kernel, smem);
    if (e != cudaSuccess) return e;
    const int threads = N < 256 ? ((N + 31) / 32) * 32 : 256;
    pm_cycle_kernel<<<F.V, threads < 64 ? 64 : threads, smem, s>>>(F, cfg, st, geo_err, pho_err, texmask, recs, hist);
    return cudaGetLastError();
}

// Room per micro-image of P >= 4 pixels: the idle state holds 16 P bytes in plane (8 P
// needed), 16 P in disp (4 + 4 ceil(P / 32), and 32 for ctl once: 40 <= 64 at P = 4), 4 P
// in sel (4); the cost vectors hold 4 K P (2 K P: a pixel has at most one test per
// neighbour, whatever max_triplet).
FilterWork filter_work(const CheckFrame& F, const StateDev& idle, float* cvec)
{
    FilterWork X;
    X.total = (size_t)F.V * F.W * F.H;
    X.mask_words = (F.W * F.H + 31) / 32;
    X.head = (uint32_t*)idle.plane;
    X.disp = (float*)(X.head + X.total);
    X.ctl = (unsigned int*)idle.disp;
    X.changed = (int*)(X.ctl + 8);
    X.mask = (uint32_t*)(X.changed + F.V);
    X.zeroed = (unsigned char*)X.ctl;
    X.zeroed_bytes = 32 + 4 * (size_t)F.V * (1 + X.mask_words);
    X.list = (int*)idle.sel;
    X.ent = (uint16_t*)cvec;
    return X;
}

static int filter_threads(const CheckFrame& F) { return std::min(256, (F.W * F.H + 31) / 32 * 32); }
static int filter_mask_smem(const CheckFrame& F, const FilterWork& X) { return F.K * X.mask_words * 4 + F.W * F.H * 6; }

cudaError_t launch_filter_apply(const CheckFrame& F, const FilterCfg& cfg, const StateDev& st, const FilterWork& X,
                                uint8_t* reason, unsigned long long* stats, cudaStream_t s)
{
    pm_filter_apply_kernel<<<F.V, filter_threads(F), filter_mask_smem(F, X), s>>>(F, cfg, st, X, reason, stats);
    return cudaGetLastError();
}

cudaError_t launch_filter(const CheckFrame& F, const FilterCfg& cfg, const StateDev& st, const FilterWork& X,
                          uint8_t* reason, unsigned long long* stats, int* err, cudaStream_t s)
{
    if (F.V <= 0) return cudaSuccess;
    const int smem_a = (1 + F.K) * F.tile_stride + F.K * (int)(sizeof(NbDir) + sizeof(int));
    const int smem_b = filter_mask_smem(F, X);
    cudaError_t e = cudaMemsetAsync(X.zeroed, 0, X.zeroed_bytes, s);
    if (e == cudaSuccess)
        e = allow_dynamic_smem((const void*)pm_filter_pairs_kernel, smem_a);
    if (e != cudaSuccess) return e;
    const int threads = filter_threads(F);
    pm_filter_pairs_kernel<<<F.V, threads, smem_a, s>>>(F, cfg, st, X);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pm_filter_resolve_kernel, threads, smem_b);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)std::max(1, std::min(F.V, sms * std::min(per_sm, 4))));
    lc.blockDim = dim3((unsigned)threads);
    lc.dynamicSmemBytes = (size_t)smem_b;
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, pm_filter_resolve_kernel, F, cfg, X, err);
    if (e != cudaSuccess) return e;
    return launch_filter_apply(F, cfg, st, X, reason, stats, s);
}

int filter_smem_bytes(const CheckFrame& F)
{
    const int N = F.W * F.H;
    return (1 + F.K) * N * 4 + 2 * N;
}

cudaError_t launch_filter_step(const CheckFrame& F, const FilterCfg& cfg, const StateDev& st, const int* step_views,
                               int n_step, uint8_t* reason, unsigned long long* stats, cudaStream_t s)
{
    if (n_step <= 0) return cudaSuccess;
    const int smem = filter_smem_bytes(F);
    const int threads = F.W * F.H < 256 ? ((F.W * F.H + 31) / 32) * 32 : 256;
    cudaError_t e = allow_dynamic_smem((const void*)pm_filter_kernel, smem);
    if (e != cudaSuccess) return e;
    pm_filter_kernel<<<n_step, threads, smem, s>>>(F, cfg, st, step_views, n_step, reason, stats);
    return cudaGetLastError();
}

cudaError_t launch_reproj(const CheckFrame& F, const FilterCfg& cfg, const StateDev& st, float* err, cudaStream_t s)
{
    const size_t total = (size_t)F.V * F.W * F.H;
    const int blocks = (int)std::min<size_t>((total + 255) / 256, 148 * 16);
    pm_reproj_kernel<<<blocks, 256, 0, s>>>(F, cfg, st, err);
    return cudaGetLastError();
}

}  // namespace pfd
