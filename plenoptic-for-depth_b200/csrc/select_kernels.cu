// select_kernels.cu -- MISimilarityMeasure::MeasureSimilarity (Util/
// MISimilarityMeasure.cpp:173-284) for many (micro-image, candidate) pairs.
//
// Both micro-images are binarised (threshold 128: 255 above, 0 otherwise).
// The candidate is shifted along the baseline in steps of 2 px; for every
// step the lane counts, over the overlap rectangle, the pixels where the
// reference micro-image equals the shifted candidate, and the similarity is
// the largest count.  The shift loop follows the reference as it runs (an
// OpenMP loop nested in a parallel region, hence sequential): step k uses the
// shift step k - 1 left behind (0 for steps 0 and 1), and once the shift
// leaves the image it stays there.  The shifted candidate is
// cv::warpAffine(INTER_NEAREST) of a translation, OpenCV's 10-bit fixed
// point: source column x + floor((rnd(-1024 sx) + 512) / 1024), source row
// floor((rnd(1024 (y - sy)) + 512) / 1024), rnd rounding half to even, 0
// outside.  Integer conversions of the host code follow x86 (NaN and
// out-of-range values give INT_MIN).
#include <algorithm>
#include <climits>
#include <cstdint>
#include "select_kernels.h"

namespace pfd {

namespace {

__device__ __forceinline__ int trunc_x86(float x) { return fabsf(x) < 2147483648.0f ? __float2int_rz(x) : INT_MIN; }
__device__ __forceinline__ int round_x86(float x) { return fabsf(x) < 2147483648.0f ? __float2int_rn(x) : INT_MIN; }

}  // namespace

// Binarised micro-images as one word per row: bit x of rows[v][y] is T(y, x) > 128.
template <class Row>
__global__ void __launch_bounds__(128) pm_binarise_kernel(const uint8_t* __restrict__ gray, int tile_stride, int W, int H,
                                                          int V, Row* __restrict__ rows)
{
    const size_t n = (size_t)V * H;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const int v = (int)(t / H), y = (int)(t - (size_t)v * H);
        const uint8_t* p = gray + (size_t)v * tile_stride + (size_t)y * W;
        Row r = 0;
        for (int x = 0; x < W; ++x) r |= (Row)(p[x] > 128 ? 1 : 0) << x;
        rows[t] = r;
    }
}

__device__ __forceinline__ int popc(uint32_t x) { return __popc(x); }
__device__ __forceinline__ int popc(uint64_t x) { return __popcll(x); }

// G lanes per pair, one shift step per lane; a step compares a whole row at once,
// the candidate's row moved by the step's column offset.  Against one pixel per lane
// with the row coordinate in double per pixel, step after step: 9.7 -> 0.97 ms for
// the 2.3 M pairs of the 4080x3068 frame (one row per lane, step after step: 1.62 ms).
template <class Row, int G>
__global__ void __launch_bounds__(128) pm_similarity_kernel(const Row* __restrict__ rows, int W, int H,
                                                            const float2* __restrict__ centers,
                                                            const int2* __restrict__ pairs, int n,
                                                            uint16_t* __restrict__ out)
{
    const int lane = threadIdx.x & (G - 1);
    const unsigned mask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
    const int p = blockIdx.x * (128 / G) + threadIdx.x / G;
    if (p >= n) return;                                  // whole groups leave together
    const int2 pr = pairs[p];
    const Row* src = rows + (size_t)pr.x * H;
    const Row* nb = rows + (size_t)pr.y * H;
    float dx = __fsub_rn(centers[pr.y].x, centers[pr.x].x), dy = __fsub_rn(centers[pr.y].y, centers[pr.x].y);
    if (fabsf(dx) < 5.0f) dx = 0.0f;
    if (fabsf(dy) < 5.0f) dy = 0.0f;
    const float norm = __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
    const float dxs = __fmul_rn(__fdiv_rn(dx, norm), 2.0f), dys = __fmul_rn(__fdiv_rn(dy, norm), 2.0f);
    int dxc = trunc_x86(__fdiv_rn((float)W, fabsf(dxs)));
    int dyc = trunc_x86(__fdiv_rn((float)H, fabsf(dys)));
    if (dxs == 0.0f) dxc = 0;
    else if (dys == 0.0f) dyc = 0;
    const int steps = dxc > dyc ? dxc : dyc;
    const Row all = W == (int)sizeof(Row) * 8 ? ~(Row)0 : ((Row)1 << W) - 1;
    int best = 0;
    for (int step = lane; step < steps && step < 4096; step += G) {
        // step k runs with the shift that step k - 1 left; shifts grow with the step, so
        // from the first one that leaves the image on nothing counts
        const float sx = step == 0 ? 0.0f : __fmul_rn((float)(step - 1), dxs);
        const float sy = step == 0 ? 0.0f : __fmul_rn((float)(step - 1), dys);
        if (fabsf(sx) >= (float)W || fabsf(sy) >= (float)H) break;
        // the fixed point's offsets: 1024 (y - sy) rounds, half to even, to 1024 y plus the
        // rounded -1024 sy (1024 y is even), so the row's is the same for every row; the
        // products are exact in single precision
        const int ox = (round_x86(__fmul_rn(-sx, 1024.0f)) + 512) >> 10;
        const int oy = (round_x86(__fmul_rn(-sy, 1024.0f)) + 512) >> 10;
        const int x1 = (int)(0.0f < sx ? sx : 0.0f), y1 = (int)(0.0f < sy ? sy : 0.0f);
        const float ex = __fsub_rn(__fadd_rn(sx, (float)W), 1.0f), ey = __fsub_rn(__fadd_rn(sy, (float)H), 1.0f);
        const int x2 = (int)floorf(ex < (float)(W - 1) ? ex : (float)(W - 1));
        const int y2 = (int)floorf(ey < (float)(H - 1) ? ey : (float)(H - 1));
        if (x2 < x1 || y2 < y1) continue;
        const Row cols = (all >> (W - 1 - x2)) & ~(((Row)1 << x1) - 1);                // columns x1 .. x2
        constexpr int bits = (int)sizeof(Row) * 8;
        const int right = ox >= 0 ? min(ox, bits) : 0, left = ox >= 0 ? 0 : min(-ox, bits);
        int c = 0;
        for (int y = y1; y <= y2; ++y) {
            const int Y = y + oy;
            Row r = (Y >= 0 && Y < H) ? nb[Y] : (Row)0;
            r = right < bits ? (Row)(r >> right) : (Row)0;
            r = left < bits ? (Row)(r << left) : (Row)0;
            c += popc((Row)(~(src[y] ^ r) & cols));
        }
        if (c > best) best = c;
    }
    best = __reduce_max_sync(mask, best);
    if (lane == 0) out[p] = (uint16_t)best;
}

size_t similarity_row_bytes(int W) { return W <= 32 ? 4 : 8; }

cudaError_t launch_similarity(const uint8_t* gray, int tile_stride, int W, int H, int V, void* rows,
                              const float2* centers, const int2* pairs, int n, uint16_t* out, cudaStream_t st)
{
    if (n <= 0 || V <= 0) return cudaSuccess;
    const unsigned bin = (unsigned)(((size_t)V * H + 127) / 128);
    if (W <= 32) {
        uint32_t* r = (uint32_t*)rows;
        pm_binarise_kernel<uint32_t><<<bin, 128, 0, st>>>(gray, tile_stride, W, H, V, r);
        if (std::max(W, H) <= 24) pm_similarity_kernel<uint32_t, 16><<<(n + 7) / 8, 128, 0, st>>>(r, W, H, centers, pairs, n, out);
        else pm_similarity_kernel<uint32_t, 32><<<(n + 3) / 4, 128, 0, st>>>(r, W, H, centers, pairs, n, out);
    } else {
        uint64_t* r = (uint64_t*)rows;
        pm_binarise_kernel<uint64_t><<<bin, 128, 0, st>>>(gray, tile_stride, W, H, V, r);
        pm_similarity_kernel<uint64_t, 32><<<(n + 3) / 4, 128, 0, st>>>(r, W, H, centers, pairs, n, out);
    }
    return cudaGetLastError();
}

}  // namespace pfd
