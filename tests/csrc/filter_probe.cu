// filter_probe.cu -- test helper: the filter's last launch (launch_filter_apply) on one
// 8x8 micro-image whose pixels all stand to be rejected by their cost, with the words
// "settled" and "a wait gave up" of the work area as given.  Returns how many pixels
// changed (64, or 0 when the launch leaves the state alone), or -1 on a CUDA error.
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include "check_kernels.h"

extern "C" int filter_apply_probe(int settled, int gave_up)
{
    constexpr int N = 64;
    // one allocation: plane, disp, cost, sel, head, disparity, reason, stats, lists, work
    constexpr size_t kBytes = 1 << 14;
    unsigned char* d = nullptr;
    if (cudaMalloc(&d, kBytes) != cudaSuccess || cudaMemset(d, 0, kBytes) != cudaSuccess) return -1;
    size_t at = 0;
    auto take = [&](size_t bytes) { unsigned char* p = d + at; at += (bytes + 255) & ~(size_t)255; return p; };
    pfd::StateDev st = {};
    st.plane = (float4*)take(16 * N);
    st.disp = (float4*)take(16 * N);
    st.cost = (float*)take(4 * N);
    st.sel = (uint32_t*)take(4 * N);
    pfd::CheckFrame F = {};
    F.V = 1; F.W = 8; F.H = 8; F.K = 1; F.tile_stride = 64;
    F.nb_ids = (const int*)take(4);
    F.nb_counts = (const int*)take(4);
    F.baseline_unit = 20.0f;
    pfd::FilterCfg cfg = {};
    cfg.min_good_neighbors = 1;
    pfd::FilterWork X = {};
    X.total = N;
    X.mask_words = 2;
    X.ctl = (unsigned int*)take(32);
    X.mask = (uint32_t*)take(8);
    X.head = (uint32_t*)take(4 * N);
    X.disp = (float*)take(4 * N);
    X.ent = (uint16_t*)take(2 * N);
    uint8_t* reason = take(N);
    unsigned long long* stats = (unsigned long long*)take(64);
    std::vector<float4> plane(N, make_float4(0.f, 0.f, 1.f, 2.f)), after(N);
    std::vector<uint32_t> head(N, 1u);                       // rejected by its cost
    unsigned int ctl[8] = {};
    ctl[pfd::kFilterSettled] = settled ? 1u : 0u;
    ctl[pfd::kFilterGaveUp] = gave_up ? 1u : 0u;
    int changed = -1;
    if (at <= kBytes && cudaMemcpy(st.plane, plane.data(), 16 * N, cudaMemcpyHostToDevice) == cudaSuccess &&
        cudaMemcpy(X.head, head.data(), 4 * N, cudaMemcpyHostToDevice) == cudaSuccess &&
        cudaMemcpy(X.ctl, ctl, sizeof(ctl), cudaMemcpyHostToDevice) == cudaSuccess &&
        pfd::launch_filter_apply(F, cfg, st, X, reason, stats, 0) == cudaSuccess &&
        cudaMemcpy(after.data(), st.plane, 16 * N, cudaMemcpyDeviceToHost) == cudaSuccess) {
        changed = 0;
        for (int i = 0; i < N; ++i) changed += std::memcmp(&plane[i], &after[i], 16) != 0;
    }
    cudaFree(d);
    return changed;
}
