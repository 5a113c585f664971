// fuse_kernels.h -- virtual-depth fusion and all-in-focus splat (fuse_kernels.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pfd {

constexpr int kFuseMaxList = 128;                 // neighbour-list entries a reference pixel visits

struct FuseFrame {
    int V, m, ppv, tile_stride;
    const uint8_t* gray;          // [V][tile_stride]
    const uint8_t* bgr;           // [V][ppv][3] or nullptr (gray in all channels)
    const float2* centers;        // [V]
    const float4* plane;          // [V * ppv] normal and disparity
    const int* lists;             // [V][max_list] view ids, -1 = no result
    const int* list_counts;       // [V]
    int max_list;
    float mla_base, min_ref_disp, max_reproj_px, max_rel_vd;
    int min_consistent;
    int raw_w, raw_h;
    unsigned int* winner;         // [raw_h * raw_w]: 1 + sequence number of the last point there, 0 = none
    float* rec;                   // [V * ppv][10]: point, normal, colour, consistent count
    unsigned int* has_rec;        // [V * ppv]: 1 where a point inside the raw frame was recorded
};

constexpr unsigned kFuseNone = 0xFFFFu;           // no consistent pixel

// Work area of the walk over the micro-images [v0, v1) (see fuse_kernels.cu): of the
// whole frame what the micro-images share, of the band what its own walks need.
struct FuseWork {
    const uint8_t* is_ref;        // [V] reference micro-images
    int v0, v1;                   // the band
    int mask_words, chosen_words; // 32-bit words per micro-image mask, per pixel's list mask
    unsigned char* zeroed;        // the part that starts each band at zero: ctl, rev_start, marks
    size_t zeroed_bytes;
    unsigned int* ctl;
    int* rev_start;               // [V + 1] offsets into rev
    int* rev_fill;
    int* changed;                 // [3][V]
    uint32_t* base;               // [V][mask_words] pixels that earlier bands mask
    int* list;                    // [band] micro-images of the round
    int2* rev;                    // [band * max_list] (reference micro-image, list entry) naming a micro-image
    uint32_t* marks;              // [band][max_list][mask_words] pixels of the entry that the micro-image masks
    uint32_t* maybe;              // [band][mask_words] pixels that can become points
    uint32_t* accepted;           // [band][mask_words] pixels that did
    uint32_t* chosen;             // [band * ppv][chosen_words] list entries of the point
    uint16_t* pair_si;            // [band * ppv][max_list] consistent pixel of each entry, or kFuseNone
};
// Lays the work area of bands of n micro-images out in buf and returns its bytes.
size_t fuse_work(const FuseFrame& F, int n, unsigned char* buf, FuseWork& X);
// Micro-images per band for a work area of at most `limit` bytes (1 or more).
int fuse_band(const FuseFrame& F, size_t limit);
// Tests, walk and points, six launches per band, and one between bands; bands in
// ascending order make the sequential walk.  Adds the launches to *launches; err gets
// flag 1 when a device wait gave up.
cudaError_t launch_fuse(const FuseFrame& F, FuseWork X, int band, int* err, cudaStream_t st, unsigned long long* launches);
// The maps from the winning points (outputs zeroed where no point landed).
cudaError_t launch_fuse_maps(const FuseFrame& F, float* vd_map, uint8_t* conf, uint8_t* aif, cudaStream_t st);
// Points in sequence order: counts per block of 1024 sequence numbers, then the
// scatter given each block's exclusive offset.
constexpr int kFuseScanBlock = 1024;
cudaError_t launch_fuse_count(const FuseFrame& F, unsigned int* block_counts, cudaStream_t st);
cudaError_t launch_fuse_compact(const FuseFrame& F, const unsigned int* block_offsets, float* points, cudaStream_t st);

}  // namespace pfd
