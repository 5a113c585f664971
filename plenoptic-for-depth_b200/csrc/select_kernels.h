// select_kernels.h -- micro-image similarity for the neighbour selection (select_kernels.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pfd {

// out[p] = MeasureSimilarity(micro-image pairs[p].x, micro-image pairs[p].y):
// gray [V][tile_stride] (W x H dense), centres [V].
// rows: V * H words of similarity_row_bytes(W) for the binarised micro-images (two
// launches).
size_t similarity_row_bytes(int W);
cudaError_t launch_similarity(const uint8_t* gray, int tile_stride, int W, int H, int V, void* rows,
                              const float2* centers, const int2* pairs, int n, uint16_t* out, cudaStream_t st);

}  // namespace pfd
