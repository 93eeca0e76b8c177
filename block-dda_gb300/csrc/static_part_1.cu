// Compile-time-plan kernels of complex FP32, part 1 of sparts::kParts.
#include "static_parts.cuh"

namespace bdda {
bool static_z_part1(const MvpGeom& g, float2* t2, int L, const float2* twz, const float2* twzc, const float2* ghat,
                    cudaStream_t st, const int* done, cudaError_t* err) {
  return sparts::dispatch_z<1>(g, t2, L, twz, twzc, ghat, st, done, err);
}
bool static_tile_part1(int pass, const TileArgs& a, cudaError_t* err) { return sparts::dispatch_tile<1>(pass, a, err); }
}  // namespace bdda
