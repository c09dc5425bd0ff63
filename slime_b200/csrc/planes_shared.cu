// planes_shared.cu -- the bit-plane band kernels of shared LCG (planes.cuh).
#include "planes.cuh"

namespace slime {

cudaError_t run_planes_shared(int joined, const BandArgs& one, const BandArgs* args, const int64_t* prefix,
                           int32_t nsearch, unsigned long long* head, int grid, cudaStream_t s) {
    return run_mode<kModeShared>(joined, one, args, prefix, nsearch, head, grid, s);
}

}  // namespace slime
