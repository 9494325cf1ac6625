// FP32 instantiation of the resident time steps.
#include "resident.cuh"

namespace aefdtd {
// The kernel with `run` planes per thread.
static ResEntry<float> entry(int run) {
    switch (run) {
        case 2: return resident_entry<float, 2, 512>();
        case 4: return resident_entry<float, 4, 512>();
        case 8: return resident_entry<float, 8, 384>();
        case 12: return resident_entry<float, 12, 256>();
        case 16: return resident_entry<float, 16, 256>();
        case 20: return resident_entry<float, 20, 256>();
        case 24: return resident_entry<float, 24, 256>();
        case 25: return resident_entry<float, 25, 256, true>();
        case 28: return resident_entry<float, 28, 256, true>();
        default: return {};
    }
}
cudaError_t launch_resident(const ResArgs<float> &A, int run, int grid, int smem, cudaStream_t s) {
    return launch_resident_entry(entry(run), A, grid, smem, s);
}
cudaError_t prepare_resident_f32(int run, int most, int smem, int &per_sm) {
    return prepare_resident_entry(entry(run), most, smem, per_sm);
}
}  // namespace aefdtd
