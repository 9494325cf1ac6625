// FP64 instantiation of the resident time steps (--fmad=false: the reference rounds every multiply and add).
#include "resident.cuh"

namespace aefdtd {
// The kernel with `run` planes per thread.
static ResEntry<double> entry(int run) {
    switch (run) {
        case 1: return resident_entry<double, 1, 512>();
        case 2: return resident_entry<double, 2, 512>();
        case 4: return resident_entry<double, 4, 384>();
        case 6: return resident_entry<double, 6, 256>();
        case 8: return resident_entry<double, 8, 256>();
        case 10: return resident_entry<double, 10, 256>();
        case 12: return resident_entry<double, 12, 256>();
        case 13: return resident_entry<double, 13, 256, true>();
        case 15: return resident_entry<double, 15, 256, true>();
        default: return {};
    }
}
cudaError_t launch_resident(const ResArgs<double> &A, int run, int grid, int smem, cudaStream_t s) {
    return launch_resident_entry(entry(run), A, grid, smem, s);
}
cudaError_t prepare_resident_f64(int run, int most, int smem, int &per_sm) {
    return prepare_resident_entry(entry(run), most, smem, per_sm);
}
}  // namespace aefdtd
