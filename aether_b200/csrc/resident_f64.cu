// FP64 instantiation of the resident time steps (--fmad=false: the reference rounds every multiply and add).
#include "resident.cuh"

namespace aefdtd {
cudaError_t launch_resident(const ResArgs<double> &A, int run, int grid, int smem, cudaStream_t s) {
    switch (run) {
        case 1: return launch_resident_run<double, 1, 512>(A, grid, smem, s);
        case 2: return launch_resident_run<double, 2, 512>(A, grid, smem, s);
        case 4: return launch_resident_run<double, 4, 384>(A, grid, smem, s);
        case 6: return launch_resident_run<double, 6, 256>(A, grid, smem, s);
        case 8: return launch_resident_run<double, 8, 256>(A, grid, smem, s);
        case 10: return launch_resident_run<double, 10, 256>(A, grid, smem, s);
        case 12: return launch_resident_run<double, 12, 256>(A, grid, smem, s);
        case 13: return launch_resident_run<double, 13, 256, true>(A, grid, smem, s);
        case 15: return launch_resident_run<double, 15, 256, true>(A, grid, smem, s);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace aefdtd
