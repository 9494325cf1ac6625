// FP32 instantiation of the resident time steps.
#include "resident.cuh"

namespace aefdtd {
cudaError_t launch_resident(const ResArgs<float> &A, int run, int grid, int smem, cudaStream_t s) {
    switch (run) {
        case 2: return launch_resident_run<float, 2, 512>(A, grid, smem, s);
        case 4: return launch_resident_run<float, 4, 512>(A, grid, smem, s);
        case 8: return launch_resident_run<float, 8, 384>(A, grid, smem, s);
        case 12: return launch_resident_run<float, 12, 256>(A, grid, smem, s);
        case 16: return launch_resident_run<float, 16, 256>(A, grid, smem, s);
        case 20: return launch_resident_run<float, 20, 256>(A, grid, smem, s);
        case 24: return launch_resident_run<float, 24, 256>(A, grid, smem, s);
        case 25: return launch_resident_run<float, 25, 256, true>(A, grid, smem, s);
        case 28: return launch_resident_run<float, 28, 256, true>(A, grid, smem, s);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace aefdtd
