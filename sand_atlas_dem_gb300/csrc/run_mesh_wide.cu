// The persistent step: mesh geometry, 768 threads (a translation unit per form: they compile in
// parallel).
#include "run_device.cuh"

namespace sdg {
int launch_run_mesh_wide(const RunArgs& A, uint32_t ctas, cudaStream_t s) { return launchRun<768, true, false>(A, ctas, s); }
}  // namespace sdg
