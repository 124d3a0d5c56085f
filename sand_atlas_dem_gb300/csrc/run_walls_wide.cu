// The persistent step: mesh geometry between planes, 768 threads (a translation unit per form: they compile in
// parallel).
#include "run_device.cuh"

namespace sdg {
int launch_run_walls_wide(const RunArgs& A, uint32_t ctas, cudaStream_t s) { return launchRun<768, true, true>(A, ctas, s); }
}  // namespace sdg
