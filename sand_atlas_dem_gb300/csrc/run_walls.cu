// The persistent step: mesh geometry between planes, 512 threads (a translation unit per form: they compile in
// parallel).
#include "run_device.cuh"

namespace sdg {
int launch_run_walls(const RunArgs& A, uint32_t ctas, cudaStream_t s) { return launchRun<512, true, true>(A, ctas, s); }
}  // namespace sdg
