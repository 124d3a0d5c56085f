// The persistent step: SDF geometry, 512 threads (a translation unit per form:
// they compile in parallel).
#include "run_device.cuh"

namespace sdg {
int launch_run_sdf(const RunArgs& A, uint32_t ctas, cudaStream_t s) {
    return A.side[0].c.wallCount ? launchRun<512, false, true>(A, ctas, s) : launchRun<512, false, false>(A, ctas, s);
}
}  // namespace sdg
