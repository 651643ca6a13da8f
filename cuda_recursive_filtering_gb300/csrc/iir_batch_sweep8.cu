// iir_batch_sweep8.cu — batch kernels on the state sweep for filters of up to 8 sections.
#include "iir_batch_sweep.cuh"
#include "iir_batch_sweep.h"
namespace iirhost {

void bsweep_kernels8(std::vector<BatchSweepKernel>& v) {
    using namespace iirgb;
    // tiles of 4096 samples, as many buffers as shared memory holds with a table each; 1024 for short segments
    v.push_back({8, 128, 32 * (8 + 1 + BSWEEP_COPIERS),
                 reinterpret_cast<const void*>(iir_batch_sweep_kernel<8, 128, 8, 9>), bsweep_smem<8, 128, 9>()});
    v.push_back({8, 32, 32 * (8 + 1 + BSWEEP_COPIERS),
                 reinterpret_cast<const void*>(iir_batch_sweep_kernel<8, 32, 8, 15>), bsweep_smem<8, 32, 15>()});
}

}  // namespace iirhost
