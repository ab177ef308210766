// FV stage launches, FP32-bulk.
#include "stage_fv.cuh"

namespace cosenu {

cudaError_t launch_fv_bulk(const tma::StageMaps &m, const StageArgs &a, int stage, int *err,
                           int nblocks, cudaStream_t s, const BatchDev *bd)
{
    switch (stage) {
    case 1: return launch_one<1, double, float>(m, a, err, nblocks, s, bd);
    case 2: return launch_one<2, float, float>(m, a, err, nblocks, s, bd);
    case 3: return launch_one<3, float, float>(m, a, err, nblocks, s, bd);
    case 4: return launch_one<4, float, double>(m, a, err, nblocks, s, bd);
    }
    return cudaErrorInvalidValue;
}

}  // namespace cosenu
