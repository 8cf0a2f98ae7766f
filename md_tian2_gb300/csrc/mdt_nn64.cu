// mdt_nn64.cu -- the generic HDNNP kernels in FP64 (mdt_nn_kernels.cuh).
#include "mdt_nn_kernels.cuh"

namespace mdt {

cudaError_t launch_nn_fp64(const LaunchCfg &c, const Batch &B, const NNDev &M, const EmtConst &E, const NNScratch &X,
                           const PropParams &P, int ngeta, int nsteps, int mode, bool surrogate) {
    return surrogate ? nn_launch_t<double, true>(c, B, M, E, X, P, ngeta, nsteps, mode)
                     : nn_launch_t<double, false>(c, B, M, E, X, P, ngeta, nsteps, mode);
}

int nn_resident_fp64(size_t sm, bool surrogate) {
    return surrogate ? nn_resident_t<double, true>(sm) : nn_resident_t<double, false>(sm);
}

}  // namespace mdt
