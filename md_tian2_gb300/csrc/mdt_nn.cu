// mdt_nn.cu -- the generic HDNNP kernels in FP32 (mdt_nn_kernels.cuh) and the launchers of both precisions.
#include "mdt_nn_kernels.cuh"

namespace mdt {

cudaError_t launch_nn(const LaunchCfg &c, const Batch &B, const NNDev &M, const EmtConst &E, const NNScratch &X,
                      const PropParams &P, int ngeta, int nsteps, int mode, int precision, bool surrogate) {
    if (precision != 1) return launch_nn_fp64(c, B, M, E, X, P, ngeta, nsteps, mode, surrogate);
    return surrogate ? nn_launch_t<float, true>(c, B, M, E, X, P, ngeta, nsteps, mode)
                     : nn_launch_t<float, false>(c, B, M, E, X, P, ngeta, nsteps, mode);
}

int nn_resident_ctas(const NNDev &M, int max_atoms, int max_beads, int ngeta, int precision, bool surrogate) {
    const size_t sm = nn_total_smem(M, max_atoms, max_beads, ngeta, precision);
    if (precision != 1) return nn_resident_fp64(sm, surrogate);
    return surrogate ? nn_resident_t<float, true>(sm) : nn_resident_t<float, false>(sm);
}

}  // namespace mdt
