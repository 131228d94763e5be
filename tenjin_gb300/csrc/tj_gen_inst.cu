// One instance of the general reverse mode's kernels (tj_gen_rev.cuh):
// TJ_INST_M = 1 or 2 materials with a plastic solid, 0: every configuration.
// TJ_INST_D >= 0: the face kernel (of that direction, if TJ_INST_M > 0), -1: the
// update kernel.
#include "tj_gen_rev.cuh"

namespace tj {

#if TJ_INST_M > 0
using GenPT = WithM<DevParamsT, TJ_INST_M, KIND_PLASTIC>;
#else
using GenPT = DevParamsT;
#endif
#if TJ_INST_D < 0
template void gen_upd_rev<GenPT>(const GenPT&, const Fp64Bufs&, const UpdPasses*, int, const GenUpd&, cudaStream_t);
#else
template void gen_flux_rev<GenPT, TJ_INST_M == 0 ? -1 : TJ_INST_D>(const GenPT&, const Fp64Bufs&, const UpdPasses*, int,
                                                                   const GenFlux&, cudaStream_t);
#endif

}  // namespace tj
