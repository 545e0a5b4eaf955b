// The integration kernel for groups of 256 threads with room for two blocks per
// SM (128 registers), for mechanisms of which two cells fit (make_shape).
#include "fcs_kernels.cuh"

namespace fcs {

cudaError_t launch_integrate_dense256(const LaunchCfg& lc, bool mixed, const DevMech& M, const KOpts& o,
                                      const SlotLayout& L, const CellIO& io, const WorkQueue& q, char* gws,
                                      cudaStream_t st) {
    return mixed ? launch_integrate_t<256, float, 2>(lc, M, o, L, io, q, gws, st)
                 : launch_integrate_t<256, double, 2>(lc, M, o, L, io, q, gws, st);
}

cudaError_t integrate_attributes_dense256(bool mixed, int* maxThreads, int* regs) {
    return mixed ? attrs_t<256, float, 2>(maxThreads, regs) : attrs_t<256, double, 2>(maxThreads, regs);
}

}  // namespace fcs
