// Instantiations of the cell-group kernels for groups of 32 threads (one
// translation unit per group size so that the build compiles them in parallel).
#include "fcs_kernels.cuh"

namespace fcs {

template<>
cudaError_t launch_integrate_g<32>(const LaunchCfg& lc, bool mixed, const DevMech& M, const KOpts& o,
                                  const SlotLayout& L, const CellIO& io, const WorkQueue& q, char* gws,
                                  cudaStream_t st) {
    return mixed ? launch_integrate_t<32, float>(lc, M, o, L, io, q, gws, st)
                 : launch_integrate_t<32, double>(lc, M, o, L, io, q, gws, st);
}

template<>
cudaError_t launch_jacobian_g<32>(const LaunchCfg& lc, const DevMech& M, const KOpts& o, const SlotLayout& L,
                                 long long nc, const double* p, const double* T, const double* Y, double* out,
                                 double* J, char* gws, cudaStream_t st) {
    return launch_jacobian_t<32>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
}

template<>
cudaError_t integrate_attributes_g<32>(bool mixed, int* maxThreads, int* regs) {
    return mixed ? attrs_t<32, float>(maxThreads, regs) : attrs_t<32, double>(maxThreads, regs);
}

}  // namespace fcs
