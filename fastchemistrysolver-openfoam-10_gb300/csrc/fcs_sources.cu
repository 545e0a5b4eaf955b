// Per-cell evaluations without a matrix: right-hand side, source terms with
// heat release, chemical time scale.  One cell group per cell.
//
// The FP64 pipe bounds them (16 to 19 SM cycles per warp instruction, 723 of
// them in a right-hand side of 53 species), once enough warps hide the latency
// of the exponentials and of the mechanism's records.  In the integrator's slot
// (matrix, twelve vectors) shared memory held an SM to 6 cells of 53 species or
// 2 of 111; a slot of its own and 80 registers let 24 warps reside.  rates() and
// tc() of 65,536 cells: 53 species 5.99 -> 5.20 ms, 111 species 23.2 -> 10.0 ms.
#include <algorithm>

#include "fcs_device.cuh"
#include "fcs_launch.h"

namespace fcs {

constexpr int kSourceRegs = 80;    // 128 (as compiled without a bound): 5.48 ms, 64: 5.18 with spills for 32 threads

template<int G>
__global__ void __launch_bounds__(G == 32 ? 32 * kSourceCells32 : G, 65536 / kSourceRegs / (G == 32 ? 32 * kSourceCells32 : G))
source_kernel(const DevMech M, const SlotLayout L, long long nc, const double* __restrict__ p,
              const double* __restrict__ T, const double* __restrict__ rho, const double* __restrict__ Y,
              double* __restrict__ out, double* __restrict__ Qdot, SourceMode mode, char* __restrict__ gws) {
    extern __shared__ __align__(16) char smem[];
    Grp<G> g;
    g.rank = threadIdx.x % G;
    const int gidInBlock = threadIdx.x / G;
    const int groupsPerBlock = blockDim.x / G;
    const long long c = (long long)blockIdx.x * groupsPerBlock + gidInBlock;
    char* base = gws ? gws + (size_t)c * L.bytes : smem + (size_t)gidInBlock * L.bytes;
    const Slot<double> s = make_slot<double>(base, L, M);
    if (c >= nc) return;  // whole group exits together
    const int ns = M.ns;
    double* y = s.v(0);
    double* f = s.v(1);
    for (int i = g.rank; i < ns; i += G) y[i] = Y[(size_t)i * nc + c];
    if (g.rank == 0) {
        y[ns] = T[c];
        s.red[37] = M.nPlog ? log(p[c]) : 0.0;
    }
    g.sync();
    if (mode == SRC_TC) {
        const double tc = tc_eval<G, double>(g, M, s, p[c], T[c], rho[c], y);
        if (g.rank == 0) out[c] = tc;
        return;
    }
    if (mode == SRC_RHS) {
        rhs_eval<G, double>(g, M, s, p[c], y, f, 1);
    } else {
        const double qd = rates_eval<G, double>(g, M, s, p[c], T[c], rho[c], y, f);
        if (Qdot && g.rank == 0) Qdot[c] = qd;
    }
    g.sync();
    const int nout = mode == SRC_RHS ? M.n : ns;
    for (int i = g.rank; i < nout; i += G) out[(size_t)i * nc + c] = f[i];
}

template<int G>
static cudaError_t launch_sources_g(const LaunchCfg& lc, const DevMech& M, const SlotLayout& L, long long nc,
                                    const double* p, const double* T, const double* rho, const double* Y,
                                    double* out, double* Qdot, SourceMode mode, char* gws, cudaStream_t st) {
    auto k = source_kernel<G>;
    const size_t sm = gws ? 0 : (size_t)L.bytes * (lc.block / G);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    k<<<lc.grid, lc.block, sm, st>>>(M, L, nc, p, T, rho, Y, out, Qdot, mode, gws);
    return cudaGetLastError();
}

cudaError_t launch_sources(const LaunchCfg& lc, const DevMech& M, const SlotLayout& L, long long nc,
                           const double* p, const double* T, const double* rho, const double* Y, double* out,
                           double* Qdot, SourceMode mode, char* gws, cudaStream_t st) {
    switch (lc.group) {
        case 32: return launch_sources_g<32>(lc, M, L, nc, p, T, rho, Y, out, Qdot, mode, gws, st);
        case 64: return launch_sources_g<64>(lc, M, L, nc, p, T, rho, Y, out, Qdot, mode, gws, st);
        case 128: return launch_sources_g<128>(lc, M, L, nc, p, T, rho, Y, out, Qdot, mode, gws, st);
        case 256: return launch_sources_g<256>(lc, M, L, nc, p, T, rho, Y, out, Qdot, mode, gws, st);
        case 512: return launch_sources_g<512>(lc, M, L, nc, p, T, rho, Y, out, Qdot, mode, gws, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace fcs
