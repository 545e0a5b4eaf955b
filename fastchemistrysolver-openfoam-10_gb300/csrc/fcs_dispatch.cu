// fcs_dispatch.cu -- run-time dispatch over the per-group-size kernel
// instantiations, and the cell classification kernel.
#include "fcs_kernels.cuh"

namespace fcs {

// Treact skip + compaction of the active cells into the work queue
__global__ void classify_kernel(CellIO io, int ns, double Treact, int* order, int* count) {
    const long long nc = io.nCells;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc;
         c += (long long)gridDim.x * blockDim.x) {
        if (io.T[c] > Treact) {
            const int k = atomicAdd(count, 1);
            order[k] = (int)c;
        } else {
            if (io.RR) for (int i = 0; i < ns; i++) io.RR[(size_t)i * nc + c] = 0;
            if (io.status) io.status[c] = FCS_CELL_SKIPPED;
            atomicAdd(reinterpret_cast<unsigned long long*>(&io.stats[ST_SKIPPED]), 1ull);
        }
    }
}

__device__ __forceinline__ int step_bin(double deltaT, double sub) {
    const double steps = deltaT / fmax(sub, 1e-300);
    int b = steps > 1 ? (int)log2(steps) : 0;
    return b < 0 ? 0 : (b >= 32 ? 31 : b);
}

__global__ void classify_bin_kernel(CellIO io, int ns, double Treact, int* bin, int* counters) {
    __shared__ int hist[kQueueBins];
    for (int b = threadIdx.x; b < kQueueBins; b += blockDim.x) hist[b] = 0;
    __syncthreads();
    const long long nc = io.nCells;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc;
         c += (long long)gridDim.x * blockDim.x) {
        if (io.T[c] > Treact) {
            const double deltaT = io.dtPerCell ? io.dtPerCell[c] : io.deltaT;
            const int b = io.attemptsValid ? attempt_bin(io.attempts[c]) : step_bin(deltaT, io.subDt[c]);
            bin[c] = b;
            atomicAdd(&hist[b], 1);
        } else {
            bin[c] = -1;
            if (io.RR) for (int i = 0; i < ns; i++) io.RR[(size_t)i * nc + c] = 0;
            if (io.status) io.status[c] = FCS_CELL_SKIPPED;
            atomicAdd(reinterpret_cast<unsigned long long*>(&io.stats[ST_SKIPPED]), 1ull);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kQueueBins; b += blockDim.x)
        if (hist[b]) atomicAdd(&counters[QC_BINS + b], hist[b]);
}

// Lanes or groups.  A lane takes a cell from its start to its end, so that a
// step of about a cell per lane lasts as long as the dearest cell; the groups
// share the cells out and last as long as all of them together.  So the dearest
// cell's cost times the lanes stands against the sum times the ratio of the two
// rates, 1.7 to 1.9 for 53 and 63 species, 2.4 for 34, 2.2 for 45 with fall-off.
// 54,000 cells of 58,368 lanes: attempts up to 1.25 to 1.4 times their mean, 34 |
// 45 | 53 | 63 species, lanes 1.7 | 3.6 | 3.3 | 4.2 s, groups 2.7 | 5.8 | 4.0 | 5.8; up
// to 2.2 (53) to 4 times, lanes 0.40 | 0.86 | 1.03 | 1.98 s, groups 0.29 | 0.80 | 0.79 |
// 1.07.  Cells all in the lowest bin (a sub-step as long as the step, eight
// attempts at most) say nothing of their spread: groups.
__device__ bool lanes_are_faster(const int* __restrict__ cells, const LaneChoice& choice) {
    float sum = 0, dearest = 0;
    int highest = 0;
    for (int b = 0; b < kQueueBins; b++) {
        if (!cells[b]) continue;
        dearest = exp2f(choice.attemptsValid ? (b + 24.5f) / 8 : b + 0.5f);
        sum += cells[b] * dearest;
        highest = b;
    }
    return highest > 0 && dearest * (float)choice.lanes <= 1.9f * sum;
}

__global__ void queue_kernel(long long nc, const int* __restrict__ bin, int* counters, int* __restrict__ order,
                             const LaneChoice choice) {
    __shared__ int start[kQueueBins];
    if (threadIdx.x == 0) {
        int s = 0;
        for (int b = kQueueBins - 1; b >= 0; b--) {
            start[b] = s;
            s += counters[QC_BINS + b];
        }
        if (blockIdx.x == 0) {
            counters[QC_LEN] = s;
            if (choice.lanes > 0) {
                const bool lanes = lanes_are_faster(counters + QC_BINS, choice);
                counters[QC_LEN_LANES] = lanes ? s : 0;
                counters[QC_LEN_GROUPS] = lanes ? 0 : s;
                choice.stats[ST_LANES] = lanes;
            }
        }
    }
    __syncthreads();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc;
         c += (long long)gridDim.x * blockDim.x) {
        const int b = bin[c];
        if (b >= 0) order[start[b] + atomicAdd(&counters[QC_FILL + b], 1)] = (int)c;
    }
}

cudaError_t launch_classify_binned(const CellIO& io, int ns, double Treact, int* bin, int* counters,
                                   cudaStream_t st) {
    const int block = 256;
    long long blocks = (io.nCells + block - 1) / block;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    classify_bin_kernel<<<(int)blocks, block, 0, st>>>(io, ns, Treact, bin, counters);
    return cudaGetLastError();
}

cudaError_t launch_queue(long long nc, const int* bin, int* counters, int* order, const LaneChoice& choice,
                         cudaStream_t st) {
    const int block = 256;
    long long blocks = (nc + block - 1) / block;
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) blocks = 1;
    queue_kernel<<<(int)blocks, block, 0, st>>>(nc, bin, counters, order, choice);
    return cudaGetLastError();
}

cudaError_t launch_integrate(const LaunchCfg& lc, bool mixed, const DevMech& M, const KOpts& o,
                             const SlotLayout& L, const CellIO& io, const WorkQueue& q, char* gws,
                             cudaStream_t st) {
    switch (lc.group) {
        case 1: return launch_lane_integrate(lc, mixed, M, o, io, q, gws, st);
        case 32: return launch_integrate_g<32>(lc, mixed, M, o, L, io, q, gws, st);
        case 64: return launch_integrate_g<64>(lc, mixed, M, o, L, io, q, gws, st);
        case 128: return launch_integrate_g<128>(lc, mixed, M, o, L, io, q, gws, st);
        case 256:
            return lc.dense ? launch_integrate_dense256(lc, mixed, M, o, L, io, q, gws, st)
                            : launch_integrate_g<256>(lc, mixed, M, o, L, io, q, gws, st);
        case 512: return launch_integrate_g<512>(lc, mixed, M, o, L, io, q, gws, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_jacobian(const LaunchCfg& lc, const DevMech& M, const KOpts& o, const SlotLayout& L,
                            long long nc, const double* p, const double* T, const double* Y, double* out,
                            double* J, char* gws, cudaStream_t st) {
    switch (lc.group) {
        case 32: return launch_jacobian_g<32>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
        case 64: return launch_jacobian_g<64>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
        case 128: return launch_jacobian_g<128>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
        case 256: return launch_jacobian_g<256>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
        case 512: return launch_jacobian_g<512>(lc, M, o, L, nc, p, T, Y, out, J, gws, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t integrate_attributes(int group, bool mixed, int* maxThreads, int* regs) {
    switch (group) {
        case 1: return lane_attributes(mixed, maxThreads, regs);
        case 32: return integrate_attributes_g<32>(mixed, maxThreads, regs);
        case 64: return integrate_attributes_g<64>(mixed, maxThreads, regs);
        case 128: return integrate_attributes_g<128>(mixed, maxThreads, regs);
        case 256: return integrate_attributes_g<256>(mixed, maxThreads, regs);
        case 512: return integrate_attributes_g<512>(mixed, maxThreads, regs);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_classify(const CellIO& io, int ns, double Treact, int* order, int* count,
                            cudaStream_t st) {
    const int block = 256;
    long long blocks = (io.nCells + block - 1) / block;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    classify_kernel<<<(int)blocks, block, 0, st>>>(io, ns, Treact, order, count);
    return cudaGetLastError();
}

}  // namespace fcs
