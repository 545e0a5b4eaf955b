// Prints the cell groups' slots as the kernels take them (host code only: no
// CUDA call), for tests/test_slot_layouts.py: the integrators' with room for a
// Jacobian chunk's values, the evaluations' and the Jacobian's own.
#include <algorithm>
#include <cstdio>

#include "fcs_device.cuh"

int main() {
    using namespace fcs;
    for (int ns : {1, 2, 9, 10, 15, 31, 32, 53, 64, 111, 140, 200, 255})
        for (int nr : {0, 1, 27, 325, 1500, 9000})
            for (int ntb : {0, 3, 40}) {
                // values of a chunk: rates, dq/dT and up to twelve d q / d C a reaction
                for (int values : {2 * 16, 2 * 64 + 64 * 5, 256 * 14}) {
                    for (int form = 0; form < 4; form++) {
                        const int room = std::max(nr, values);
                        const SlotLayout L = make_layout(ns, nr, ntb, form & 1, form & 2, 1, room);
                        std::printf("step %d %d %d %d %d  %d %d %d %d %d %d %d %d %d %d %d %d %d %d %d\n", ns, ntb, form & 1,
                                    form >> 1, room, L.ld, L.offJ64, L.offLU64, L.offLU32, L.offVec, L.offVec32, L.offSp,
                                    L.offInvD, L.offScale, L.offPiv, L.offRx, L.offTb, L.offTable, L.offRed, L.bytes);
                    }
                    const SlotLayout J = make_jacobian_layout(ns, ntb, values);
                    std::printf("jac %d %d %d  %d %d %d %d %d %d %d %d\n", ns, ntb, values, J.ld, J.offJ64, J.offVec, J.offSp,
                                J.offRx, J.offTb, J.offRed, J.bytes);
                }
                const SlotLayout S = make_source_layout(ns, nr, ntb);
                std::printf("source %d %d %d  %d %d %d %d %d %d\n", ns, nr, ntb, S.offVec, S.offSp, S.offRx, S.offTb,
                            S.offRed, S.bytes);
            }
    return 0;
}
