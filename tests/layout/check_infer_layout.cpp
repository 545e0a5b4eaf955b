// Checks on the host who writes which bytes of the inference kernel's
// activations (fcs_infer_layout.h): what a warp stages of the last layer's
// outputs and what its neighbour writes as the next tile's input share no byte.
#include <cstdio>
#include <vector>

#include "fcs_infer_layout.h"

using namespace fcs;

int main() {
    // owner[b]: 1 + the warp whose next input covers byte b
    std::vector<int> owner(4 * kActChunkBytes, 0);
    for (int q = 0; q < 4; q++)
        for (int part = 0; part < 2; part++)
            for (int r = 0; r < 16; r++)
                for (int k = 0; k < 256; k++)
                    for (int b = 0; b < 2; b++) {
                        int& o = owner[act_offset(input_row(q, part) + r, k) + b];
                        if (o) return std::printf("input byte written twice: %d %d %d %d\n", q, part, r, k), 1;
                        o = 1 + 2 * q + part;
                    }
    for (int q = 0; q < 4; q++)
        for (int part = 0; part < 2; part++) {
            std::vector<int> used(owner.size(), 0);
            for (int u = 0; u < 16; u++) {
                unsigned banks = 0;
                for (int r = 0; r < 32; r++) {
                    const int at = stage_offset(q, part) + 4 * stage_index(32 * q + r, u);
                    banks |= 1u << (at / 4 % 32);
                    if (at % 4 || at < 0 || at + 4 > (int)owner.size()) return std::printf("offset %d\n", at), 1;
                    for (int b = 0; b < 4; b++) {
                        if (used[at + b]++) return std::printf("staged twice: %d %d %d %d\n", q, part, r, u), 1;
                        // every network has at least 128 input columns (padding included)
                        if (at + b >= 2 * kActChunkBytes || owner[at + b] != 1 + 2 * q + part)
                            return std::printf("not its own: %d %d %d %d\n", q, part, r, u), 1;
                    }
                }
                if (banks != 0xffffffffu) return std::printf("bank conflict: %d %d %d\n", q, part, u), 1;
            }
            for (int r = 0; r < 32; r += 2) {  // the stores' reads: 16 columns of two rows
                unsigned banks = 0;
                for (int u = 0; u < 32; u++)
                    banks |= 1u << ((stage_offset(q, part) / 4 + stage_index(r + (u >> 4), u & 15)) % 32);
                if (banks != 0xffffffffu) return std::printf("bank conflict in the reads: %d %d %d\n", q, part, r), 1;
            }
        }
    std::printf("ok\n");
    return 0;
}
