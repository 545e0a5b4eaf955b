// Checks the cell groups' reaction lists (fcs_lists.h) on the host: for random
// mechanisms, every sum taken term by term in the lists' order equals, bit for
// bit, the same sum taken by walking the species' incidence lists in reaction
// order, and every index stays inside what the kernels allocate.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "fcs_lists.h"

using namespace fcs;

static int fail(const char* what, int a, int b) {
    std::printf("FAILED %s %d %d\n", what, a, b);
    return 1;
}

int main(int argc, char** argv) {
    const int ns = std::atoi(argv[1]), nr = std::atoi(argv[2]), seed = std::atoi(argv[3]);
    std::mt19937 rng(seed);
    auto pick = [&](int n) { return int(rng() % unsigned(n)); };
    std::vector<RxnInfo> rx(nr > 0 ? nr : 1);
    std::vector<std::vector<int>> inc(ns);
    const int sp0 = nr / 3, nsp = nr / 5;
    for (int r = 0; r < nr; r++) {
        RxnInfo& x = rx[r];
        x = RxnInfo{};
        x.nl = int8_t(1 + pick(pick(8) ? 3 : kMaxL));
        x.nr = int8_t(1 + pick(pick(8) ? 3 : kMaxR));
        for (int q = 0; q < x.nl; q++) { x.sl[q] = uint8_t(pick(ns)); inc[x.sl[q]].push_back(r << 1); }
        for (int q = 0; q < x.nr; q++) { x.sr[q] = uint8_t(pick(ns)); inc[x.sr[q]].push_back(r << 1 | 1); }
        x.rev = int8_t(pick(3));
        x.tb = pick(5) ? -1 : 0;
        x.plog = pick(7) ? -1 : 0;
    }
    const HostLists H = build_lists(ns, rx, nr, inc, sp0, nsp);
    if ((int)H.ev.size() != nr) return fail("ev", (int)H.ev.size(), nr);
    std::uniform_real_distribution<double> u(0.1, 3.0);
    std::vector<double> q(nr), dq(nr), kf(nr), kr(nr), C(ns);
    for (int r = 0; r < nr; r++) { q[r] = u(rng) - 1.5; dq[r] = u(rng) - 1.5; kf[r] = u(rng); kr[r] = u(rng); }
    for (double& c : C) c = u(rng);
    // the reference: column owners walking the incidence lists
    const int n = ns + 1;
    std::vector<double> J((size_t)n * n, 0.0);
    for (int j = 0; j < ns; j++)
        for (int v : inc[j]) {
            const int r = v >> 1;
            const RxnInfo& x = rx[r];
            double& w = J[(size_t)ns * n + j];
            double& t = J[(size_t)j * n + ns];
            w = v & 1 ? w + q[r] : w - q[r];
            t = v & 1 ? t + dq[r] : t - dq[r];
            if ((v & 1) && !x.rev) continue;
            double d = v & 1 ? -kr[r] : kf[r];
            bool skipped = false;
            for (int k = 0; k < (v & 1 ? x.nr : x.nl); k++) {
                const int s = v & 1 ? x.sr[k] : x.sl[k];
                if (!skipped && s == j) { skipped = true; continue; }
                d *= C[s];
            }
            for (int k = 0; k < x.nl; k++) J[(size_t)x.sl[k] * n + j] -= d;
            for (int k = 0; k < x.nr; k++) J[(size_t)x.sr[k] * n + j] += d;
        }
    auto run = [&](const HostSums& S, int g, int lane, const std::vector<double>& val, double v0, size_t limit) {
        const uint32_t e = S.elem[32 * g + lane];
        for (uint32_t k = 0; k < (e & 0xffff); k++) {
            const uint32_t c = S.con[S.off[g] + 32 * k + lane];
            if ((c >> 1) >= limit) std::exit(fail("index", int(c >> 1), int(limit)));
            v0 += c & 1 ? val[c >> 1] : -val[c >> 1];
        }
        return v0;
    };
    std::vector<int> seen(ns, 0);
    for (int g = 0; g < H.prod.groups(); g++)
        for (int l = 0; l < 32; l++) {
            const uint32_t e = H.prod.elem[32 * g + l];
            if (l && (e & 0xffff) > (H.prod.elem[32 * g] & 0xffff)) return fail("order", g, l);
            if (e >> 16 == 0xffff) continue;
            const int i = int(e >> 16);
            if (i >= ns || seen[i]++) return fail("species", i, g);
            if (run(H.prod, g, l, q, 0.0, nr) != J[(size_t)ns * n + i]) return fail("production", i, g);
        }
    for (int i = 0; i < ns; i++)
        if (!seen[i]) return fail("missing species", i, 0);
    for (int v = 0; v < kJacVariants; v++) {
        const HostChunks& K = H.jac[v];
        std::vector<double> M((size_t)n * n, 0.0), val;
        int ng = 0;
        for (int c = 0, c0 = 0; c0 < nr; c++, c0 += K.size) {
            const int c1 = std::min(nr, c0 + K.size);
            val.assign(K.values, 0.0);
            for (int k = c0; k < c1; k++) {
                const RxnEv& x = K.ev[k];
                if (x.r < c0 || x.r >= c1) return fail("chunk", x.r, c);
                if ((x.r >= sp0 && x.r < sp0 + nsp) != (k >= K.chunk[c].special)) return fail("special", x.r, c);
                val[x.r - c0] = q[x.r];
                val[K.size + x.r - c0] = dq[x.r];
                if (x.ent + x.nl + (x.rev ? x.nr : 0) > K.values) return fail("values", x.ent, K.values);
                for (int a = 0; a < x.nl; a++) {
                    double d = kf[x.r];
                    for (int b = 0; b < x.nl; b++) if (b != int(x.first >> (2 * a) & 3)) d *= C[x.sl[b]];
                    val[x.ent + a] = d;
                }
                for (int a = 0; x.rev && a < x.nr; a++) {
                    double d = -kr[x.r];
                    for (int b = 0; b < x.nr; b++) if (b != int(x.first >> (8 + 3 * a) & 7)) d *= C[x.sr[b]];
                    val[x.ent + x.nl + a] = d;
                }
            }
            if (K.chunk[c].group0 != ng) return fail("groups", c, ng);
            for (; ng < K.chunk[c].groupEnd; ng++)
                for (int l = 0; l < 32; l++) {
                    const uint32_t e = K.sums.elem[32 * ng + l];
                    if (l && (e & 0xffff) > (K.sums.elem[32 * ng] & 0xffff)) return fail("order", ng, l);
                    if (e >> 16 == 0xffff) continue;
                    const int i = int(e >> 24), j = int(e >> 16 & 0xff);
                    if (i > ns || j > ns) return fail("target", i, j);
                    double& m = M[(size_t)i * n + j];
                    m = run(K.sums, ng, l, val, m, val.size());
                }
        }
        if (ng != K.sums.groups()) return fail("all groups", ng, K.sums.groups());
        for (size_t k = 0; k < M.size(); k++)
            if (M[k] != J[k]) return fail("matrix", int(k / n), int(k % n));
    }
    std::printf("ok\n");
    return 0;
}
