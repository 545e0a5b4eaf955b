// fcs_lists.h -- reaction lists of the cell-group kernels, built once per
// mechanism on the host (fcs_capi.cu) and read by fcs_device.cuh.
//
// A cell group evaluates reactions one per thread and then sums their terms
// per species (rates) and per Jacobian element.  Both are lists here:
//   * RxnEv records sorted so that the reactions of one warp take the same
//     branches (a divergent branch costs a whole warp's FP64 instruction on
//     either side);
//   * per sum, its terms in the order the packed reactions are added (the
//     order is part of the result), the sums sorted by length and laid out 32
//     side by side, so that a warp reads its terms as one line and its lanes
//     end together.
#pragma once
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <utility>
#include <vector>

#include "../../include/fcs.h"
#include "fcs_internal.h"

namespace fcs {

constexpr int kTroe = FCS_RXN_TROE_FALLOFF, kSri = FCS_RXN_SRI_FALLOFF;

// Terms of sums, one after another: sum k is val[begin[k] .. begin[k + 1]).
struct Terms {
    std::vector<uint32_t> target, val;
    std::vector<int> begin;
    void start(uint32_t t) {
        target.push_back(t);
        begin.push_back((int)val.size());
    }
    void clear() {
        target.clear();
        val.clear();
        begin.clear();
    }
};

// Sums, 32 to a group: elem[32 g + lane] = target << 16 | terms, the group's
// terms from con[off[g]] on, term k of a lane at off[g] + 32 k + lane, each
// value index << 1 | (1: added, 0: subtracted).  From kLongSum terms on (a
// species' production only: a Jacobian chunk's sums have at most 36,864)
// elem says kLongSum and len[32 g + lane] how many.
struct HostSums {
    std::vector<uint32_t> elem, len;
    std::vector<int> off;
    std::vector<uint32_t> con;
    int groups() const { return (int)off.size(); }

    // t's sums appended, longest first
    void append(const Terms& t) {
        const int n = (int)t.target.size();
        auto begin = [&](int k) { return k < n ? t.begin[k] : (int)t.val.size(); };
        auto length = [&](int k) { return begin(k + 1) - begin(k); };
        int longest = 0;
        for (int k = 0; k < n; k++) longest = std::max(longest, length(k));
        std::vector<int> at(longest + 2, 0), order(n);
        for (int k = 0; k < n; k++) at[longest - length(k) + 1]++;
        for (int l = 0; l <= longest; l++) at[l + 1] += at[l];
        for (int k = 0; k < n; k++) order[at[longest - length(k)]++] = k;
        for (int g = 0; g < n; g += 32) {
            const int most = length(order[g]);
            const size_t base = con.size();
            if (base + 32 * (size_t)most > INT_MAX) throw std::length_error("reaction lists exceed 2^31 terms");
            off.push_back((int)base);
            con.resize(base + 32 * (size_t)most, 0);
            for (int l = 0; l < 32; l++) {
                if (g + l >= n) { elem.push_back(kNoSum); continue; }
                const int k = order[g + l], m = length(k);
                elem.push_back(t.target[k] << 16 | std::min<uint32_t>(m, kLongSum));
                if ((uint32_t)m >= kLongSum) {
                    len.resize(elem.size());
                    len.back() = (uint32_t)m;
                }
                const uint32_t* v = t.val.data() + begin(k);
                for (int q = 0; q < m; q++) con[base + 32 * (size_t)q + l] = v[q];
            }
        }
    }
};

// One chunking of the Jacobian's reactions: chunk c holds the packed
// reactions [c size, (c + 1) size).  Values of a chunk: its net rates q
// (size), dq/dT (size), then d q / d C of every reactant occurrence and, for
// reactions with a reverse rate, product occurrence.  Targets: row << 8 |
// column of the N x N matrix; the species' net production is summed in the
// temperature row, dq/dT in the temperature column.
struct HostChunks {
    int size = 0, values = 0;  // values: most doubles any chunk needs
    std::vector<RxnEv> ev;     // sorted within each chunk, special reactions last
    std::vector<JacChunk> chunk;
    HostSums sums;
};

struct HostLists {
    std::vector<RxnEv> ev;     // all reactions: plain ones, third-body ones, the special block
    int evThird = 0, evSpecial = 0, evTroe = 0, evSri = 0;  // first position of each part
    std::vector<int> tbRow, tbTerm;  // third-body columns by matrix row (DevMech)
    HostSums prod;             // net production per species over q[r]
    HostChunks jac[kJacVariants];
};

// The lists as one block of device memory, each part on a 16-byte boundary.
struct ListBlock {
    struct Sums { size_t elem, off, con, len; };
    struct Jac { size_t ev, chunk; Sums sums; };
    std::vector<char> bytes;
    size_t ev = 0, wiw = 0, RuInvW = 0, tbRow = 0, tbTerm = 0;
    Sums prod{};
    Jac jac[kJacVariants]{};
    template<class T>
    size_t put(const std::vector<T>& v) {
        const size_t o = (bytes.size() + 15) & ~size_t(15);
        bytes.resize(o + std::max<size_t>(1, v.size()) * sizeof(T));
        if (!v.empty()) std::memcpy(bytes.data() + o, v.data(), v.size() * sizeof(T));
        return o;
    }
    Sums put(const HostSums& s) {
        Sums o;
        o.elem = put(s.elem);
        o.off = put(s.off);
        o.con = put(s.con);
        o.len = put(s.len);
        return o;
    }
    static SumLists sums(const char* base, const Sums& o, const HostSums& s) {
        return SumLists{s.groups(), reinterpret_cast<const uint32_t*>(base + o.elem),
                        reinterpret_cast<const int*>(base + o.off), reinterpret_cast<const uint32_t*>(base + o.con),
                        reinterpret_cast<const uint32_t*>(base + o.len)};
    }
};

inline RxnEv make_ev(const RxnInfo& x, int r) {
    RxnEv e{};
    e.A = x.A; e.beta = x.beta; e.Ta = x.Ta;
    for (int q = 0; q < kMaxL; q++) e.sl[q] = x.sl[q];
    for (int q = 0; q < kMaxR; q++) e.sr[q] = x.sr[q];
    e.nl = x.nl; e.nr = x.nr; e.rev = x.rev; e.kind = x.kind;
    e.tb = x.tb; e.plog = x.plog; e.r = r; e.tind = x.tind;
    for (int q = 0; q < x.nl; q++) {
        int f = 0;
        while (x.sl[f] != x.sl[q]) f++;
        e.first |= uint32_t(f) << (2 * q);
    }
    for (int q = 0; q < x.nr; q++) {
        int f = 0;
        while (x.sr[f] != x.sr[q]) f++;
        e.first |= uint32_t(f) << (8 + 3 * q);
    }
    return e;
}

// Fall-off kinds last, each to itself: a Troe and an SRI rate are some 300
// FP64 instructions each, so the kernels give each kind its own warp.
inline int falloff_class(const RxnEv& e) { return e.kind == kTroe ? 1 : e.kind == kSri ? 2 : 0; }

// Reactions that take the same path next to each other, the dearest kind first.
inline void sort_ev(std::vector<RxnEv>& v) {
    std::vector<std::pair<uint64_t, int>> key(v.size());
    for (size_t k = 0; k < v.size(); k++) {
        const RxnEv& e = v[k];
        uint64_t w = falloff_class(e);
        w = w << 1 | (e.plog < 0);
        w = w << 1 | (e.tind != 0);
        w = w << 1 | (e.tb >= 0);
        w = w << 4 | uint64_t(e.rev);
        w = w << 8 | uint64_t(e.nl);
        w = w << 8 | uint64_t(e.nr);
        key[k] = {w << 32 | uint32_t(e.r), (int)k};
    }
    std::sort(key.begin(), key.end());
    std::vector<RxnEv> sorted;
    sorted.reserve(v.size());
    for (const auto& k : key) sorted.push_back(v[k.second]);
    v.swap(sorted);
}

// First position of fall-off class c or above in v
inline int first_of(const std::vector<RxnEv>& v, int c) {
    int k = 0;
    while (k < (int)v.size() && falloff_class(v[k]) < c) k++;
    return k;
}

// Values of a chunk of `size` reactions: their net rates, dq/dT and d q / d C
// of every occurrence that has one; the most any chunk needs.
inline int chunk_values(const std::vector<RxnInfo>& rx, int nr, int size) {
    int most = 0;
    for (int c0 = 0; c0 < nr; c0 += size) {
        int n = 2 * size;
        for (int r = c0; r < std::min(nr, c0 + size); r++) n += rx[r].nl + (rx[r].rev ? rx[r].nr : 0);
        most = std::max(most, n);
    }
    return most;
}

// rx: the packed reactions; inc[i]: (reaction << 1 | product) of species i in
// reaction order; [spBegin, spBegin + nSp): the special block; want: the
// chunkings to build (all when null).
inline HostLists build_lists(int ns, const std::vector<RxnInfo>& rx, int nr, const std::vector<std::vector<int>>& inc,
                             int spBegin, int nSp, const bool* want = nullptr) {
    HostLists H;
    auto special = [&](int r) { return r >= spBegin && r < spBegin + nSp; };
    std::vector<RxnEv> part[3];
    for (int r = 0; r < nr; r++) part[special(r) ? 2 : rx[r].tb >= 0 ? 1 : 0].push_back(make_ev(rx[r], r));
    for (auto& p : part) {
        sort_ev(p);
        H.ev.insert(H.ev.end(), p.begin(), p.end());
    }
    H.evThird = (int)part[0].size();
    H.evSpecial = H.evThird + (int)part[1].size();
    H.evTroe = H.evSpecial + first_of(part[2], 1);
    H.evSri = H.evSpecial + first_of(part[2], 2);
    {
        std::vector<std::vector<int>> rows(ns);
        for (int r = 0; r < nr; r++) {
            if (rx[r].tb < 0) continue;
            for (int q = 0; q < rx[r].nl; q++) rows[rx[r].sl[q]].push_back(rx[r].tb << 1);
            for (int q = 0; q < rx[r].nr; q++) rows[rx[r].sr[q]].push_back(rx[r].tb << 1 | 1);
        }
        for (int i = 0; i < ns; i++) {
            if (rows[i].empty()) continue;
            H.tbRow.push_back(i);
            H.tbRow.push_back((int)H.tbTerm.size());
            H.tbTerm.insert(H.tbTerm.end(), rows[i].begin(), rows[i].end());
        }
        H.tbRow.push_back(0);
        H.tbRow.push_back((int)H.tbTerm.size());
    }
    {
        Terms t;
        for (int i = 0; i < ns; i++) {
            t.start(i);
            t.val.insert(t.val.end(), inc[i].begin(), inc[i].end());
        }
        H.prod.append(t);
    }
    // scratch of a column: its terms in the order they are added, then by row
    Terms t;
    std::vector<uint32_t> w, tc;
    struct Term { int row; uint32_t val; };
    size_t longest = 0;
    for (const auto& l : inc) longest = std::max(longest, l.size());
    std::vector<Term> col(longest * (kMaxL + kMaxR));
    std::vector<int> rows, count(ns, 0), where(ns, 0);
    for (int v = 0; v < kJacVariants; v++) {
        HostChunks& J = H.jac[v];
        J.size = kJacChunk[v];
        J.values = chunk_values(rx, nr, J.size);
        if (want && !want[v]) continue;
        std::vector<size_t> at(ns, 0);  // position in inc[i]
        for (int c0 = 0; c0 < nr; c0 += J.size) {
            const int c1 = std::min(nr, c0 + J.size);
            std::vector<RxnEv> main, sp;
            for (int r = c0; r < c1; r++) (special(r) ? sp : main).push_back(make_ev(rx[r], r));
            sort_ev(main);
            sort_ev(sp);
            const int at0 = (int)(J.ev.size() + main.size());
            JacChunk ch{at0, at0 + first_of(sp, 1), at0 + first_of(sp, 2), J.sums.groups(), 0, {}};
            main.insert(main.end(), sp.begin(), sp.end());
            // value index of every occurrence of the chunk's reactions
            std::vector<int> ent(c1 - c0);
            int n = 2 * J.size;
            for (int r = c0; r < c1; r++) {
                ent[r - c0] = n;
                n += rx[r].nl + (rx[r].rev ? rx[r].nr : 0);
            }
            for (RxnEv& e : main) e.ent = ent[e.r - c0];
            J.ev.insert(J.ev.end(), main.begin(), main.end());
            t.clear();
            for (int j = 0; j < ns; j++) {
                w.clear();
                tc.clear();
                Term* end = col.data();
                int seen[2] = {-1, -1}, occ[2] = {0, 0};  // occurrence of j on the side so far
                for (; at[j] < inc[j].size() && (inc[j][at[j]] >> 1) < c1; at[j]++) {
                    const int r = inc[j][at[j]] >> 1, side = inc[j][at[j]] & 1, l = r - c0;
                    const RxnInfo& x = rx[r];
                    w.push_back(uint32_t(l) << 1 | side);
                    tc.push_back(uint32_t(J.size + l) << 1 | side);
                    if (seen[side] != r) { seen[side] = r; occ[side] = 0; }
                    // the occ-th slot of this side that holds j
                    int slot = 0, k = occ[side]++;
                    const uint8_t* s = side ? x.sr : x.sl;
                    for (;; slot++)
                        if (s[slot] == j && k-- == 0) break;
                    if (side && !x.rev) continue;
                    const uint32_t val = uint32_t(ent[l] + (side ? x.nl : 0) + slot);
                    for (int q = 0; q < x.nl; q++) *end++ = Term{x.sl[q], val << 1};
                    for (int q = 0; q < x.nr; q++) *end++ = Term{x.sr[q], val << 1 | 1};
                }
                if (!w.empty()) {
                    t.start(uint32_t(ns) << 8 | uint32_t(j));
                    t.val.insert(t.val.end(), w.begin(), w.end());
                    t.start(uint32_t(j) << 8 | uint32_t(ns));
                    t.val.insert(t.val.end(), tc.begin(), tc.end());
                }
                rows.clear();
                for (const Term* c = col.data(); c < end; c++)
                    if (count[c->row]++ == 0) rows.push_back(c->row);
                std::sort(rows.begin(), rows.end());
                for (const int i : rows) {
                    t.start(uint32_t(i) << 8 | uint32_t(j));
                    where[i] = (int)t.val.size();
                    t.val.resize(t.val.size() + count[i]);
                    count[i] = 0;
                }
                for (const Term* c = col.data(); c < end; c++) t.val[where[c->row]++] = c->val;
            }
            J.sums.append(t);
            ch.groupEnd = J.sums.groups();
            J.chunk.push_back(ch);
        }
    }
    return H;
}

}  // namespace fcs
