// Host side of the cooperative kernels: the wide-index mechanism image
// (coop.h) built from a finalized Model's symbolic phase or from a
// reference-layout KinMech (the same pattern, slots and scatter lists).
#include <string.h>

#include <algorithm>

#include "coop.h"
#include "mech.h"

namespace sgb {

namespace {
uint32_t align16(size_t v) { return (uint32_t)((v + 15) / 16 * 16); }

// What the image needs, from either source (a Model or a reference-layout KinMech).
struct Desc {
    uint32_t n = 0, R = 0, nnz = 0;
    std::vector<std::vector<uint32_t>> reactants;                   // per reaction, equation order
    std::vector<std::vector<std::pair<uint32_t, int32_t>>> net;     // per reaction, (species, change)
    std::vector<std::vector<std::vector<uint32_t>>> jac_slot;       // [r][p][e] -> compact slot
    std::vector<uint8_t> pattern;                                   // n x n after fill-in
    std::vector<uint32_t> slot;                                     // n x n -> compact slot or ~0u
};

bool build_image(const Desc &d, std::vector<uint8_t> *out);

}   // namespace

bool coop_image(const Model &m, std::vector<uint8_t> *out) {
    if (!m.finalized) return false;
    Desc d;
    d.n = m.n();
    d.R = m.R();
    d.nnz = m.sym.nnz;
    for (const Reaction &rx : m.reactions) {
        d.reactants.push_back(rx.reactants);
        d.net.push_back(rx.net);
        d.jac_slot.push_back(rx.jac_slot);
    }
    d.pattern = m.sym.pattern;
    d.slot = m.sym.slot;
    return build_image(d, out);
}

bool coop_image(const KinMech &k, std::vector<uint8_t> *out) {
    Desc d;
    d.n = k.species_count;
    d.R = k.reaction_count;
    d.nnz = k.nnz;
    const uint32_t n = d.n;
    if (n == 0 || n > KIN_MAX_SPECIES || d.R > KIN_MAX_REACTIONS) return false;
    d.pattern.assign((size_t)n * n, 0);
    d.slot.assign((size_t)n * n, ~0u);
    auto put = [&](uint32_t i, uint32_t j, uint32_t s) {
        d.pattern[(size_t)i * n + j] = 1;
        d.slot[(size_t)i * n + j] = s;
    };
    for (uint32_t i = 0; i < n; ++i) {
        put(i, i, k.diag[i]);
        for (uint32_t e = k.lower_begin[i]; e < k.lower_begin[i + 1]; ++e) put(i, k.lower[e].col, k.lower[e].index);
        for (uint32_t e = k.upper_begin[i]; e < k.upper_begin[i + 1]; ++e) put(i, k.upper[e].col, k.upper[e].index);
    }
    for (uint32_t r = 0; r < d.R; ++r) {
        const KinReaction &rx = k.reactions[r];
        std::vector<uint32_t> re;
        for (uint32_t p = 0; p < rx.reactant_count; ++p) re.push_back(rx.reactant[p]);
        std::vector<std::pair<uint32_t, int32_t>> nt;
        for (uint32_t e = 0; e < rx.net_count; ++e) nt.push_back({rx.net_species[e], (int32_t)rx.net_coef[e]});
        std::vector<std::vector<uint32_t>> js(rx.reactant_count, std::vector<uint32_t>(rx.net_count));
        for (uint32_t p = 0; p < rx.reactant_count; ++p)
            for (uint32_t e = 0; e < rx.net_count; ++e) js[p][e] = rx.jac_index[p][e];
        d.reactants.push_back(re);
        d.net.push_back(nt);
        d.jac_slot.push_back(js);
    }
    return build_image(d, out);
}

namespace {

bool build_image(const Desc &d, std::vector<uint8_t> *out) {
    const uint32_t n = d.n, R = d.R;
    if (n == 0 || n > 256) return false;   // pattern rows are 256-bit masks
    auto pat_at = [&](uint32_t i, uint32_t j) { return d.pattern[(size_t)i * n + j] != 0; };

    CoopMech h;
    memset(&h, 0, sizeof(h));
    h.n = n;
    h.R = R;
    h.ld = n | 1u;
    h.nnz = d.nnz;

    std::vector<uint16_t> reac((size_t)R * 4, 0);
    for (uint32_t r = 0; r < R; ++r) {
        if (d.reactants[r].size() > 3) return false;
        reac[(size_t)r * 4] = (uint16_t)d.reactants[r].size();
        for (size_t p = 0; p < d.reactants[r].size(); ++p) reac[(size_t)r * 4 + 1 + p] = (uint16_t)d.reactants[r][p];
    }
    // RHS terms per species, reactions ascending
    std::vector<std::vector<CoopTerm>> fs(n);
    for (uint32_t r = 0; r < R; ++r)
        for (auto &e : d.net[r]) fs[e.first].push_back({r, (float)e.second});
    for (uint32_t i = 0; i < n; ++i) h.fun_terms += (uint32_t)fs[i].size();
    // Jacobian terms per compact slot, (r, p, e) ascending; entries = slots some reaction scatters into
    std::vector<std::vector<CoopTerm>> js(d.nnz);
    for (uint32_t r = 0; r < R; ++r)
        for (size_t p = 0; p < d.reactants[r].size(); ++p)
            for (size_t e = 0; e < d.net[r].size(); ++e) {
                const uint32_t sl = d.jac_slot[r][p][e];
                if (sl >= d.nnz) return false;
                js[sl].push_back({r | ((uint32_t)p << 24), (float)(-d.net[r][e].second)});
            }
    std::vector<uint32_t> slot_row(d.nnz), slot_col(d.nnz);
    for (uint32_t i = 0; i < n; ++i)
        for (uint32_t j = 0; j < n; ++j) {
            uint32_t s = d.slot[(size_t)i * n + j];
            if (s != ~0u) {
                slot_row[s] = i;
                slot_col[s] = j;
            }
        }
    std::vector<uint32_t> jpos, jrow(n + 1, 0);
    std::vector<uint16_t> jcol;
    for (uint32_t s = 0; s < d.nnz; ++s) {   // slots are row-major, so entries come out sorted by row
        if (js[s].empty()) continue;
        h.jac_terms += (uint32_t)js[s].size();
        jpos.push_back(slot_row[s] * h.ld + slot_col[s]);
        jcol.push_back((uint16_t)slot_col[s]);
        jrow[slot_row[s] + 1]++;
    }
    h.nj = (uint32_t)jpos.size();
    for (uint32_t i = 0; i < n; ++i) jrow[i + 1] += jrow[i];
    std::vector<uint32_t> pat((size_t)n * 8, 0u);
    std::vector<uint16_t> lcnt(n, 0), ucnt(n, 0);
    for (uint32_t i = 0; i < n; ++i)
        for (uint32_t j = 0; j < n; ++j)
            if (pat_at(i, j)) {
                pat[(size_t)i * 8 + (j >> 5)] |= 1u << (j & 31);
                if (i > j) lcnt[j]++;
                if (i < j) ucnt[i]++;
            }
    for (uint32_t k = 0; k < n; ++k) {
        h.l_entries += lcnt[k];
        h.u_entries += ucnt[k];
        h.lu_updates += (uint64_t)lcnt[k] * ucnt[k];
    }
    // pairs and grouped lists
    std::vector<uint32_t> pair, fgrp, fdst, jgrp, jdst;
    std::vector<CoopWide> fterm, jterm;
    std::vector<uint32_t> pair_at((size_t)R * 3, 0u);
    for (uint32_t r = 0; r < R; ++r) {
        const std::vector<uint32_t> &re = d.reactants[r];
        if (R > 0xffffffu) return false;
        for (size_t p = 0; p < re.size(); ++p) {
            uint32_t other = 0, c = 0;
            for (size_t q = 0; q < re.size(); ++q)
                if (q != p) other |= re[q] << (16 * c++);
            pair_at[(size_t)r * 3 + p] = (uint32_t)pair.size() / 2;
            pair.push_back(r | c << 24);
            pair.push_back(other);
        }
    }
    h.pairs = (uint32_t)pair.size() / 2;
    bool wide_ok = true;
    auto wide = [&](uint32_t index, float coef) {
        const double v = coef;
        uint64_t b;
        memcpy(&b, &v, 8);
        wide_ok = wide_ok && (uint32_t)b == 0;
        return CoopWide{index, (uint32_t)(b >> 32)};
    };
    // lists[order[..]] in groups of 32, longest first; dst_words words of `dst` per list
    auto group = [&](const std::vector<std::vector<CoopWide>> &lists, const std::vector<std::vector<uint32_t>> &target,
                     std::vector<uint32_t> *grp, std::vector<uint32_t> *dst, std::vector<CoopWide> *terms) {
        std::vector<uint32_t> order(lists.size());
        for (uint32_t e = 0; e < order.size(); ++e) order[e] = e;
        std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return lists[x].size() > lists[y].size(); });
        const size_t words = target.empty() ? 1 : target[0].size();
        for (size_t g0 = 0; g0 < order.size(); g0 += 32) {
            const size_t len = lists[order[g0]].size();
            grp->push_back((uint32_t)terms->size());
            grp->push_back((uint32_t)len);
            for (size_t l = 0; l < 32; ++l)
                for (size_t q = 0; q < words; ++q) dst->push_back(g0 + l < order.size() ? target[order[g0 + l]][q] : ~0u);
            for (size_t k = 0; k < len; ++k)
                for (size_t l = 0; l < 32; ++l) {
                    const bool on = g0 + l < order.size() && k < lists[order[g0 + l]].size();
                    terms->push_back(on ? lists[order[g0 + l]][k] : CoopWide{~0u, 0u});
                }
        }
    };
    {
        std::vector<std::vector<CoopWide>> fl(n), jl;
        std::vector<std::vector<uint32_t>> ft(n), jt;
        for (uint32_t i = 0; i < n; ++i) {
            ft[i] = {i};
            for (const CoopTerm &t : fs[i]) fl[i].push_back(wide(t.index, t.coef));
        }
        uint32_t e = 0;
        for (uint32_t sl = 0; sl < d.nnz; ++sl) {
            if (js[sl].empty()) continue;
            jt.push_back({jpos[e], e});
            jl.push_back({});
            for (const CoopTerm &t : js[sl]) jl.back().push_back(wide(pair_at[(size_t)(t.index & 0xffffffu) * 3 + (t.index >> 24)], t.coef));
            ++e;
        }
        group(fl, ft, &fgrp, &fdst, &fterm);
        group(jl, jt, &jgrp, &jdst, &jterm);
        if (!wide_ok) return false;   // a net change that is no small integer
    }

    // layout
    size_t off = align16(sizeof(CoopMech));
    auto place = [&](uint32_t *field, size_t bytes) {
        *field = (uint32_t)off;
        off = align16(off + bytes);
    };
    place(&h.off_reac, reac.size() * 2);
    place(&h.off_pair, pair.size() * 4);
    place(&h.off_fgrp, fgrp.size() * 4);
    place(&h.off_fdst, fdst.size() * 4);
    place(&h.off_fterm, fterm.size() * sizeof(CoopWide));
    place(&h.off_jgrp, jgrp.size() * 4);
    place(&h.off_jdst, jdst.size() * 4);
    place(&h.off_jterm, jterm.size() * sizeof(CoopWide));
    place(&h.off_jrow, jrow.size() * 4);
    place(&h.off_jcol, jcol.size() * 2);
    place(&h.off_pat, pat.size() * 4);
    place(&h.off_lcnt, lcnt.size() * 2);
    if (off > 0xffffffffu) return false;
    h.bytes = (uint32_t)off;
    out->assign(off, 0);
    uint8_t *b = out->data();
    memcpy(b, &h, sizeof(h));
    auto put = [&](uint32_t o, const void *src, size_t bytes) {
        if (bytes) memcpy(b + o, src, bytes);
    };
    put(h.off_reac, reac.data(), reac.size() * 2);
    put(h.off_jrow, jrow.data(), jrow.size() * 4);
    put(h.off_jcol, jcol.data(), jcol.size() * 2);
    put(h.off_pat, pat.data(), pat.size() * 4);
    put(h.off_lcnt, lcnt.data(), lcnt.size() * 2);
    put(h.off_pair, pair.data(), pair.size() * 4);
    put(h.off_fgrp, fgrp.data(), fgrp.size() * 4);
    put(h.off_fdst, fdst.data(), fdst.size() * 4);
    put(h.off_fterm, fterm.data(), fterm.size() * sizeof(CoopWide));
    put(h.off_jgrp, jgrp.data(), jgrp.size() * 4);
    put(h.off_jdst, jdst.data(), jdst.size() * 4);
    put(h.off_jterm, jterm.data(), jterm.size() * sizeof(CoopWide));
    return true;
}

}   // namespace

}   // namespace sgb
