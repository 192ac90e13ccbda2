// Schedule image of the lane-group kernels (kin_group.cuh): a mechanism's RHS, Jacobian,
// elimination and solve work laid out for G lanes per cell. Built on the host from a KinMech
// and staged into shared memory once per CTA.
//
// Every element keeps the reference's operation order (src/sim/kinetics/kin_solver.h:40-139):
//   rates     k_r times its reactants, in equation order
//   f[s]      src[s], then its reactions ascending, one lane per species
//   d(r, p)   k_r times the other reactants, once per (reaction, reactant); -J entry (s, j) = its
//             terms (r, p, e) ascending, one lane per entry
//   LU        pivot by pivot (KIJ): element (i, j) takes its updates in ascending pivot order, as
//             the row-by-row elimination gives them
//   solves    row i takes its columns ascending (L) / descending (U), then 1/U(i,i)
// Lists whose lengths differ (reactant counts, terms per species or entry) are sorted by length
// so that a round of G lanes wastes little; a lane whose list has ended takes a term that changes
// nothing (-0 times the +0 kept behind the last element: acc + -0 is acc, bit for bit).
// Indexes are byte offsets into the cell's arrays, so a lane spends no arithmetic on them.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "../../include/simstack_gpu.h"

namespace sgb {

// Offsets in 32-bit words from the image start.
struct GroupHead {
    uint32_t n, R, ld, pairs;       // species, reactions, dense row stride (odd), (reaction, reactant) pairs
    uint32_t rx;                    // [R] r | s0 << 8 | s1 << 14 | s2 << 20 | count << 26, by count descending
    uint32_t pr;                    // [pairs] r | s0 << 8 | s1 << 14 | count << 26: the factors besides k_r
    uint32_t fround;                // [ceil(n/G)] {first word, terms}: RHS rounds
    uint32_t forder;                // [ceil(n/G) * G] species of the round's lane (kGroupNone: idle)
    uint32_t jrounds, jround;       // [jrounds] {first word, terms}: Jacobian rounds
    uint32_t jdst;                  // [jrounds * G] byte offset in the LU (kGroupNone: idle)
    uint32_t nzero, zero;           // [nzero] byte offsets of the fill-in: -J is zero there
    uint32_t pivot;                 // [n] {rows, row count, tasks, task count}: rows as byte offsets of row i's
                                    // start, tasks as the byte offset of (i, j) | that of row i's start << 16,
                                    // both padded to G with row n, a spare row nothing reads
    uint32_t mask;                  // [n] {columns < i, columns > i} of row i's filled pattern
    uint32_t rr;                    // [R] reactants of reaction r: s0 | s1 << 6 | s2 << 12 | count << 18, by reaction
    uint32_t pfirst;                // [R] position in `pr` of (r, 0); (r, p) follow one another in `pidx`
    uint32_t pidx;                  // [pairs] positions in `pr`, reaction by reaction
    uint32_t words;                 // image size, a multiple of 4
    uint32_t odd_coef;              // some net change is not +-1, +-2, +-4
};
static_assert(sizeof(GroupHead) % 16 == 0, "image alignment");
constexpr uint32_t kGroupNone = 0xffffu;
// The size of the shipped mechanism, which has kernels of its own with n a constant (any mechanism of that
// many species under Rodas3 runs them).
constexpr uint32_t kGroupExact = 17;
// term words: the byte offset of the rate or product in bits 0..15, the coefficient's top 16
// bits as a double (FP64 image) or a float (FP32 images) in bits 16..31
constexpr uint32_t kGroupNoReactant = 0x8000u;   // RHS terms: bit 15, a reaction without reactants
constexpr uint32_t kGroupNoTerm = 0x80000000u;   // coefficient -0

// Element sizes of a lane precision (0 FP64, 1 f32 Delta, 4 mixed double-float): rates, the
// Jacobian's products, the LU.
inline uint32_t group_rate_bytes(uint32_t prec) { return prec == 1 ? 4u : 8u; }
inline uint32_t group_lu_bytes(uint32_t prec) { return prec == 0 ? 8u : 4u; }

// The image for G lanes per cell and a lane precision. False if the record is not what the
// reference's symbolic phase makes (lists out of order, slots that do not agree): the table walk then
// runs as it stands.
inline bool group_image(const KinMech &k, uint32_t G, uint32_t prec, std::vector<uint32_t> *out) {
    const bool wide = prec == 0;
    const uint32_t rsz = group_rate_bytes(prec), lsz = group_lu_bytes(prec);
    const uint32_t n = k.species_count, R = k.reaction_count;
    if (n == 0 || n > KIN_MAX_SPECIES || R > KIN_MAX_REACTIONS || k.nnz > KIN_MAX_NNZ) return false;
    constexpr uint32_t kFree = 0xffffffffu;
    std::vector<uint32_t> slot((size_t)n * n, kFree), cell(k.nnz, kFree);
    auto put = [&](uint32_t i, uint32_t j, uint32_t s) {
        if (s >= k.nnz || j >= n || slot[i * n + j] != kFree || cell[s] != kFree) return false;
        slot[i * n + j] = s;
        cell[s] = i * n + j;
        return true;
    };
    for (uint32_t i = 0; i < n; ++i) {
        if (!put(i, i, k.diag[i])) return false;
        for (uint32_t e = k.lower_begin[i], last = 0; e < k.lower_begin[i + 1]; ++e) {
            const uint32_t j = k.lower[e].col;
            if (j >= i || (e > k.lower_begin[i] && j <= last) || !put(i, j, k.lower[e].index)) return false;
            last = j;
        }
        for (uint32_t e = k.upper_begin[i], last = n; e < k.upper_begin[i + 1]; ++e) {
            const uint32_t j = k.upper[e].col;
            if (j <= i || j >= last || !put(i, j, k.upper[e].index)) return false;
            last = j;
        }
    }
    auto at = [&](uint32_t i, uint32_t j) { return slot[i * n + j] != kFree; };
    // the elimination lists must be the pattern's: row i divides by its lower columns ascending and
    // updates exactly the columns of row kk right of the pivot
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t d = k.div_begin[i];
        for (uint32_t kk = 0; kk < i; ++kk) {
            if (!at(i, kk)) continue;
            if (d >= k.div_begin[i + 1]) return false;
            const KinLuDiv &v = k.lu_div[d++];
            if (v.ik != slot[i * n + kk] || v.kk != slot[kk * n + kk]) return false;
            uint64_t want = 0, got = 0;
            for (uint32_t j = kk + 1; j < n; ++j)
                if (at(kk, j)) want |= 1ull << j;
            for (uint32_t s = v.sub_begin; s < v.sub_end; ++s) {
                const uint32_t ij = cell[k.lu_sub[s].ij], kj = cell[k.lu_sub[s].kj];
                if (ij == kFree || kj == kFree || ij / n != i || kj / n != kk || ij % n != kj % n) return false;
                if (got >> (ij % n) & 1) return false;
                got |= 1ull << (ij % n);
            }
            if (want != got) return false;
        }
        if (d != k.div_begin[i + 1]) return false;
    }
    auto coef = [&](int c, uint32_t *w) {   // the coefficient's top 16 bits; false if it has more
        uint64_t bits;
        if (wide) {
            const double v = c;
            memcpy(&bits, &v, 8);
            *w = (uint32_t)(bits >> 48) << 16;
            return (bits & 0xffffffffffffull) == 0;
        }
        const float v = (float)c;
        uint32_t b;
        memcpy(&b, &v, 4);
        *w = b & 0xffff0000u;
        return (b & 0xffffu) == 0;
    };
    GroupHead h;
    memset(&h, 0, sizeof(h));
    h.n = n;
    h.R = R;
    h.ld = n | 1u;
    std::vector<uint32_t> w(sizeof(GroupHead) / 4, 0u);
    auto align4 = [&]() { while (w.size() & 3) w.push_back(0u); };
    // rates
    std::vector<uint32_t> order(R);
    for (uint32_t r = 0; r < R; ++r) order[r] = r;
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t a, uint32_t b) { return k.reactions[a].reactant_count > k.reactions[b].reactant_count; });
    h.rx = (uint32_t)w.size();
    for (uint32_t r : order) {
        const KinReaction &rx = k.reactions[r];
        uint32_t v = r | (uint32_t)rx.reactant_count << 26;
        for (uint32_t p = 0; p < rx.reactant_count; ++p) v |= (uint32_t)rx.reactant[p] << (8 + 6 * p);
        w.push_back(v);
    }
    // the products k_r prod_{q != p} y_q
    struct Pair { uint32_t r, p, word; };
    std::vector<Pair> pairs;
    for (uint32_t r = 0; r < R; ++r) {
        const KinReaction &rx = k.reactions[r];
        for (uint32_t p = 0; p < rx.reactant_count; ++p) {
            uint32_t v = r, c = 0;
            for (uint32_t q = 0; q < rx.reactant_count; ++q)
                if (q != p) v |= (uint32_t)rx.reactant[q] << (8 + 6 * c++);
            pairs.push_back({r, p, v | c << 26});
        }
    }
    std::stable_sort(pairs.begin(), pairs.end(), [](const Pair &a, const Pair &b) { return (a.word >> 26) > (b.word >> 26); });
    h.pairs = (uint32_t)pairs.size();
    std::vector<uint32_t> pair_at((size_t)R * 3, 0u);
    h.pr = (uint32_t)w.size();
    for (uint32_t q = 0; q < pairs.size(); ++q) {
        w.push_back(pairs[q].word);
        pair_at[pairs[q].r * 3 + pairs[q].p] = q;
    }
    // gather lists: rounds of G lanes, terms of a lane's list one below the other
    struct List { uint32_t dst; std::vector<uint32_t> terms; };
    auto gather = [&](std::vector<List> &lists, uint32_t rounds, uint32_t none, uint32_t *o_round, uint32_t *o_dst) {
        std::stable_sort(lists.begin(), lists.end(), [](const List &a, const List &b) { return a.terms.size() > b.terms.size(); });
        align4();
        *o_round = (uint32_t)w.size();
        w.resize(w.size() + 2 * rounds);
        *o_dst = (uint32_t)w.size();
        for (uint32_t e = 0; e < rounds * G; ++e) w.push_back(e < lists.size() ? lists[e].dst : kGroupNone);
        for (uint32_t q = 0; q < rounds; ++q) {
            const uint32_t len = q * G < lists.size() ? (uint32_t)lists[q * G].terms.size() : 0u;
            w[*o_round + 2 * q] = (uint32_t)w.size();
            w[*o_round + 2 * q + 1] = len;
            for (uint32_t e = 0; e < len; ++e)
                for (uint32_t l = 0; l < G; ++l) {
                    const uint32_t at_ = q * G + l;
                    w.push_back(at_ < lists.size() && e < lists[at_].terms.size() ? lists[at_].terms[e] : none | kGroupNoTerm);
                }
        }
    };
    std::vector<List> rows(n);
    for (uint32_t s = 0; s < n; ++s) rows[s].dst = s;
    for (uint32_t r = 0; r < R; ++r) {
        const KinReaction &rx = k.reactions[r];
        for (uint32_t e = 0; e < rx.net_count; ++e) {
            const int c = rx.net_coef[e];
            uint32_t cw;
            if (!coef(c, &cw)) return false;
            if (c != 1 && c != -1 && c != 2 && c != -2 && c != 4 && c != -4) h.odd_coef = 1;
            rows[rx.net_species[e]].terms.push_back(r * rsz | (rx.reactant_count ? 0u : kGroupNoReactant) | cw);
        }
    }
    gather(rows, (n + G - 1) / G, R * rsz, &h.fround, &h.forder);
    std::vector<List> entries;
    std::vector<uint32_t> entry((size_t)n * n, kFree);
    for (uint32_t r = 0; r < R; ++r) {
        const KinReaction &rx = k.reactions[r];
        for (uint32_t p = 0; p < rx.reactant_count; ++p)
            for (uint32_t e = 0; e < rx.net_count; ++e) {
                const uint32_t c = rx.net_species[e] * n + rx.reactant[p];
                if (slot[c] == kFree || rx.jac_index[p][e] != slot[c]) return false;
                if (entry[c] == kFree) {
                    entry[c] = (uint32_t)entries.size();
                    entries.push_back({(c / n * h.ld + c % n) * lsz, {}});
                }
                uint32_t cw;
                if (!coef(-(int)rx.net_coef[e], &cw)) return false;
                entries[entry[c]].terms.push_back(pair_at[r * 3 + p] * lsz | cw);
            }
    }
    h.jrounds = ((uint32_t)entries.size() + G - 1) / G;
    gather(entries, h.jrounds, h.pairs * lsz, &h.jround, &h.jdst);
    h.zero = (uint32_t)w.size();
    for (uint32_t c = 0; c < n * n; ++c)
        if (slot[c] != kFree && entry[c] == kFree) w.push_back((c / n * h.ld + c % n) * lsz);
    h.nzero = (uint32_t)w.size() - h.zero;
    // elimination
    align4();
    h.pivot = (uint32_t)w.size();
    w.resize(w.size() + 4 * n);
    for (uint32_t q = 0; q < n; ++q) {
        const uint32_t r0 = (uint32_t)w.size();
        for (uint32_t i = q + 1; i < n; ++i)
            if (at(i, q)) w.push_back(i * h.ld * lsz);
        while ((w.size() - r0) % G) w.push_back(n * h.ld * lsz);
        const uint32_t t0 = (uint32_t)w.size();
        for (uint32_t i = q + 1; i < n; ++i)
            for (uint32_t j = q + 1; j < n; ++j)
                if (at(i, q) && at(q, j)) w.push_back((i * h.ld + j) * lsz | (i * h.ld * lsz) << 16);
        while ((w.size() - t0) % G) w.push_back((n * h.ld + n - 1) * lsz | (n * h.ld * lsz) << 16);
        w[h.pivot + 4 * q] = r0;
        w[h.pivot + 4 * q + 1] = t0 - r0;
        w[h.pivot + 4 * q + 2] = t0;
        w[h.pivot + 4 * q + 3] = (uint32_t)w.size() - t0;
    }
    align4();
    h.mask = (uint32_t)w.size();
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t lo = 0, hi = 0;
        for (uint32_t j = 0; j < n; ++j)
            if (j != i && at(i, j)) (j < i ? lo : hi) |= 1u << j;
        w.push_back(lo);
        w.push_back(hi);
    }
    h.rr = (uint32_t)w.size();
    for (uint32_t r = 0; r < R; ++r) {
        const KinReaction &rx = k.reactions[r];
        uint32_t v = (uint32_t)rx.reactant_count << 18;
        for (uint32_t p = 0; p < rx.reactant_count; ++p) v |= (uint32_t)rx.reactant[p] << (6 * p);
        w.push_back(v);
    }
    h.pfirst = (uint32_t)w.size();
    for (uint32_t r = 0, q = 0; r < R; q += k.reactions[r++].reactant_count) w.push_back(q);
    h.pidx = (uint32_t)w.size();
    for (uint32_t r = 0; r < R; ++r)
        for (uint32_t p = 0; p < k.reactions[r].reactant_count; ++p) w.push_back(pair_at[r * 3 + p]);
    for (uint32_t e = 0; e < 8 * G; ++e) w.push_back(0u);   // gathers read up to a batch past a list
    align4();
    h.words = (uint32_t)w.size();
    memcpy(w.data(), &h, sizeof(h));
    out->swap(w);
    return true;
}

// Shared memory of one cell, in elements (double, float, or float pairs), and the stride that puts a
// warp's cells on different banks: 8 lanes of a cell touch rows `ld` (odd) apart.
inline uint32_t group_cell_bytes(const GroupHead &h, uint32_t prec, uint32_t G) {
    const uint32_t elem = group_lu_bytes(prec), banks = 128u / elem;
    const uint32_t lu = (h.n + 1u) * h.ld, products = h.pairs + 1u;
    // FP64 and f32: LU (and its spare row), products, k, rates (one spare each), five species vectors and
    // four stage vectors; mixed: k, rates, products, four species and four stage vectors as float pairs,
    // then the FP32 LU, products and x
    uint32_t words = prec == 4 ? 2u * (h.R + h.R + 1u + h.pairs + 8u * h.n) + lu + products + h.n
                               : lu + products + h.R + h.R + 1u + 9u * h.n;
    words += words & 1u;
    while (words % banks != G % banks) words += 2u;   // G is a multiple of 8
    return words * elem;
}

}   // namespace sgb
