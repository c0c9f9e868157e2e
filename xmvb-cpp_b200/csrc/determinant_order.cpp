// Order of a plan's determinants and the form of its structure reduction.
#include "determinant_order.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <set>
#include <utility>

namespace vbcore {
namespace {

// Determinants with the same alpha-only orbitals (alpha minus beta) pair a set of alpha strings with a
// set of beta strings: for singly ionic structures X + {d} with the complement of X minus {e}, every
// d != e, n - |X| strings of each spin.  Determinants alone in their set (the covalent ones, d = e)
// join a set that holds both their strings.  Sets are cut into blocks; the blocks are taken when they
// are dense enough that the padding of their pair products stays below the gathers they replace (40 %
// filled, ten determinants per block on average) and the list is not tiny.
bool determinant_blocks(const vb_expansion& ex, DeterminantBlocks* out, std::vector<long long>* order) {
    const long long nd = ex.n_determinants;
    if (nd < 512 || ex.n_alpha_strings >= 0xFFFF || ex.n_beta_strings >= 0xFFFF) return false;
    std::map<uint64_t, std::vector<long long>> sets;
    for (long long d = 0; d < nd; ++d)
        sets[ex.alpha_strings[ex.det_alpha[d]] & ~ex.beta_strings[ex.det_beta[d]]].push_back(d);
    if ((long long)sets.size() > nd / 4) {
        // covalent lists: every determinant alone
        long long alone = 0;
        for (const auto& s : sets) alone += s.second.size() == 1;
        if (2 * alone > nd) return false;
    }
    std::vector<std::vector<long long>> groups;
    std::vector<long long> singles;
    for (auto& s : sets) {
        if (s.second.size() == 1)
            singles.push_back(s.second[0]);
        else
            groups.push_back(std::move(s.second));
    }
    std::vector<std::vector<int>> with_alpha(ex.n_alpha_strings);  // groups that hold an alpha string
    std::vector<std::set<int>> betas(groups.size());
    for (size_t g = 0; g < groups.size(); ++g) {
        std::set<int> a;
        for (long long d : groups[g]) {
            a.insert(ex.det_alpha[d]);
            betas[g].insert(ex.det_beta[d]);
        }
        for (int x : a) with_alpha[x].push_back((int)g);
    }
    for (long long d : singles) {
        int best = -1;
        for (int g : with_alpha[ex.det_alpha[d]])
            if (betas[g].count(ex.det_beta[d]) && (best < 0 || groups[g].size() < groups[best].size())) best = g;
        if (best >= 0)
            groups[best].push_back(d);
        else
            groups.push_back({d});
    }
    DeterminantBlocks b;
    std::vector<long long> sorted;
    long long cells = 0;
    int max_a = 0, max_b = 0;
    b.first.push_back(0);
    for (auto& g : groups) {
        std::vector<int> as, bs;
        for (long long d : g) {
            as.push_back(ex.det_alpha[d]);
            bs.push_back(ex.det_beta[d]);
        }
        for (std::vector<int>* v : {&as, &bs}) {
            std::sort(v->begin(), v->end());
            v->erase(std::unique(v->begin(), v->end()), v->end());
        }
        std::map<std::pair<int, int>, long long> at;
        for (long long d : g)
            if (!at.emplace(std::make_pair(ex.det_alpha[d], ex.det_beta[d]), d).second) return false;  // repeated
        // chunks of nearly equal size
        const int ca = ((int)as.size() + 7) / 8, cb = ((int)bs.size() + 7) / 8;
        for (int x = 0; x < ca; ++x)
            for (int y = 0; y < cb; ++y) {
                const int a0 = (int)as.size() * x / ca, a1 = (int)as.size() * (x + 1) / ca;
                const int b0 = (int)bs.size() * y / cb, b1 = (int)bs.size() * (y + 1) / cb;
                BlockStrings block;
                std::memset(&block, 0xFF, sizeof(block));
                int count = 0;
                for (int i = a0; i < a1; ++i)
                    for (int k = b0; k < b1; ++k) {
                        const auto it = at.find({as[i], bs[k]});
                        if (it == at.end()) continue;
                        block.cell[8 * (i - a0) + k - b0] = (unsigned char)count++;
                        sorted.push_back(it->second);
                    }
                if (count == 0) continue;
                block.n_alpha = (unsigned char)(a1 - a0);
                block.n_beta = (unsigned char)(b1 - b0);
                for (int i = a0; i < a1; ++i) block.alpha[i - a0] = (uint16_t)as[i];
                for (int k = b0; k < b1; ++k) block.beta[k - b0] = (uint16_t)bs[k];
                cells += (long long)(a1 - a0) * (b1 - b0);
                max_a = std::max(max_a, a1 - a0);
                max_b = std::max(max_b, b1 - b0);
                b.max_dets = std::max(b.max_dets, count);
                b.strings.push_back(block);
                b.first.push_back((int)sorted.size());
                ++b.n;
            }
    }
    b.max_a = max_a * max_a;
    b.max_b = max_b * max_b;
    if ((long long)sorted.size() != nd || 5 * nd < 2 * cells || nd < 10LL * b.n) return false;
    *out = std::move(b);
    *order = std::move(sorted);
    return true;
}

// Groups of the list in the given order; false where a structure alone has too many rows or repeats a
// determinant.
bool resident_groups(const vb_expansion& ex, const std::vector<long long>& order, const StructureTerms& terms,
                     ResidentGroups* out) {
    ResidentGroups r;
    const int n_str = ex.n_structures;
    const std::vector<long long>&off = terms.off, &det = terms.det;
    const std::vector<double>& coef = terms.coef;
    std::vector<std::pair<uint64_t, uint64_t>> key(n_str);  // doubly occupied, occupied orbitals
    for (int I = 0; I < n_str; ++I)
        if (off[I] < off[I + 1]) {
            const long long d = order[det[off[I]]];
            const uint64_t a = ex.alpha_strings[ex.det_alpha[d]], b = ex.beta_strings[ex.det_beta[d]];
            key[I] = {a & b, a | b};
        }
    r.order.resize(n_str);
    for (int i = 0; i < n_str; ++i) r.order[i] = i;
    std::stable_sort(r.order.begin(), r.order.end(), [&](int x, int y) { return key[x] < key[y]; });
    std::vector<int> owner(ex.n_determinants, -1);  // group that last took the determinant
    r.off.push_back(0);
    for (int i0 = 0; i0 < n_str;) {
        const int g = (int)r.groups.size();
        std::vector<int> used;
        int i1 = i0;
        for (; i1 < n_str && i1 - i0 < kDenseStructures; ++i1) {
            const int I = r.order[i1];
            const size_t before = used.size();
            for (long long t = off[I]; t < off[I + 1]; ++t) {
                if (t > off[I] && det[t] == det[t - 1]) return false;  // one coefficient per structure and determinant
                if (owner[det[t]] != g) {
                    owner[det[t]] = g;
                    used.push_back((int)det[t]);
                }
            }
            if (used.size() > (size_t)kDenseRows) {
                if (i1 == i0) return false;
                used.resize(before);
                break;
            }
        }
        std::sort(used.begin(), used.end());
        for (int i = i0; i < i1; ++i) {
            const int I = r.order[i];
            for (long long t = off[I]; t < off[I + 1]; ++t) {
                r.term_row.push_back(
                    (unsigned short)(std::lower_bound(used.begin(), used.end(), (int)det[t]) - used.begin()));
                r.coef.push_back(coef[t]);
            }
            r.off.push_back((long long)r.coef.size());
        }
        r.groups.push_back({(int)r.rows.size(), (int)used.size(), i0, i1 - i0});
        r.rows.insert(r.rows.end(), used.begin(), used.end());
        r.max_rows = std::max(r.max_rows, (int)used.size());
        i0 = i1;
    }
    *out = std::move(r);
    return true;
}

StructureTerms structure_terms(const vb_expansion& ex, const std::vector<long long>& order) {
    StructureTerms s;
    const long long n_terms = ex.term_offsets[ex.n_determinants];
    s.off.assign(ex.n_structures + 1, 0);
    for (long long t = 0; t < n_terms; ++t) ++s.off[ex.term_structure[t] + 1];
    for (int I = 0; I < ex.n_structures; ++I) s.off[I + 1] += s.off[I];
    s.det.resize(n_terms);
    s.coef.resize(n_terms);
    std::vector<long long> next(s.off.begin(), s.off.end() - 1);
    for (long long i = 0; i < ex.n_determinants; ++i)
        for (long long t = ex.term_offsets[order[i]]; t < ex.term_offsets[order[i] + 1]; ++t) {
            const long long at = next[ex.term_structure[t]]++;
            s.det[at] = i;
            s.coef[at] = ex.term_coefficient[t];
        }
    return s;
}

std::vector<long long> positions(const std::vector<long long>& order) {
    std::vector<long long> pos(order.size());
    for (size_t i = 0; i < order.size(); ++i) pos[order[i]] = (long long)i;
    return pos;
}

// Every determinant at the structure group of the first structure that uses it; within a group's range in
// alpha-major order (the spin-pair records of neighbouring determinant pairs stay neighbours).
std::vector<long long> first_structure_order(const vb_expansion& ex) {
    const long long nd = ex.n_determinants;
    std::vector<long long> order(nd), first(nd, (long long)ex.n_structures);
    for (long long d = 0; d < nd; ++d) {
        order[d] = d;
        for (long long t = ex.term_offsets[d]; t < ex.term_offsets[d + 1]; ++t)
            first[d] = std::min<long long>(first[d], ex.term_structure[t]);
    }
    std::stable_sort(order.begin(), order.end(), [&](long long x, long long y) {
        const long long gx = first[x] / kBandGroup, gy = first[y] / kBandGroup;
        if (gx != gy) return gx < gy;
        if (ex.det_alpha[x] != ex.det_alpha[y]) return ex.det_alpha[x] < ex.det_alpha[y];
        return ex.det_beta[x] < ex.det_beta[y];
    });
    return order;
}

}  // namespace

long long tiled_segments(const vb_expansion& ex, const std::vector<long long>& position) {
    const long long tiles = (ex.n_determinants + kBandTileRows - 1) / kBandTileRows;
    std::vector<long long> keys;
    keys.reserve((size_t)ex.term_offsets[ex.n_determinants]);
    for (long long d = 0; d < ex.n_determinants; ++d)
        for (long long t = ex.term_offsets[d]; t < ex.term_offsets[d + 1]; ++t)
            keys.push_back((long long)(ex.term_structure[t] / kBandGroup) * tiles + position[d] / kBandTileRows);
    std::sort(keys.begin(), keys.end());
    return (long long)(std::unique(keys.begin(), keys.end()) - keys.begin());
}

DeterminantOrder determinant_order(const vb_expansion& ex) {
    DeterminantOrder out;
    const long long nd = ex.n_determinants;
    DeterminantBlocks blocks;
    std::vector<long long> by_block;
    if (ex.n_alpha_electrons > 0 && ex.n_beta_electrons > 0 && determinant_blocks(ex, &blocks, &by_block)) {
        out.terms = structure_terms(ex, by_block);
        bool take = resident_groups(ex, by_block, out.terms, &out.groups);
        if (!take || (long long)out.groups.rows.size() > 4 * nd) {
            // Groups that read every row more than four times hold few structures; they are kept where they
            // still read less than the tiled form, whose groups always hold kBandGroup.  14 orbitals, singly
            // ionic (64 determinants a structure, eight structures a group, rows 4.4 times): 542 ms, tiled
            // 2112 ms in this order and 613 ms in the order below.  With the tiled form a determinant pair is
            // 0.09 ns cheaper by blocks and a segment takes 2.8 ns per 32 columns (same list), so the blocks pay
            // for one more segment per determinant.
            const long long segments = tiled_segments(ex, positions(by_block));
            if (take && (long long)out.groups.rows.size() > kBandTileRows * segments) {
                out.groups = ResidentGroups();
                take = false;
            }
            take = take || segments - tiled_segments(ex, positions(first_structure_order(ex))) < nd;
        }
        if (take) {
            out.order = std::move(by_block);
            out.blocks = std::move(blocks);
            return out;
        }
    }
    std::vector<long long> order = first_structure_order(ex), caller(nd);
    for (long long d = 0; d < nd; ++d) caller[d] = d;
    if (2 * tiled_segments(ex, positions(order)) <= tiled_segments(ex, caller)) out.order = std::move(order);
    out.terms = structure_terms(ex, out.order.empty() ? caller : out.order);
    return out;
}

}  // namespace vbcore
