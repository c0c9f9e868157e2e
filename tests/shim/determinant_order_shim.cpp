// The determinant order and reduction form that a plan would choose for an expansion, without a GPU.
#include "determinant_order.h"

#include <cstdint>

// out: blocks, structure groups of the dense reduction (0: tiled), rows they read together, tiled segments in
// the chosen order and in the caller's.  position [n_det]: of every determinant in the chosen order.
// coefficients [n_str x n_det] (or null): what the groups' terms add up to, by position.
extern "C" int order_of(const vb_expansion* ex, long long* out, long long* position, double* coefficients) {
    const vbcore::DeterminantOrder c = vbcore::determinant_order(*ex);
    const long long nd = ex->n_determinants;
    std::vector<long long> pos(nd), caller(nd);
    for (long long i = 0; i < nd; ++i) {
        caller[i] = i;
        pos[c.order.empty() ? i : c.order[i]] = i;
    }
    for (long long d = 0; d < nd; ++d) position[d] = pos[d];
    out[0] = c.blocks.n;
    out[1] = (long long)c.groups.groups.size();
    out[2] = (long long)c.groups.rows.size();
    out[3] = vbcore::tiled_segments(*ex, pos);
    out[4] = vbcore::tiled_segments(*ex, caller);
    if (coefficients)
        for (const auto& g : c.groups.groups)
            for (int s = g.first; s < g.first + g.structures; ++s)
                for (long long t = c.groups.off[s]; t < c.groups.off[s + 1]; ++t)
                    coefficients[(long long)c.groups.order[s] * nd + c.groups.rows[g.first_row + c.groups.term_row[t]]] +=
                        c.groups.coef[t];
    return 0;
}
