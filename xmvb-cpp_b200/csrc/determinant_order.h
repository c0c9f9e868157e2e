// Order of a plan's determinants and the form of its structure reduction (host code).
#pragma once

#include <vector>

#include "kernels.h"
#include "vbcore.h"

namespace vbcore {

// Blocks of (at most 8 alpha strings) x (at most 8 beta strings) that the determinant list fills (see
// BlockPairArgs); block h holds determinants first[h] .. first[h + 1] - 1 of the new order.
struct DeterminantBlocks {
    int n = 0, max_a = 0, max_b = 0, max_dets = 0;
    std::vector<int> first;
    std::vector<BlockStrings> strings;
};

// Structure groups whose rows fit shared memory together (BandReduceArgs::groups): up to kDenseStructures
// structures and kDenseRows rows.  Structures with the same doubly occupied and empty orbitals share their
// determinants, so they are taken one after the other: order[i] is the caller's index of structure i, and
// off, coef and term_row list the terms in this order.
struct RowGroup {
    int first_row, rows, first, structures;
};
struct ResidentGroups {
    std::vector<RowGroup> groups;
    std::vector<int> rows, order;
    std::vector<long long> off;
    std::vector<double> coef;
    std::vector<unsigned short> term_row;
    int max_rows = 0;
};

// Terms by structure, positions of their determinants ascending.
struct StructureTerms {
    std::vector<long long> off, det;
    std::vector<double> coef;
};

struct DeterminantOrder {
    std::vector<long long> order;  // determinant of the caller's list at every position; empty: the caller's order
    DeterminantBlocks blocks;      // n == 0: none
    ResidentGroups groups;         // empty: the tiled reduction
    StructureTerms terms;          // in this order
};

// Lists whose determinants fill blocks of (alpha strings) x (beta strings) are ordered by block: the pair
// kernel then works on whole blocks and the band reduction gathers the rows of each structure group.
// Otherwise structures that share few determinants (ionic structures: determinants cluster by occupation
// pattern) leave each structure group of the tiled reduction reading a row tile for a handful of its rows.
// Placing every determinant at the first structure that uses it makes the determinants of consecutive
// structures contiguous; this reorder is taken when it at least halves the (structure group, row tile)
// segments.
DeterminantOrder determinant_order(const vb_expansion& ex);

// (structure group, row tile) segments of the tiled reduction with determinant d at position[d]: what it
// streams for every 32 columns, in tiles of kBandTileRows rows.
long long tiled_segments(const vb_expansion& ex, const std::vector<long long>& position);

}  // namespace vbcore
