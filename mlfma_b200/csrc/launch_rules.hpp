// Rules that fit a launch's tile to a block's shared memory.  A launch shape is
// kept per operator, but a mixed operator runs its kernels in two element sizes
// (8-byte complex float, 16-byte complex double) and a shape that one of them
// was timed with need not fit the other, so each launch asks for its own.
// Plain C++: the rules are checked on the CPU.
#pragma once

#include <algorithm>
#include <cstddef>

namespace mlfma {

// Static shared memory of the kernels below, with room to spare (the many-rhs
// aggregation, whose stencils are static, has its own bound at setup).
constexpr size_t kSmemStatic = 1024;

// Near field of one product.  Blocks of k_near_sym: per_sm per SM, but at least
// four tiles each, so that a small operator leaves room for the kernels beside it.
inline int near_sym_blocks(int tiles, int per_sm, int sms) {
    return std::max(1, std::min(tiles / 4, std::max(1, per_sm) * sms));
}
// Which kernel a product runs: k_near_direct where it is chosen and there are quads,
// except in a mixed operator's solves, which keep the order of k_near_sym's sums.
inline bool near_runs_quads(bool chosen, bool quads, bool solve, bool mixed) {
    return chosen && quads && !(solve && mixed);
}
// Whether a solve's product differs from the operator's own and has its own graph.
inline bool near_solve_differs(bool chosen, bool quads, bool mixed) {
    return near_runs_quads(chosen, quads, false, mixed) != near_runs_quads(chosen, quads, true, mixed);
}

// Aggregation child by child (k_m2m): up to eight children's theta passes.
// elem: bytes of a complex value.
inline size_t m2m_smem(int rows, int child_nph, size_t elem) {
    return static_cast<size_t>(8) * rows * child_nph * 2 * elem;
}
// Parent rows per block: `rows`, halved until the tile fits.
inline int m2m_fit_rows(int rows, int child_nph, size_t elem, size_t limit) {
    while (rows > 1 && m2m_smem(rows, child_nph, elem) > limit) rows /= 2;
    return rows;
}

// Aggregation with the children summed first (k_m2m_sum): the band of child rows
// (bound: all of them), the theta pass's rows, and the stencils (w taps a row).
inline size_t m2m_sum_smem(int rows, int child_nth, int parent_nph, int child_nph, int w, size_t elem) {
    return static_cast<size_t>(child_nth + rows) * child_nph * 2 * elem +
           static_cast<size_t>(rows + parent_nph) * w * (elem / 2 + sizeof(int));
}
// Parent rows per block: `rows`, halved until the tile fits; 0 where not even one
// row does (k_m2m).
inline int m2m_sum_fit_rows(int rows, int child_nth, int parent_nph, int child_nph, int w, size_t elem, size_t limit) {
    while (rows >= 1 && m2m_sum_smem(rows, child_nth, parent_nph, child_nph, w, elem) + kSmemStatic > limit) rows /= 2;
    return rows;
}

// Many-rhs anterpolation (k_l2l_m): `pairs` column pairs and the theta stencils.
inline size_t l2l_m_smem(int pairs, int parent_nth, int child_nth, int w, size_t elem) {
    return static_cast<size_t>(parent_nth) * 2 * pairs * 64 * elem +
           static_cast<size_t>(child_nth) * w * (elem / 2 + 2 * sizeof(int));
}
// Column pairs per block: 2 where asked for and where they fit, else 1 (which
// setup has checked).
inline int l2l_m_fit_pairs(int pairs, int parent_nth, int child_nth, int w, size_t elem, size_t limit) {
    return pairs > 1 && l2l_m_smem(pairs, parent_nth, child_nth, w, elem) + kSmemStatic <= limit ? pairs : 1;
}

}  // namespace mlfma
