// CPU check of the launch rules (launch_rules.hpp): over grids of every size that
// setup accepts and both element sizes, the chosen tile fits the block's shared
// memory wherever the smallest one does, is never larger than asked for, and is
// not given up while it fits.  Run by tests/test_launch_rules.py.
#include "launch_rules.hpp"

#include <cstdio>
using namespace mlfma;

static int bad = 0;
#define CHECK(c)                                                            \
    do {                                                                    \
        if (!(c) && bad++ < 20) std::printf("line %d: %s\n", __LINE__, #c); \
    } while (0)

// The near field's kernel and graph: a solve has its own only where a mixed
// operator's products run quads, so that one chosen grid serves both elsewhere.
static void near_rules() {
    for (bool chosen : {false, true})
        for (bool quads : {false, true})
            for (bool mixed : {false, true}) {
                CHECK(near_runs_quads(chosen, quads, false, mixed) == (chosen && quads));
                CHECK(near_runs_quads(chosen, quads, true, mixed) == (chosen && quads && !mixed));
                CHECK(near_solve_differs(chosen, quads, mixed) == (chosen && quads && mixed));
            }
    for (int tiles : {1, 3, 4, 1000, 100000})
        for (int per_sm : {0, 1, 5}) {
            const int b = near_sym_blocks(tiles, per_sm, 148);
            CHECK(b >= 1 && b <= 148 * (per_sm ? per_sm : 1) && (b == 1 || 4 * b <= tiles));
        }
}

int main() {
    near_rules();
    const size_t limit = 232448;  // opt-in shared memory of a block
    for (size_t elem : {8u, 16u})
        for (int nth = 4; nth <= 160; ++nth) {
            const int nph = 2 * nth;
            // child by child: rows as tuned with either element size
            for (int rows : {1, 2, 3, 4, 8, 16}) {
                const int got = m2m_fit_rows(rows, nph, elem, limit);
                CHECK(got >= 1 && got <= rows);
                CHECK(m2m_smem(got, nph, elem) <= limit || got == 1);
                if (m2m_smem(rows, nph, elem) <= limit) CHECK(got == rows);
            }
            // children summed first: fewer rows before the kernel is given up
            for (int w : {2, 4, 6, 8, 10})
                for (int cth = 4; cth <= nth; ++cth)
                    for (int rows : {1, 2, 4, 8, 16, 32, 64}) {
                        auto fits = [&](int r) {
                            return m2m_sum_smem(r, cth, nph, 2 * cth, w, elem) + kSmemStatic <= limit;
                        };
                        const int got = m2m_sum_fit_rows(rows, cth, nph, 2 * cth, w, elem, limit);
                        CHECK(got <= rows && (got ? fits(got) : !fits(1)));
                        if (got && 2 * got <= rows) CHECK(!fits(2 * got));
                    }
            for (int w : {8, 12, 16, 24, 32})
                for (int cth = 4; cth <= nth; ++cth) {
                    if (l2l_m_smem(1, nth, cth, w, elem) + kSmemStatic > limit) continue;  // refused at setup
                    for (int pairs : {1, 2}) {
                        const int got = l2l_m_fit_pairs(pairs, nth, cth, w, elem, limit);
                        CHECK(got >= 1 && got <= pairs);
                        CHECK(l2l_m_smem(got, nth, cth, w, elem) + kSmemStatic <= limit);
                        if (l2l_m_smem(pairs, nth, cth, w, elem) + kSmemStatic <= limit) CHECK(got == pairs);
                    }
                }
        }
    // the grids of a root of 16 wavelengths, tuned in complex float: two pairs of
    // 58 rows and 16 rows of 68 columns fit 8-byte elements and not 16-byte ones
    CHECK(l2l_m_fit_pairs(2, 58, 34, 12, 8, limit) == 2);
    CHECK(l2l_m_fit_pairs(2, 58, 34, 12, 16, limit) == 1);
    CHECK(m2m_fit_rows(16, 68, 8, limit) == 16);
    CHECK(m2m_fit_rows(16, 68, 16, limit) == 8);
    // and rows of the summed aggregation
    CHECK(m2m_sum_fit_rows(64, 45, 158, 90, 6, 8, limit) == 64);
    CHECK(m2m_sum_fit_rows(64, 45, 158, 90, 6, 16, limit) == 16);
    std::printf(bad ? "%d FAILED\n" : "ALL OK\n", bad);
    return bad != 0;
}
