// What the host decides from a plan's numbers alone: whether they are sound, and which form of the kernel a product takes.
#pragma once
#include <stdint.h>

namespace agcn {

constexpr int SPMM_ERR_TUPLE = 1;     // malformed tuple (degree, row count or chunk length)
constexpr int SPMM_ERR_ROW = 2;       // rows out of range, overlapping or not ascending
constexpr int SPMM_ERR_LOC = 4;       // nonzero range outside [0, nnz)
constexpr int SPMM_ERR_COL = 8;       // column index outside [0, n_cols)

// Error bits are single words of the host so that blocks can store to them without atomics.
constexpr int PLAN_WORD_ZERO = 0, PLAN_WORD_CARRY = 1, PLAN_WORD_PIECES = 2, PLAN_WORD_FULL = 3;
constexpr int PLAN_WORD_TAIL = PLAN_WORD_PIECES;            // uncut plans, which have no pieces
constexpr int PLAN_WORD_LONGEST = PLAN_WORD_FULL;           // cut plans, which do not count full tuples
constexpr int PLAN_WORD_ERR = 4;      // then one word per SPMM_ERR_* bit
constexpr int PLAN_ERR_BITS = 4;
constexpr int SPMM_ERR_PIECES = 1 << PLAN_ERR_BITS;         // has no word: more pieces than there is room for

// SPMM_ERR_* of what the plan's kernel left in the host's words (most_pieces: INT64_MAX for plans that are not cut).
template <typename Words>
int plan_faults(const Words &words, int64_t most_pieces)
{
    int err = 0;
    for (int k = 0; k < PLAN_ERR_BITS; k++) err |= words[PLAN_WORD_ERR + k] != 0 ? 1 << k : 0;
    return err == 0 && words[PLAN_WORD_PIECES] > most_pieces ? SPMM_ERR_PIECES : err;
}

// What a rule may ask of an uncut plan.
struct UncutPlan {
    int64_t n_units, n_blocks, nnz;
    bool wide;                // 16-byte loads would take the form of five blocks per SM at this width (spmm_wide_form)
    int sm_count;
};

// Rows that cross units are finished inside the launch while it is a few waves of thread blocks (5 per SM), where a second
// launch costs more than blocks that wait for a counter.
inline bool spmm_many_units(int64_t n_units, int sm_count) { return n_units > (int64_t)20 * sm_count; }

// Whether a pass that gathers `width` columns (a multiple of 8) and stores `columns` of them loads rows of X 32 bytes per lane:
// half the load instructions, two rows with each where they have 65 to 128 columns, and more bytes in flight.  It gains where the 16-byte lanes of a slot are not
// all used or, beyond 64 columns, where the gather comes from L2; rows of 64 and 128 columns otherwise keep HBM or the ports
// of L2 as busy 16 bytes at a time.  It never gains up to 32 columns (4-25 % slower), and gains although its forms spill 12 to 24
// bytes of registers (three gathers at four blocks do not: 1-9 % slower).  The additions inside a row of more than 32 nonzeros come in
// another order.  This is the rule on plan and width; rows of X have to begin on 32-byte boundaries as well (spmm_run_prepared), so
// the same values in rows that do and in rows that do not can give other bits.  A product issued in parts has the whole one's.
// Time with / without, B200.  More than 20 units per SM, 250 000 dense rows of 490, 500 000 skewed of 30, 500 000 power law of
// 12, 2.4 M of 25, 1 M of 8: dim 40: .96 .95 .97 .98 .96;  48: .97 .97 .97 .98 .97;  56: .98 1.02 .99 - .99;  64: 1.00 1.01 .96
// 1.00 .98;  72: .88 .94 .93 .95 .94;  80: .85 .96 .93 - .94;  88: .91 1.00 - - -;  96: .92 1.02 1.01 .94 1.02;  112: .95 1.00
// .97 - .98;  128: .98 1.02 1.00 1.02 .98.  Dense, up to 48 columns, not taken up to 40 units per SM, [26] 60 000 of 150, [30] 100 000 of 100, [33] 30 000
// of 400, [34] 40 000 of 300, dims 37, 40, 45, 48: 1.01 1.00 1.02 1.00, 1.00 .99 1.01 1.00, 1.02 1.01 1.02 1.01, 1.00 1.00 1.01 1.00;  taken, [43] 60 000 of 250: .99
// .98 1.00 .99.  (The largest loss that is left: 300 000 power law of 15 [26], dims 40, 45, 48: 1.02 1.02 1.00.)
// Fewer, 60 000 dense of 150, 150 000 power law of 10, 200 000 of 20, 100 000 skewed of 20 (in the form of five blocks): 40:
// .98 .99 1.02 .97;  64: 1.00 .99 1.00 1.05;  72: .96 .96 .96 .93;  80: .96 .97 - .95;  96: .97 .97 - .98;  112: .99 .98 - 1.05;
// 128: .99 .97 .99 1.04.  Dense, not taken up to 11.5 units per SM (the last round of blocks is a good part of them), [6.7] 13 000 of 180, [7.9] 10 000 of
// 250, [9.6] 8 000 of 400, [10.8] 9 000 of 400, dims 72, 88, 96, 112, 128: 1.06 1.05 1.06 1.04 1.03, 1.04 1.04 1.04 1.03 1.02, 1.05 1.05 1.06 1.05 1.03, 1.02 1.03 1.04
// 1.03 1.01;  taken, [14] 20 000 of 250, [18] 60 000 of 100: .97 .98 .98 .98 .98, .96 .95 .96 .98 .98.
// Fewer and not dense: 97 to 128 columns that are no multiple of 4, whose rows of Y are stored element by element, not taken, 90 000 power law of
// 12, 120 000 of 10, 150 000 of 20, 80 000 skewed of 20, 150 000 of 12, dims 103, 109, 119, 127: 1.04 1.07 1.08 1.09, 1.03 1.06 1.07 1.08, 1.01 1.03 1.04 1.05, 1.02 1.05
// 1.07 1.07, 1.01 1.04 1.05 1.08;  such up to 96, taken, the same, dims 69, 77, 85, 93: .95 .98 1.01 1.00, .94 .97 1.00 1.01, .97 .98 .99 .99, .88 .91 .94 .97, .92 .94
// .96 .98.  (Left: 60 000 skewed of 25, dims 112, 120, 128: 1.00 1.01 1.02, and rows of Y that are unaligned by base or stride alone, which the rule does
// not look at, so that bits do not depend on Y.)
inline bool spmm_octets(const UncutPlan &p, int width, int columns)
{
    const bool dense = p.nnz >= 250 * p.n_blocks;
    if (width <= 32) return false;
    if (spmm_many_units(p.n_units, p.sm_count)) {
        if (width <= 48) return !dense || p.n_units > (int64_t)40 * p.sm_count;
        return width > 64 && (width <= 88 || dense);
    }
    if (width <= 64 || (dense && 2 * p.n_units <= (int64_t)23 * p.sm_count)) return false;
    return width <= 96 || (!p.wide && (dense || columns % 4 == 0));
}

// What a rule may ask of a cut plan.
struct CutPlan {
    int64_t n_units, n_rows, nnz;
    int64_t longest;          // nonzeros of the longest row
    int sm_count;
};

// Thread blocks per SM, 3 or 4, of the form that a product of few thread blocks takes at `width` columns; 0: as any product.
//
// Cut plans of more thread blocks than the deep form takes, by how many the SMs hold at once.  Blocks of even graphs take
// equally long, so what counts is that they are one round: up to three per SM eight gathers a lane with 80 registers
// beat seven with 64.  Where there are hub rows, whose full pieces go first, and rows short enough that a piece holds several,
// blocks get lighter towards the end.  Up to four per SM a second round of light blocks then costs little, the less the
// longer the longest row is, compared with the others, and the more rows of X a warp reads at a time: always up to 32 columns,
// where the longest row has 190 times the average up to 64, 290 times beyond (pieces of 128 lose at any width: none).
// 17 to 32 columns, with four gathers at five blocks otherwise, gain with seven at four blocks as far as four per SM, with hub
// rows 6.3.
// Time with three per SM / without, B200, blocks per SM and the longest row as multiple of the average in brackets.
// Up to three, dims 16, 32, 64, 128: even rows 40 000 of 10, 20 000 of 20, 10 000 of 60, 14 000 of 30 [2.8-3.0]: .92 .73 .86 .79, .92
// .73 .87 .81, .94 .74 .85 .83, .83 .75 .88 .82;  power law, 16 384 of 9 [2.8]: .95 .94 .91 .91.
// Three to four, dims 16, 32, 36, 60, 64, 100, 128; taken at all of them: power law, 25 000 of 7 [3.5, 479], 28 000 of 6 [3.5, 544],
// 35 000 of 5 [3.9, 652], 30 000 of 9 [3.8, 464], 25 000 of 12 [3.9, 301], 24 000 of 12 [3.7, 292]: .94 .90 .91 .90 .89 .88 .90, .92 .85 .86 .86 .90 .84 .90, .93
// .90 .86 .86 .90 .84 .90, .96 .90 .90 .89 .90 .86 .90, .96 .91 .89 .88 .94 .95 1.01, .96 .89 .89 .88 .90 .92 .99;  skewed, 20 000 of 11 [3.8, 342],
// 22 000 of 14 [4.0, 295]: .97 .96 .92 .93 .94 .90 .90, .93 .93 .89 .88 .88 .85 .84.
// Taken up to 64: power law, 20 000 of 10 [3.7, 280], 20 000 of 14 [3.5, 217], 18 000 of 12 [4.0, 225], 20 000 of 15 [3.7, 200]: .90 .89 .89 .90 .93 .97
// 1.04, .94 .88 .88 .89 .90 .90 .96, .95 .92 .90 .91 .95 1.04 1.14, .95 .89 .93 .96 1.00 1.03 1.08;  skewed, 20 000 of 16 [4.0, 237]: .94 .91 .89 .88
// .90 .84 .84.
// Taken up to 32: power law, 16 384 of 20 [3.9, 128], 14 000 of 22 [3.7, 103], 18 000 of 18 [3.9, 152], 20 000 of 16 [3.9, 188]: .94 .93 1.01 1.02
// 1.07 1.10 1.16, .95 .94 1.01 1.02 1.07 1.11 1.16, .97 .96 1.04 1.07 1.09 1.13 1.20, .95 .92 .97 1.03 1.07 1.08 1.14;  skewed, 12 000 of 20 [3.8, 114], 16 000 of 22
// [4.0, 138]: .92 .91 .91 .92 .95 1.00 1.05, .95 .89 .92 .94 .99 1.03 1.06.
// Not taken: pieces of 128, power law, 16 384 of 25 [3.8, 103], 18 000 of 22 [3.7, 128]: 1.04 1.05 1.10 1.12 1.15 1.20 1.24, 1.01 1.01 1.09 1.09 1.13 1.17 1.22;
// above four, power law, 25 000 of 14 [4.4]: 1.00 .97 1.06 1.08 1.12 1.17 1.21;  dense, 3 500 of 110, 4 000 of 110 [3.5, 4.0], dims 16, 32, 64, 128: 1.10 1.05
// 1.16 1.22, 1.18 1.09 1.20 1.14.
// 17 to 32 columns, four blocks / five: even, 25 000 of 25, 50 000 of 8 [3.5]: .87, .89;  dense, 7 000 of 100 [4.0]: .88;  power law,
// 16 384 of 25 [3.8], 30 000 of 20 [4.2], 40 000 of 14 [4.6], 50 000 of 10 [5.8]: .90, .88, .89, .92;  skewed, 25 000 of 30 [4.8], 40 000 of 15 [6.3]: .86,
// .90;  not taken: even, 30 000 of 12 [4.2]: 1.23;  dense, 5 000 of 100 [4.6]: 1.14;  skewed, 60 000 of 20 [9.0]: 1.10.
inline int spmm_few_form(const CutPlan &p, int width)
{
    const int64_t sm = p.sm_count;
    const bool uneven = p.longest * p.n_rows > 4 * p.nnz && p.nnz < 32 * p.n_rows;
    if (p.n_units <= 3 * sm) return 3;
    const int64_t times = width <= 32 ? 0 : width <= 64 ? 190 : 290;
    if (uneven && p.n_units <= 4 * sm && p.nnz <= 2700 * sm && p.longest * p.n_rows >= times * p.nnz) return 3;
    return p.n_units <= 4 * sm || (uneven && 10 * p.n_units <= 63 * sm) ? 4 : 0;
}

}  // namespace agcn
