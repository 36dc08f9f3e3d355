// nw_range.cuh -- which Needleman-Wunsch calls fit the 16-bit registers of the lane-split
// kernel (sw_split.cu).  Plain C++ without CUDA, so that a CPU test can ask it.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstdlib>

namespace gb2 {

// The floor that stands for cells outside the matrix, and the largest g = -(gap_open +
// gap_extend) at which the floor less a re-centring of 32g stays in 16 bits.
constexpr int32_t kNwFloor = -31000;
constexpr int32_t kNwWrapFree = (32768 + kNwFloor) / 32;

// Whether bands up to maxb of pairs up to qmax x rmax run in lanes = 2^lg lanes of `regs`
// registers.  The right padding needs mismatch >= 2 * (go + ge) and gap terms that are not
// gains, and the score table match - mismatch <= 255.
//
// A register holds H + g * (qi + ri), less 32g every 16 rows.  Every real cell lies in
// [-bottom, top]:
//   matches and mismatches, at most one per base of the shorter sequence;
//   the initial row, go + ri * ge, and the band's own width of gap terms;
//   `drift`, what the rows and columns of the lanes, and the rows since they were last
//   re-centred, put on the register beside that.
// The floor's life: cells left of the reference start and above row 0 start at it.  They
// are computed like the others, with no matches, so a row adds mismatch + 2g to them and
// 16 rows, which the next re-centring takes back but for 16 * mismatch.  Only a diagonal
// move gains, and it brings a cell left of the start one position nearer to it: at most
// maxb of them before the cell is a neighbour of a real one.  So such a cell is at most
//   floor + 18 * (mismatch + 2g) + maxb * max(mismatch, 0)
// at any time, and at least the floor; 500 are to spare below the lowest real cell.
inline bool nw_split_fits(int64_t match, int64_t mismatch, int64_t go, int64_t ge, int64_t maxb,
                          int64_t qmax, int64_t rmax, int regs, int lg)
{
    const int64_t g = -(go + ge);
    if (g < 0 || g > 255 || ge > 0 || mismatch < -2 * g || mismatch > 255 || match < mismatch ||
        match - mismatch > 255)
        return false;
    const int64_t lanes = (int64_t)1 << lg, cols = 2 * (int64_t)regs * lanes;
    const int64_t len = std::min(qmax, rmax) + 1, mp = std::max<int64_t>(match, 0);
    const int64_t drift = g * (36 + 4 * lanes + 2 * maxb + cols);
    const int64_t top = mp * len + drift;
    const int64_t bottom = std::max<int64_t>(-mismatch, 0) * len + g * (maxb + 2) + std::abs(go) -
                           maxb * ge + drift;
    const int64_t climb = 18 * (mp + 2 * g) + maxb * std::max<int64_t>(mismatch, 0);
    return top <= 32000 && bottom + climb + 500 <= -kNwFloor;
}

}  // namespace gb2
