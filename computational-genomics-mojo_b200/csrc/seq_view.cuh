// seq_view.cuh -- one side of a pair list.  Plain C++ without CUDA, so that a CPU test can
// include it.
#pragma once
#include <algorithm>
#include <cstdint>

namespace gb2 {

// Device view of one SequenceBatch side of a pair list.
struct SeqView {
    const uint64_t *packed;  // packed words resident on the device
    const int64_t *offsets;  // word offset of each sequence (SequenceBatch.offsets)
    const int64_t *lengths;  // bases of each sequence (SequenceBatch.lengths)
    int64_t word_base;       // offsets[i] - word_base indexes `packed`
    int64_t n_words;         // words in `packed` (reads are clamped to it)
    // Host only: about how many bases the pairs of the view have together.  Kernels are
    // chosen by the mean length; the words do not tell it, since sequences may share words
    // (all against all), leave gaps, or be more than the view's pairs.
    int64_t bases;
};

// About how many of `bases`, of `count` sequences, belong to m of them.
inline int64_t bases_share(int64_t bases, int64_t m, int64_t count)
{
    return count > 0 ? (int64_t)((double)bases * (double)m / (double)count) : 0;
}

// Pairs [p0, p0 + m) of a view of n.
inline SeqView part_of(SeqView v, int64_t p0, int64_t m, int64_t n)
{
    v.offsets += p0;
    v.lengths += p0;
    v.bases = bases_share(v.bases, m, n);
    return v;
}

// Mean length of a view's n pairs, the longest of which has `longest` bases.
inline double mean_length(const SeqView &v, int64_t n, int64_t longest)
{
    return std::min((double)v.bases / (double)n, (double)longest);
}

}  // namespace gb2
