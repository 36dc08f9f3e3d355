// CPU model of the lane-split Needleman-Wunsch kernel's arithmetic, and the rule by which
// the library admits a call to it (nw_range.cuh), for test_nw_split_range.py.
//
// The model keeps the kernel's registers as it does: G lanes of R registers with a low and a
// high half, rows skewed by lane and half, 16-bit sums that wrap, cells outside the matrix
// computed and never masked after the start, all registers re-centred every 16 steps.
#include <cstdint>
#include <vector>

#include "nw_range.cuh"

namespace {

int16_t wrap(int32_t v) { return (int16_t)(uint16_t)(uint32_t)v; }

int16_t max3(int16_t a, int16_t b, int16_t c) { return std::max(a, std::max(b, c)); }

}  // namespace

extern "C" int nw_fits(int64_t match, int64_t mismatch, int64_t go, int64_t ge, int64_t maxb,
                       int64_t qmax, int64_t rmax, int regs, int lg)
{
    return gb2::nw_split_fits(match, mismatch, go, ge, maxb, qmax, rmax, regs, lg);
}

// Score of q[0, qlen) against r[0, rlen) (both not empty), band b, in 2^lg lanes of R
// registers.  wrapping: re-centre without the limit that keeps the sum in 16 bits (a planted
// mistake).
extern "C" int32_t nw_model(const uint8_t *q, int32_t qlen, const uint8_t *r, int32_t rlen,
                            int32_t match, int32_t mismatch, int32_t go, int32_t ge, int32_t b,
                            int R, int lg, int wrapping)
{
    const int G = 1 << lg;
    const int32_t g = -(go + ge), floor = gb2::kNwFloor;
    const int16_t limit = wrapping || g <= gb2::kNwWrapFree ? INT16_MIN : wrap(floor + 32 * g);
    struct Lane {
        std::vector<int16_t> lo, hi;
        int16_t hl_lo, hl_hi;
    };
    std::vector<Lane> lanes(G);
    int32_t drift = -g * (2 + b);
    auto init = [&](int32_t j) {
        const int32_t ri = j - b;
        if (ri < 0 || j > 2 * b)
            return (int16_t)floor;
        return wrap((ri == 0 ? 0 : go + ri * ge) + drift + g * j);
    };
    for (int l = 0; l < G; ++l) {
        Lane &n = lanes[l];
        n.hl_lo = n.hl_hi = (int16_t)floor;
        for (int h = 0; h < R; ++h) {
            n.lo.push_back(init(2 * R * l + h));
            n.hi.push_back(init(2 * R * l + R + h));
        }
    }
    const int32_t fo = rlen - qlen + b, steps = qlen + 2 * G - 1;
    if (fo < 0 || fo > 2 * b)
        return -1000000;
    auto equal = [&](int32_t row, int32_t j) {
        const int32_t ri = row - b + j;
        return row >= 0 && row < qlen && j <= 2 * b && ri >= 0 && ri < rlen && q[row] == r[ri];
    };
    auto sub = [&](int32_t row, int32_t j) {
        return (equal(row, j) ? match : mismatch) + 2 * g;
    };
    for (int32_t t = 0; t < steps; ++t) {
        if (t > 0 && t % 16 == 0) {
            auto centre = [&](int16_t &v) {
                v = std::max(wrap(std::max(v, limit) - 32 * g), (int16_t)floor);
            };
            for (Lane &n : lanes) {
                for (int h = 0; h < R; ++h) {
                    centre(n.lo[h]);
                    centre(n.hi[h]);
                }
                centre(n.hl_lo);
                centre(n.hl_hi);
            }
            drift -= 32 * g;
        }
        // one register of every lane after another, as a warp runs
        std::vector<int16_t> first_lo(G), first_hi(G);
        for (int h = 0; h < R; ++h) {
            for (int l = 0; l < G; ++l) {
                Lane &n = lanes[l];
                const int32_t c0 = 2 * R * l, row = t - 2 * l;
                const int16_t up_lo = h + 1 < R ? n.lo[h + 1] : first_hi[l];
                const int16_t up_hi =
                    h + 1 < R ? n.hi[h + 1] : l + 1 < G ? first_lo[l + 1] : (int16_t)floor;
                int16_t lo = max3(std::max(wrap(n.lo[h] + sub(row, c0 + h)), up_lo), n.hl_lo,
                                  (int16_t)floor);
                int16_t hi = max3(std::max(wrap(n.hi[h] + sub(row - 1, c0 + R + h)), up_hi),
                                  n.hl_hi, (int16_t)floor);
                if (t < 2 * G) {
                    if (row < 0)
                        lo = n.lo[h];
                    if (row < 1)
                        hi = n.hi[h];
                    if (row == 0 && c0 + h < b)
                        lo = (int16_t)floor;
                    if (row == 1 && c0 + h + R < b)
                        hi = (int16_t)floor;
                }
                n.lo[h] = n.hl_lo = lo;
                n.hi[h] = n.hl_hi = hi;
                if (h == 0) {
                    first_lo[l] = lo;
                    first_hi[l] = hi;
                }
            }
        }
        std::vector<int16_t> in(G);
        for (int l = 0; l < G; ++l)
            in[l] = l == 0 ? (int16_t)floor : lanes[l - 1].hl_hi;
        for (int l = 0; l < G; ++l) {
            Lane &n = lanes[l];
            n.hl_hi = n.hl_lo;
            n.hl_lo = in[l];
            const int32_t row = t - 2 * l, cf = fo - 2 * R * l;
            const int32_t less = drift + g * (fo + 2 * qlen);
            if (row == qlen - 1 && cf >= 0 && cf < R)
                return n.lo[cf] - less;
            if (row == qlen && cf >= R && cf < 2 * R)
                return n.hi[cf - R] - less;
        }
    }
    return INT32_MIN;  // never: the final cell lies in some lane's columns
}
