// sw_split.cu -- banded Smith-Waterman and Needleman-Wunsch for any band, with
// one pair's band row split over G lanes and two cells per 32-bit register.
//
// Computes smith_waterman_banded (genomics/cpu/align_cpu.mojo:229-309) and
// needleman_wunsch_banded (:312-377, band rows sized as its indexing intends)
// bit-exactly.  Band coordinates, recurrence and the E' scaling are those of
// sw_kernels.cu: row qi, column j in [0, 2b], ri = qi - b + j; cell (qi, j)
// reads diag (qi-1, j), up (qi-1, j+1), left (qi, j-1).
//
// Split.  G lanes (a power of two, 1..32) own a pair; lane l keeps columns
// [2Rl, 2Rl + 2R) in R registers of two 16-bit halves: column 2Rl + h in the
// low half of register h, column 2Rl + R + h in its high half.  At step t lane
// l runs row t' = t - 2l in the low halves and row t' - 1 in the high halves,
// so the cells of a register, and of two lanes, are never each other's
// neighbours within a step:
//   left of h = 0   low: the previous lane's last high half (row t', its last
//                   step); high: this lane's last low half (row t'-1)
//   up of h = R-1   low: this lane's first high half (row t'-1, earlier in the
//                   step); high: the next lane's first low half (row t'-2, the
//                   same step), one shuffle started after register 0.
// A pair's rows then need 2 shuffles per step and about R + 2G registers'
// worth of latency, whatever the band: the kernel with one thread per pair
// keeps 2b+1 columns on one thread, which leaves 8 warps per SM for band 128
// and makes the longest pair of a batch its critical path.
//
// Any band in a fixed register count.  2RG >= 2b+1 columns are computed; those
// past 2b never match.  With gap costs g = -(go+ge) >= -mismatch and ge <= 0 they
// change nothing: a path that leaves column 2b to the right by k columns and
// comes back pays at least -ge per column out (E) and g per column back, and
// each way back advances one row, while staying on column 2b costs at most
// -mismatch per row.  So H at column 2b is the same with or without them, E at
// column 2b only feeds columns past it, and a column past 2b never exceeds the
// real cell its value came from, which precedes it in row-major order (the
// first maximum is a real cell).  The same holds for rows past the query end
// and cells past the reference end when they never match, and cells left of
// the reference start or above row 0 are zero when they never match.  One mask
// of equality bits per 16 columns is therefore all the boundary handling: the
// step has no masked variant.  Needleman-Wunsch needs mismatch >= 2(go+ge) for
// the same argument, and its cells left of the reference start sit at a floor
// below every real value: they are computed too, and nw_range.cuh shows how far they
// rise.
//
// Scores of any length in 16 bits (Smith-Waterman).  Registers hold H - base
// with base per pair, and the maximum is found by keys (H - base) * 8 + tag, so
// H - base stays in [0, 4094].  Every 16 steps the pair's largest value M is
// checked and base moved.  Floor: every cell is at least M - S with
// S = (2RG + 2G) * (match - mismatch + g): D = 2RG rows up, some cell has at
// least M - D * match, and from it every cell of the row is reached with D
// diagonal or up moves and at most 2RG left moves.  M is kept at or above
// S + 16 * -mismatch while base > 0, so the floor at H = base never binds.
// Needleman-Wunsch: registers hold H + g * (qi + ri) less 2g per row (the up and
// left moves then add nothing: two DPX instructions per two cells), re-centred
// every 16 steps; the host checks that the values fit (nw_range.cuh).
//
// What bounds it: instructions, which issue at about 0.65 per cycle and scheduler (see
// sw_kernels.cu), 5.5 per register of two cells and 0.5 for its substitution term, one
// 16-byte load of the score table per four registers (NW: 2 and 0.5); at R = 33 a row of
// 66 columns takes 500 cycles.  Short batches are bound by the chain from register to
// register: one warp per scheduler takes 19 R + 150 cycles per row.  256 threads a block,
// two blocks per SM: each block's table takes 64 KB.  (With 16-bit sums kept off the chain,
// max(H_diag + sub, E', H_left) - g, the chain is 15 R + 207 but full batches take 5-9%
// longer: the mixed bands below 1.50 against 1.38 ms.)
// Measured (ms, before: the register kernels of one thread per pair or 2-8 lanes in
// int32, and for other bands the literal kernel with int64 rows in memory; then this
// kernel with a logic op and a high product per register in place of the table):
//   Smith-Waterman, 100,000 pairs of 100-300 bp, band 40       57.9 -> 0.67 -> 0.57
//   50,000 pairs of 100-2,000 bp, bands 16/32/64/128 per pair  5.66 -> 1.73 -> 1.22
//   4,000 pairs of 2-10 kbp, band 128                          13.5 -> 2.84 -> 2.56
//   Needleman-Wunsch, 20,000 pairs of 100-1,000 bp, band 64    46.7 -> 0.46 -> 0.36
//   500,000 reads, band 32                                     2.44 -> 1.38 -> 1.19
// The one-thread kernel stays for short reads of bands 16 and 32 in large batches: its
// row of 33 registers takes 425 cycles against 500 and its pairs need no start
// (400,000 reads, band 32: 0.72 against 0.89 ms); split_choose compares both.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "gb2_internal.cuh"
#include "nw_range.cuh"

namespace gb2 {
namespace {

constexpr uint32_t kSent = 0xC000u;          // -16384: start of the E chain
constexpr int32_t kNwNeg = -1000000;

struct SplitConsts {
    uint32_t x4, x8, x64k, half, one;
    uint32_t dm;      // match - mismatch
    uint32_t sub2;    // mismatch + g (Smith-Waterman) or + 2g, both halves
    uint32_t neg_g2;  // -g in both halves, mod 2^32
    uint32_t ge2;     // ge in both halves
    uint32_t ng2;     // g in both halves
    int32_t go, ge, g;
};

__device__ __forceinline__ uint32_t mad_hi(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// 16-base word k of a sequence of len bases at `w`, clamped into the sequence's own
// words (words outside it are masked by the equality mask).
__device__ __forceinline__ uint32_t word16(const uint32_t *w, int32_t len, int32_t k)
{
    const int32_t last = (((len + 31) >> 5) << 1) - 1;
    return __ldg(w + max(min(k ^ 1, last), 0));
}

// Fields [lo, hi) of 16-column word i (column 16i + f at bits 31-2f, 30-2f).
__device__ __forceinline__ uint32_t field_mask(int32_t lo, int32_t hi, int i)
{
    const uint32_t a = (uint32_t)min(max(lo - 16 * i, 0), 16) * 2;
    const uint32_t b = (uint32_t)min(max(hi - 16 * i, 0), 16) * 2;
    return __funnelshift_rc(0xFFFFFFFFu, 0u, a) & ~__funnelshift_rc(0xFFFFFFFFu, 0u, b);
}

// Needleman-Wunsch: register value of the initial row (row -1) at column j, with
// `drift` = g * (-2 - b + j) less the re-centring so far.
__device__ __forceinline__ uint32_t nw_init(int32_t j, int32_t b, int32_t go, int32_t ge,
                                            int32_t drift)
{
    const int32_t ri = j - b;
    const int32_t v = (ri == 0 ? 0 : go + ri * ge) + drift;
    return (uint32_t)(uint16_t)(int16_t)(ri < 0 || j > 2 * b ? kNwFloor : v);
}

// One step over the lane's R registers.  cw: the equality bits of row t' and, one bit
// above them, those of row t'-1 shifted so column R + h sits where column h does; tab, l16:
// the score table and the lane's place in its rows.  hl / el: the
// left neighbours of register 0.  Returns the last register's H and E' through
// hl / el, and the row keys (Smith-Waterman) through klo / khi.  START
// (Needleman-Wunsch): halves of rows before 0 are held at the initial row, and
// row 0's cells left of the reference start set to the floor.
template <int R, bool NW, bool START>
__device__ __forceinline__ void split_step(uint32_t (&Hr)[R], const uint32_t *cw,
                                           const char *tab, uint32_t l16, uint32_t &hl,
                                           uint32_t &el,
                                           int32_t &klo, int32_t &khi, int G,
                                           uint32_t last_mask, const SplitConsts &c, int32_t row,
                                           int32_t b, int32_t c0)
{
    constexpr int NG = (R + 7) / 8;  // key groups: register h in group h % NG, tag 7 - h / NG
    const uint32_t floor2 = (uint32_t)(uint16_t)(int16_t)kNwFloor * 0x00010001u;
    uint32_t h0 = 0, nx = 0;
    uint32_t gk[NG], pend[NG], sub[4];
    const uint32_t hold = START ? (row < 0 ? 0x0000FFFFu : 0u) | (row < 1 ? 0xFFFF0000u : 0u) : 0u;
#pragma unroll
    for (int h = 0; h < R; ++h) {
        if ((h & 3) == 0) {  // row of the table: the byte of these four columns
            const char *const row =
                tab + __byte_perm(cw[h >> 4], l16, 0x7704 | ((3 - ((h >> 2) & 3)) << 4));
            if (h + 1 < R) {
                const uint4 v = *reinterpret_cast<const uint4 *>(row);
                sub[0] = v.x;
                sub[1] = v.y;
                sub[2] = v.z;
                sub[3] = v.w;
            } else {
                sub[0] = *reinterpret_cast<const uint32_t *>(row);
            }
        }
        const uint32_t up = (h + 1 < R) ? Hr[h + 1 < R ? h + 1 : h] : __byte_perm(h0, nx, 0x5432);
        uint32_t hn;
        const uint32_t old = Hr[h];
        if (!NW) {
            const uint32_t e = __viaddmax_s16x2(el, c.ge2, up);
            const uint32_t tt = __vimax3_s16x2(e, hl, c.ng2);
            hn = __viaddmax_s16x2(Hr[h], sub[h & 3], tt) * c.one + c.neg_g2;
            el = e;
        } else {
            hn = __vimax3_s16x2(__viaddmax_s16x2(Hr[h], sub[h & 3], up), hl, floor2);
            if (START) {
                hn = (hn & ~hold) | (old & hold);
                // row 0, left of the reference start: outside, although the initial
                // row's 0 is its upper neighbour (column b - 1)
                const int32_t j = c0 + h;
                if (row == 0 && j < b)
                    hn = (hn & 0xFFFF0000u) | (floor2 & 0x0000FFFFu);
                if (row == 1 && j + R < b)
                    hn = (hn & 0x0000FFFFu) | (floor2 & 0xFFFF0000u);
            }
        }
        hl = hn;
        Hr[h] = hn;
        if (h == 0) {
            h0 = hn;
            nx = __shfl_down_sync(0xffffffffu, hn, 1, G);
            nx = NW ? (nx & last_mask) | (floor2 & ~last_mask) : nx & last_mask;
        }
        if (!NW) {
            const int f = h % NG, i = h / NG;
            const uint32_t key = hn * c.x8 + (uint32_t)(7 - i) * 0x00010001u;
            if (i == 0)
                gk[f] = key;
            else if (i & 1)
                pend[f] = key;
            else
                gk[f] = __vimax3_u16x2(gk[f], pend[f], key);
            if ((i & 1) && h + NG >= R)
                gk[f] = __vimax3_u16x2(gk[f], pend[f], pend[f]);
        }
    }
    if (!NW) {
        // 32-bit keys: (H - base) * 8 + tag on top, low-half flag and group below
        int32_t lo = 0, hi = 0;
#pragma unroll
        for (int f = 0; f < NG; ++f) {
            const int32_t a = (int32_t)(gk[f] * c.x64k + (uint32_t)(NG - 1 - f + 8));
            const int32_t d = (int32_t)((gk[f] & 0xFFFF0000u) | (uint32_t)(NG - 1 - f));
            lo = f == 0 ? a : max(lo, a);
            hi = f == 0 ? d : max(hi, d);
        }
        klo = lo;
        khi = hi;
    }
}

constexpr int kSplitThreads = 256;

// WIDE_G: Needleman-Wunsch with g above kNwWrapFree (a kernel of its own: the branch alone
// costs the others 1.4%, band 64).
template <int R, bool NW, bool WIDE_G>
__global__ void __launch_bounds__(kSplitThreads, 2)
split_kernel(SeqView q, SeqView r, SplitConsts c, SplitWork work, const int32_t *__restrict__ bands,
             int32_t band, gb2_sw_result *__restrict__ out)
{
    constexpr int NE = (2 * R + 15) / 16;  // 16-column words of a lane's columns
    constexpr int NB = (R + 15) / 16;      // words of its high columns
    constexpr int NG = (R + 7) / 8;
    const int lane = threadIdx.x & 31;
    constexpr int WARPS = kSplitThreads / 32;
    const uint32_t FULL = 0xffffffffu;
    const uint32_t floor2 = (uint32_t)(uint16_t)(int16_t)kNwFloor * 0x00010001u;
    extern __shared__ uint4 smem_tab[];
    score_table_fill(smem_tab, c.sub2, c.dm, kSplitThreads);
    __syncthreads();
    const char *const tab = (const char *)smem_tab;
    const uint32_t l16 = (uint32_t)(lane & 15) * 16;

    // Tasks: the pairs of one warp, a run of a segment's queue (longest first).  The
    // first task of a warp is given by its place in the grid, the segments in turn: if
    // the warps asked for it, an SM whose warps start together would take the longest
    // pairs for itself (50,000 mixed pairs: SMs busy 0.6 to 4.2 M cycles).  After
    // that a warp takes from the segment whose next pair is longest, so that no long
    // pair starts last.
    const int64_t rank = warp_rank();
    const int64_t warps = (int64_t)gridDim.x * WARPS;
    bool first_task = true;
    {
        for (;;) {
            int si = 0;
            int64_t base0 = 0;
            if (first_task) {
                si = (int)(rank % work.count);
                base0 = rank / work.count * (32 >> work.lg[si]);
            } else {
                if (work.count > 1) {
                    uint32_t key = 0;  // length + 1 of the segment's next pair, segment
                    if (lane < work.count) {
                        int64_t m;
                        const int32_t *__restrict__ qu = pairs_resolve(work.list[lane], m);
                        const int64_t given =
                            (warps - lane + work.count - 1) / work.count * (32 >> work.lg[lane]);
                        const int64_t at =
                            given + *(const volatile int *)work.list[lane].counter;
                        if (at < m)
                            key = ((uint32_t)min(q.lengths[qu ? (int64_t)qu[at] : at],
                                                 (int64_t)0x1FFFFFF0) + 1) * 8 + lane;
                    }
                    key = __reduce_max_sync(FULL, key);
                    if (key == 0)
                        break;
                    si = (int)(key & 7);
                }
                if (lane == 0)
                    base0 = atomicAdd(work.list[si].counter, 32 >> work.lg[si]);
                base0 = __shfl_sync(FULL, base0, 0) +
                        (warps - si + work.count - 1) / work.count * (32 >> work.lg[si]);
            }
            const int lg = work.lg[si], G = 1 << lg, gl = lane & (G - 1);
            int64_t n;
            const int32_t *__restrict__ queue = pairs_resolve(work.list[si], n);
            if (base0 >= n) {
                if (!first_task && work.count == 1)
                    break;
                first_task = false;
                continue;
            }
            first_task = false;
            const int64_t slot = base0 + (lane >> lg);
            const bool valid = slot < n;
            const int64_t pi = valid ? (queue ? (int64_t)queue[slot] : slot)
                                     : (queue ? (int64_t)queue[base0] : base0);
            const int32_t b = bands ? bands[pi] : band;
            const int32_t qlen = valid ? (int32_t)q.lengths[pi] : 0;
            const int32_t rlen = valid ? (int32_t)r.lengths[pi] : 0;
            // an empty sequence has no word of its own: its reads go to the array's first
            const uint32_t *const qp = reinterpret_cast<const uint32_t *>(
                q.packed + (qlen > 0 ? q.offsets[pi] - q.word_base : 0));
            const uint32_t *const rp = reinterpret_cast<const uint32_t *>(
                r.packed + (rlen > 0 ? r.offsets[pi] - r.word_base : 0));
            const int32_t c_high = work.high[si], c_low = work.low[si];
            const int32_t steps =
                __reduce_max_sync(FULL, qlen > 0 ? qlen + 2 * G - 1 : 0);
            const int32_t skew = 2 * gl, c0 = 2 * R * gl;
            // zero in the pair's first lane / the value past its last lane
            const uint32_t first_mask = gl == 0 ? 0u : 0xFFFFFFFFu;
            const uint32_t last_mask = gl == G - 1 ? 0u : 0xFFFFFFFFu;

            uint32_t Hr[R];
#pragma unroll
            for (int h = 0; h < R; ++h) {
                Hr[h] = 0;
                if (NW) {
                    const int32_t d = -c.g * (2 + b);
                    Hr[h] = nw_init(c0 + h, b, c.go, c.ge, d + c.g * (c0 + h)) |
                            nw_init(c0 + h + R, b, c.go, c.ge, d + c.g * (c0 + h + R)) << 16;
                }
            }
            uint32_t win[NE], ep[NE], em[NE];
            // window of row -skew: r[-skew - b + c0 ..); the stream feeding it follows on
            const int32_t p0 = c0 - skew - b;
            const uint32_t rsh = (uint32_t)(p0 & 15) * 2;
            int32_t rk = p0 >> 4;
            uint32_t rr0 = word16(rp, rlen, rk), rr1;
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                const uint32_t nw = word16(rp, rlen, rk + i + 1);
                win[i] = __funnelshift_l(nw, rr0, rsh);
                rr0 = nw;
                ep[i] = 0;
                em[i] = 0;
            }
            rk += NE + 1;
            rr1 = word16(rp, rlen, rk);
            const uint32_t qsh = (uint32_t)((-skew) & 15) * 2;
            int32_t qk = (-skew) >> 4;
            uint32_t qr0 = word16(qp, qlen, qk), qr1 = word16(qp, qlen, qk + 1);
            qk += 1;
            uint32_t qw = 0, rw = 0;
            // rows [tlo, thi) of this lane lie inside the matrix
            const int32_t cols = min(max(2 * b + 1 - c0, 0), 2 * R);
            const int32_t tlo = max(0, b - c0);
            const int32_t thi = min(qlen, rlen - cols + b - c0 + 1);
            const uint32_t inner = cols == 0 || qlen == 0 ? 0xFFFFFFFFu
                                   : thi > tlo            ? (uint32_t)(thi - tlo - 1)
                                                          : 0u;

            uint32_t hl = NW ? floor2 : 0u, el = kSent | (kSent << 16);
            // Smith-Waterman: registers hold H - base.  bkey / bt: the lane's first
            // maximum since base last moved, and its step; skey / srow / sscore: before
            int32_t base = 0, thr = 0x7FFFF, bkey = 0, bt = 0;
            int32_t skey = 0, srow = 0, sscore = 0;
            const int32_t fo = rlen - qlen + b;  // Needleman-Wunsch: column of the final cell
            int32_t drift = -c.g * (2 + b);      // of row -1 at column 0
            if (NW && valid && gl == 0 && (qlen <= 0 || rlen <= 0 || fo < 0 || fo > 2 * b)) {
                gb2_sw_result res;
                res.score = qlen == 0 && fo >= 0 && fo <= 2 * b
                                ? (rlen == 0 ? 0 : c.go + rlen * c.ge)
                                : kNwNeg;
                res.query_end = qlen - 1;
                res.ref_end = rlen - 1;
                out[pi] = res;
            }
            // one row: eq receives its equality bits, ep holds the previous row's
            auto one_row = [&](int32_t t, uint32_t (&eq)[NE], const uint32_t (&ep)[NE]) {
                const int32_t row = t - skew;
                // columns that lie inside the matrix at this row
                if ((uint32_t)(row - tlo - 1) >= inner) {
                    const int32_t ri0 = row - b + c0;
                    const bool live = row >= 0 && row < qlen;
                    const int32_t lo = max(-ri0, 0), hi = live ? min(cols, rlen - ri0) : 0;
#pragma unroll
                    for (int i = 0; i < NE; ++i)
                        em[i] = field_mask(lo, max(hi, lo), i) & 0x55555555u;
                }
                const uint32_t qrep = mad_hi(qw, c.x4, 0u) * 0x55555555u;
                qw *= c.x4;
#pragma unroll
                for (int i = 0; i < NE; ++i) {
                    const uint32_t x = win[i] ^ qrep;
                    eq[i] = ~(x | mad_hi(x, c.half, 0u)) & em[i];
                }
                uint32_t cw[NB];
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    constexpr int A = R / 16, S = 2 * (R % 16) + 1;
                    static_assert(S < 32, "one word back");
                    const uint32_t nxt = (A + i + 1 < NE) ? ep[A + i + 1 < NE ? A + i + 1 : 0] : 0u;
                    cw[i] = __funnelshift_l(nxt, ep[A + i < NE ? A + i : 0], S) | eq[i];
                }
#pragma unroll
                for (int i = 0; i < NE; ++i)
                    win[i] = win[i] * c.x4 + mad_hi(i + 1 < NE ? win[i + 1 < NE ? i + 1 : i] : rw,
                                                    c.x4, 0u);
                rw *= c.x4;
                int32_t klo = 0, khi = 0;
                if (NW && t < 2 * G)
                    split_step<R, NW, true>(Hr, cw, tab, l16, hl, el, klo, khi, G, last_mask, c,
                                            row, b, c0);
                else
                    split_step<R, NW, false>(Hr, cw, tab, l16, hl, el, klo, khi, G, last_mask, c,
                                             row, b, c0);
                // hand the last column's high half to the next lane; the low half is the
                // left neighbour of this lane's high columns
                if (!NW) {
                    uint32_t in = __shfl_up_sync(FULL, __byte_perm(hl, el, 0x7632), 1, G);
                    in = (in & first_mask) | (~first_mask & (kSent << 16));
                    hl = __byte_perm(in, hl, 0x5410);
                    el = __byte_perm(in, el, 0x5432);
                    // the high halves complete row t'-1; its low halves came a step earlier
                    if (khi > thr) {
                        bkey = khi;
                        bt = t;
                    }
                    thr = max(thr, khi | 0x7FFFF);
                    if (klo > thr) {
                        bkey = klo;
                        bt = t;
                    }
                    thr = max(thr, klo | 0x7FFFF);
                } else {
                    uint32_t in = __shfl_up_sync(FULL, hl, 1, G);
                    in = (in & first_mask) | (~first_mask & floor2);
                    hl = __byte_perm(in, hl, 0x5432);
                    if (row == qlen - 1 || row == qlen) {
                        const int32_t cf = fo - c0;
                        const bool low = row == qlen - 1;
                        const int32_t want = low ? cf : cf - R;
                        if (valid && qlen > 0 && rlen > 0 && fo <= 2 * b && want >= 0 &&
                            want < R) {
                            uint32_t v = 0;
#pragma unroll
                            for (int h = 0; h < R; ++h)
                                if (want == h)
                                    v = Hr[h];
                            const int32_t s = (int32_t)(int16_t)(low ? v : v >> 16);
                            // drift of row qlen - 1 at column fo
                            gb2_sw_result res;
                            res.score = s - (drift + c.g * (fo + 2 * qlen));
                            res.query_end = qlen - 1;
                            res.ref_end = rlen - 1;
                            out[pi] = res;
                        }
                    }
                }
            };
            // the row of a key of step t, and its column
            auto key_row = [&](int32_t key, int32_t t) { return t - skew - ((key & 8) ? 0 : 1); };
            for (int32_t t0 = 0; t0 < steps; t0 += 16) {
                qw = __funnelshift_l(qr1, qr0, qsh);
                qr0 = qr1;
                qr1 = word16(qp, qlen, ++qk);
                rw = __funnelshift_l(rr1, rr0, rsh);
                rr0 = rr1;
                rr1 = word16(rp, rlen, ++rk);
                if (NW && t0 > 0) {  // re-centre: 2g per row
                    const uint32_t d2 = (uint32_t)(uint16_t)(int16_t)(-32 * c.g) * 0x00010001u;
                    if (WIDE_G) {  // the sum below wraps: no cell under floor + 32g
                        const uint32_t lim2 =
                            (uint32_t)(uint16_t)(int16_t)(kNwFloor + 32 * c.g) * 0x00010001u;
#pragma unroll
                        for (int h = 0; h < R; ++h)
                            Hr[h] = __vmaxs2(Hr[h], lim2);
                        hl = __vmaxs2(hl, lim2);
                    }
#pragma unroll
                    for (int h = 0; h < R; ++h)
                        Hr[h] = __viaddmax_s16x2(Hr[h], d2, floor2);
                    hl = __viaddmax_s16x2(hl, d2, floor2);
                    drift -= 32 * c.g;
                }
                if (!NW && c_high >= 0) {
                    uint32_t m2 = Hr[0];
#pragma unroll
                    for (int h = 1; h < R; ++h)
                        m2 = __vmaxu2(m2, Hr[h]);
                    int32_t m = max((int32_t)(m2 & 0xFFFFu), (int32_t)(m2 >> 16));
                    for (int o = 1; o < G; o <<= 1)
                        m = max(m, __shfl_xor_sync(FULL, m, o));
                    const int32_t target = (c_low + c_high) / 2;
                    int32_t d = 0;
                    if (m > c_high)
                        d = m - target;
                    else if (m < c_low && base > 0)
                        d = -min(base, target - m);
                    if (d != 0) {
                        const uint32_t d2 = (uint32_t)(uint16_t)(int16_t)(-d) * 0x00010001u;
#pragma unroll
                        for (int h = 0; h < R; ++h)
                            Hr[h] = __viaddmax_s16x2_relu(Hr[h], d2, 0u);
                        hl = __viaddmax_s16x2_relu(hl, d2, 0u);
                        el = __viaddmax_s16x2(el, d2, kSent | (kSent << 16));
                        // the band's left edge stays where it is
                        hl &= first_mask | 0xFFFF0000u;
                        el = (el & (first_mask | 0xFFFF0000u)) | (~first_mask & kSent);
                        if (bkey > 0) {
                            sscore = (bkey >> 19) + base;
                            srow = key_row(bkey, bt);
                            skey = bkey;
                            bkey = 0;
                        }
                        base += d;
                        thr = (min(max(sscore - base, -1), 4095) << 19) | 0x7FFFF;
                    }
                }
                const int32_t t1 = min(t0 + 16, steps);
                for (int32_t t = t0; t < t1; t += 2) {  // an odd count runs one empty row more
                    uint32_t em1[NE];
                    one_row(t, em1, ep);
                    one_row(t + 1, ep, em1);
                }
            }
            if (!NW) {
                // first maximum of the pair: score, then the smaller row, then column
                int32_t score = sscore, bq = srow, key = skey, col = 0;
                if (bkey > 0) {  // since base last moved: larger than all before
                    score = (bkey >> 19) + base;
                    bq = key_row(bkey, bt);
                    key = bkey;
                }
                if (key > 0) {
                    const int32_t h = (7 - ((key >> 16) & 7)) * NG + (NG - 1 - (key & 7));
                    col = c0 + h + ((key & 8) ? 0 : R);
                }
                for (int o = 1; o < G; o <<= 1) {
                    const int32_t os = __shfl_xor_sync(FULL, score, o);
                    const int32_t oq = __shfl_xor_sync(FULL, bq, o);
                    const int32_t oc = __shfl_xor_sync(FULL, col, o);
                    if (os > score || (os == score && (oq < bq || (oq == bq && oc < col)))) {
                        score = os;
                        bq = oq;
                        col = oc;
                    }
                }
                if (valid && gl == 0) {
                    gb2_sw_result res;
                    res.score = score;
                    res.query_end = score > 0 ? bq : 0;
                    res.ref_end = score > 0 ? bq - b + col : 0;
                    out[pi] = res;
                }
            }
        }
    }
}

constexpr int kRegs[kSplitShapes] = {5, 9, 13, 17, 21, 25, 29, 33};

template <bool NW, bool WIDE_G, typename F>
auto with_shape(int shape, F f)
{
    switch (shape) {
    case 0: return f(split_kernel<kRegs[0], NW, WIDE_G>);
    case 1: return f(split_kernel<kRegs[1], NW, WIDE_G>);
    case 2: return f(split_kernel<kRegs[2], NW, WIDE_G>);
    case 3: return f(split_kernel<kRegs[3], NW, WIDE_G>);
    case 4: return f(split_kernel<kRegs[4], NW, WIDE_G>);
    case 5: return f(split_kernel<kRegs[5], NW, WIDE_G>);
    case 6: return f(split_kernel<kRegs[6], NW, WIDE_G>);
    default: return f(split_kernel<kRegs[7], NW, WIDE_G>);
    }
}

template <typename F>
auto with_kernel(bool nw, bool wide_g, int shape, F f)
{
    return !nw      ? with_shape<false, false>(shape, f)
           : wide_g ? with_shape<true, true>(shape, f)
                    : with_shape<true, false>(shape, f);
}

template <typename K>
cudaError_t split_smem(K *kern, bool nw, bool wide_g, int shape)
{
    static std::atomic<uint64_t> done[3][kSplitShapes];  // one pointer type for all shapes
    return allow_smem(kern, kScoreTableBytes, done[wide_g ? 2 : nw ? 1 : 0][shape]);
}

int occupancy(bool nw, int shape)
{
    auto occ = [&](auto kern) {
        int nb = 0;
        if (split_smem(kern, nw, false, shape) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kSplitThreads,
                                                          kScoreTableBytes) != cudaSuccess)
            cudaGetLastError();
        return std::max(nb, 1);
    };
    return with_kernel(nw, false, shape, occ);
}

}  // namespace

int split_regs(int shape) { return kRegs[shape]; }

int split_grid(bool nw, int shape, int lg, int64_t n, int sm_count)
{
    // a block per warp's work while there are SMs without one: the warps of a block take
    // the first tasks of the grid in turn
    const int64_t per = 32 >> lg;
    return (int)std::min<int64_t>((n + per - 1) / per,
                                  (int64_t)sm_count * split_blocks_per_sm(nw, shape));
}

int split_blocks_per_sm(bool nw, int shape)
{
    struct Table {
        int v[2][kSplitShapes];
        Table()
        {
            for (int s = 0; s < kSplitShapes; ++s) {
                v[0][s] = occupancy(false, s);
                v[1][s] = occupancy(true, s);
            }
        }
    };
    static const Table t;
    return t.v[nw ? 1 : 0][shape];
}

bool split_rebase(const SwParams &p, int shape, int lg, int32_t *low, int32_t *high)
{
    const int64_t G = 1 << lg, cols = 2 * (int64_t)kRegs[shape] * G;
    const int64_t g = -(p.go + p.ge), mm = -p.mismatch, m = std::max(p.match, 0);
    const int64_t lo = (cols + 2 * G) * (m + mm + g) + 16 * mm + g + 1;
    const int64_t hi = 4094 - 17 * m;
    *low = (int32_t)std::min<int64_t>(lo, 1 << 20);
    *high = (int32_t)hi;
    // the spread argument looks 2RG rows up inside the matrix: a value above
    // `high` needs at least high / match rows
    return lo + 128 <= hi && (m == 0 || hi / m >= 2 * cols + 2 * G + 16);
}

// Fitted to 400,000 reads (150 vs 200 bp, band 33: 125, 181, 220, 286, 324, 388, 434, 500
// cycles per warp and row for the shapes in order; Needleman-Wunsch 7.1 R + 74) and to
// 150-600 Smith-Waterman pairs of 3-9 kbp, one warp per scheduler (244, 318, 381, 464, 524,
// 606, 676, 785; Needleman-Wunsch is priced with the same, its own chain not measured).  `rows`: rows a warp runs beside those of its pairs.
// Pairs of one length run in rounds of four warps per scheduler, the last round as long
// as its fullest scheduler (150 bp, band 32: 20,000 pairs R = 9, 17, one thread per pair
// 97, 81, 79 us; 40,000: 155, 146, 111).  Of ragged pairs the longest come first: the
// larger of all the work and the longest pair bounds the batch and about a third of the
// other shows beside it; while all warps are resident the schedulers with one warp more
// set the pace (16,000 pairs of 2-10 kbp, band 128: R = 33, 2,000 warps, 7.5 ms; R = 17,
// 4,000 warps, 6.0; 4,000 pairs: R = 9 2.8 ms, 17 2.9, 33 4.3).
double split_time(double issue, double chain, double warps, double rows, const SplitLoad &l)
{
    if (l.max_rows <= 1.25 * l.mean_rows) {
        const double full = std::floor(warps / 4), rest = std::ceil(warps - 4 * full);
        const double row = full * std::max(4 * issue, chain) +
                           (rest > 0 ? std::max(rest * issue, chain) : 0.0);
        return row * (l.max_rows + rows);
    }
    const double busy = warps <= 4 ? std::ceil(warps) : warps;
    const double total = busy * issue * (l.mean_rows + rows), longest = chain * l.max_rows;
    return std::max(total, longest) + 0.35 * std::min(total, longest);
}

SplitChoice split_choose(const SwParams &p, int32_t band, const SplitLoad &l, bool nw,
                         bool long_scores, int only_shape)
{
    SplitChoice best{-1, 0, 0.0};
    for (int s = 0; s < kSplitShapes; ++s) {
        const int R = kRegs[s];
        int lg = 0;  // more lanes of the same shape only add padding
        while (lg <= 5 && 2 * R * (1 << lg) < 2 * (int64_t)band + 1)
            ++lg;
        int32_t low, high;
        if ((only_shape >= 0 && s != only_shape) || lg > 5 ||
            (!nw && long_scores && !split_rebase(p, s, lg, &low, &high)))
            continue;
        const double warps = (double)l.pairs * (1 << lg) / 32 / (4.0 * l.sm_count);
        // 15,000 cycles: the start of a pair, which the one-thread kernel has not
        const double t = 15000 + split_time(nw ? 7.1 * R + 74 : 13.3 * R + 60, 19.2 * R + 148,
                                            warps, 2.0 * (1 << lg), l);
        if (best.shape < 0 || t < best.cost)
            best = SplitChoice{s, lg, t};
    }
    return best;
}

cudaError_t launch_split(bool nw, int shape, SeqView q, SeqView r, SwParams p, int32_t band,
                         const int32_t *bands, const SplitWork &work, gb2_sw_result *out, int grid,
                         cudaStream_t st)
{
    const uint32_t g = (uint32_t)(-(p.go + p.ge)), dm = (uint32_t)(p.match - p.mismatch);
    SplitConsts c;
    c.x4 = 4;
    c.x8 = 8;
    c.x64k = 65536;
    c.half = 0x80000000u;
    c.one = 1;
    c.dm = dm;
    c.sub2 = ((uint32_t)p.mismatch + (nw ? 2 * g : g)) * 0x00010001u;
    c.neg_g2 = 0u - g * 0x00010001u;
    c.ng2 = g * 0x00010001u;
    c.ge2 = (uint32_t)(uint16_t)p.ge * 0x00010001u;
    c.go = p.go;
    c.ge = p.ge;
    c.g = (int32_t)g;
    const bool wide_g = nw && c.g > kNwWrapFree;
    auto go = [&](auto kern) {
        const cudaError_t e = split_smem(kern, nw, wide_g, shape);
        if (e != cudaSuccess)
            return e;
        kern<<<grid, kSplitThreads, kScoreTableBytes, st>>>(q, r, c, work, bands, band, out);
        return cudaGetLastError();
    };
    return with_kernel(nw, wide_g, shape, go);
}

}  // namespace gb2
