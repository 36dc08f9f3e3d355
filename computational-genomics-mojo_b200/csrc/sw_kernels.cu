// sw_kernels.cu -- banded Smith-Waterman on sm_100a.
//
// Computes smith_waterman_banded (genomics/cpu/align_cpu.mojo:229-309)
// bit-exactly: score plus the first maximum cell in row-major order.
//
// Band coordinates: row qi (query position), column j in [0, 2B],
// ri = qi - B + j.  Cell (qi, j) reads diag (qi-1, j), up (qi-1, j+1) and
// left (qi, j-1) (align_cpu.mojo:277-279); E extends along the row from the
// left cell's E and opens from up (:282-283); F opens from the left H with
// no extension (:287).
//
// Register kernel (sw_band_kernel<B, G, K>): G lanes of a warp own one pair;
// lane l owns band columns [l*K, l*K + K) and keeps their H values in
// registers.  Lane l processes row t - l at step t: its first column takes
// the left neighbour's last column of the same row (computed by lane l-1 one
// step earlier, passed by warp shuffle) and its last column takes as "up"
// the right neighbour's first column of the previous row (computed by lane
// l+1 in the first phase of the same step, passed by shuffle).  With G == 1
// a thread owns the whole band row and no shuffles run.
//
// Exactness of the register kernel rests on three facts, valid when
// gap_extend <= 0, gap_open + gap_extend <= 0 and mismatch <= 0 (the host
// checks these and otherwise uses the literal kernel):
//  1. E only influences H through max(E, 0), and with gap_extend <= 0 a
//     non-positive E never becomes positive along the row, so carrying
//     E+ = max(E, 0) reproduces every H.  The reference's -1000000 start of
//     the E chain at j == 0 and the zero E of a skipped cell (:282) both
//     become E+ = 0 on the left boundary.
//  2. Cells left of the reference start (ri < 0) are skipped (zero) in the
//     reference; giving them a never-matching base makes the recurrence
//     produce exactly zero there, so no per-cell masking is needed.
//  3. Cells past the reference end (ri >= rlen) or past the query end never
//     feed a cell inside the matrix (every dependency has column <= ri and
//     row <= qi), so they are computed but excluded from the maximum.
// Padding columns past 2B in the last lane are forced to zero so column 2B
// sees the out-of-band "up" value 0 (:278).
#include "gb2_internal.cuh"

namespace gb2 {

__device__ __forceinline__ void sw_cell(int32_t hdiag, int32_t hup, int32_t hleft,
                                        int32_t eleft, int32_t sub, int32_t goe,
                                        int32_t ge, int32_t &hn, int32_t &en)
{
    // E+ = max(E_left + ge, H_up + go + ge, 0)
    en = __viaddmax_s32_relu(hup, goe, eleft + ge);
    // H = max(H_diag + sub, E+, H_left + go + ge, 0)
    hn = __viaddmax_s32_relu(hleft, goe, __viaddmax_s32(hdiag, sub, en));
}

// Writes the result of one pair from the group's packed best key.
__device__ __forceinline__ void sw_store(gb2_sw_result *out, int64_t pi, uint64_t key, int B)
{
    gb2_sw_result res;
    if (key == 0) {
        res.score = 0;
        res.query_end = 0;
        res.ref_end = 0;
    } else {
        int32_t best = (int32_t)(key >> 42);
        int32_t bq = 0x1FFFFF - (int32_t)((key >> 21) & 0x1FFFFF);
        int32_t bj = 0x1FFFFF - (int32_t)(key & 0x1FFFFF);
        res.score = best;
        res.query_end = bq;
        res.ref_end = bq - B + bj;
    }
    out[pi] = res;
}

template <int B, int G, int K>
__global__ void __launch_bounds__(128)
sw_band_kernel(SeqView q, SeqView r, SwParams p, PairList pl, gb2_sw_result *__restrict__ out)
{
    int64_t n;
    const int32_t *__restrict__ queue = pairs_resolve(pl, n);
    int *const queue_counter = pl.counter;
    constexpr int W = 2 * B + 1;
    static_assert(G * K >= W, "band does not fit");
    static_assert(G == 1 || K >= 2, "pipelined lanes need two columns");
    static_assert(32 % G == 0, "G divides the warp");
    constexpr int CPAD = W - (G - 1) * K;  // first padding column of the last lane
    static_assert(CPAD >= 1 && CPAD <= K, "G is not minimal");
    constexpr int NW = (K + 31) / 32;  // 64-bit window words per lane
    constexpr int PAIRS_PER_WARP = 32 / G;

    const int lane = threadIdx.x & 31;
    const int gl = lane % G;
    const int gw = lane / G;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (gw * G));
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);

    const int32_t goe = p.go + p.ge;
    const int32_t ge = p.ge;
    const int32_t m = p.match, mm = p.mismatch;

    // A warp's first pairs go by its place in the grid, one to an SM first: if the warps
    // asked for them, the SMs that start first would take them all from a class with fewer
    // pairs than the call (6,000 pairs of 2,000 bp, bands 16-128, +5/-4/-10/-1, the int32
    // kernel for the 1,500 of band 128 beside the lane-split one: 3.5 -> 1.65 ms).
    int64_t base = warp_rank() * PAIRS_PER_WARP;
    for (bool asked = false;; asked = true) {
        if (queue_counter && asked) {
            int64_t b0 = 0;
            if (lane == 0)
                b0 = atomicAdd(queue_counter, PAIRS_PER_WARP);
            base = __shfl_sync(0xffffffffu, b0, 0) + warps_total * PAIRS_PER_WARP;
        }
        if (base >= n)
            break;
        const int64_t slot = base + gw;
        if (slot < n) {
            const int64_t pi = queue ? (int64_t)queue[slot] : slot;
            const int64_t qoff = q.offsets[pi] - q.word_base;
            const int64_t roff = r.offsets[pi] - r.word_base;
            const int32_t qlen = (int32_t)q.lengths[pi], rlen = (int32_t)r.lengths[pi];

            int32_t H[K];
#pragma unroll
            for (int c = 0; c < K; ++c)
                H[c] = 0;
            int32_t h_in = 0, e_in = 0;
            int32_t best = 0, bq = 0, bj = 0;
            const int steps = qlen > 0 ? qlen + G - 1 : 0;
            for (int t = 0; t < steps; ++t) {
                const int qi = t - gl;
                const bool row_live = (qi >= 0) && (qi < qlen);
                const int64_t ri0 = (int64_t)qi - B + gl * K;
                uint64_t eq[NW];
                if (row_live) {
                    const uint64_t qw = __ldg(q.packed + qoff + (qi >> 5));
                    const uint64_t qb = (qw >> (62 - 2 * (qi & 31))) & 3u;
                    const uint64_t qrep = qb * 0x5555555555555555ull;
                    // NW+1 consecutive words cover the K-base window at ri0
                    const int64_t w = roff + (ri0 >> 5);
                    const int sh = (int)(ri0 & 31) * 2;
                    uint64_t words[NW + 1];
#pragma unroll
                    for (int i = 0; i <= NW; ++i) {
                        int64_t wi = w + i;
                        wi = wi < 0 ? 0 : (wi >= r.n_words ? r.n_words - 1 : wi);
                        words[i] = __ldg(r.packed + wi);
                    }
#pragma unroll
                    for (int i = 0; i < NW; ++i) {
                        const uint64_t win =
                            sh ? ((words[i] << sh) | (words[i + 1] >> (64 - sh))) : words[i];
                        const uint64_t x = win ^ qrep;
                        eq[i] = ~(x | (x >> 1)) & 0x5555555555555555ull;
                    }
                    if (ri0 < 0) {  // columns before the reference start never match
                        const int64_t nneg = -ri0;
#pragma unroll
                        for (int i = 0; i < NW; ++i) {
                            const int64_t cnt = nneg - 32 * i;
                            if (cnt >= 32)
                                eq[i] = 0;
                            else if (cnt > 0)
                                eq[i] &= (~0ull) >> (2 * cnt);
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < NW; ++i)
                        eq[i] = 0;
                }

                // phase 1: first column
                int32_t hn, en;
                {
                    const int32_t sub = ((eq[0] >> 62) & 1u) ? m : mm;
                    const int32_t hup = (K > 1) ? H[K > 1 ? 1 : 0] : 0;
                    sw_cell(H[0], hup, h_in, e_in, sub, goe, ge, hn, en);
                    if (CPAD == 0 && gl == G - 1)
                        hn = 0;
                    H[0] = hn;
                }
                int32_t up_next = 0;
                if (G > 1) {
                    up_next = __shfl_down_sync(gmask, hn, 1, G);
                    if (gl == G - 1)
                        up_next = 0;
                }
                int32_t hl = hn, el = en;
                // phase 2: remaining columns, left to right
#pragma unroll
                for (int c = 1; c < K; ++c) {
                    const int32_t sub =
                        ((eq[c >> 5] >> (62 - 2 * (c & 31))) & 1u) ? m : mm;
                    const int32_t hup = (c + 1 < K) ? H[c + 1 < K ? c + 1 : c] : up_next;
                    sw_cell(H[c], hup, hl, el, sub, goe, ge, hn, en);
                    if (c >= CPAD && gl == G - 1)
                        hn = 0;
                    H[c] = hn;
                    hl = hn;
                    el = en;
                }
                if (G > 1) {
                    h_in = __shfl_up_sync(gmask, hl, 1, G);
                    e_in = __shfl_up_sync(gmask, el, 1, G);
                    if (gl == 0) {
                        h_in = 0;
                        e_in = 0;
                    }
                }
                // first maximum of this row inside the matrix: key = H*256 + (255-c)
                if (row_live) {
                    int32_t rk = 0;
                    if (ri0 + K - 1 < rlen) {
#pragma unroll
                        for (int c = 0; c < K; ++c)
                            rk = max(rk, H[c] * 256 + (255 - c));
                    } else {
                        const int64_t lim = (int64_t)rlen - ri0;  // columns c < lim are inside
#pragma unroll
                        for (int c = 0; c < K; ++c)
                            rk = max(rk, (c < lim) ? H[c] * 256 + (255 - c) : 0);
                    }
                    if ((rk >> 8) > best) {
                        best = rk >> 8;
                        bq = qi;
                        bj = gl * K + 255 - (rk & 255);
                    }
                }
            }
            uint64_t key = 0;
            if (best > 0)
                key = ((uint64_t)best << 42) | ((uint64_t)(0x1FFFFF - bq) << 21) |
                      (uint64_t)(0x1FFFFF - bj);
#pragma unroll
            for (int off = 1; off < G; off <<= 1) {
                const uint64_t o = __shfl_xor_sync(gmask, key, off, G);
                key = o > key ? o : key;
            }
            if (gl == 0)
                sw_store(out, pi, key, B);
        }
        if (!queue_counter)
            base += warps_total * PAIRS_PER_WARP;
    }
}

// ---------------------------------------------------------------------------
// Packed int16x2 kernel (sw_pack16_kernel<B>): one thread per pair, two cells
// per 32-bit register, one DPX instruction advancing both.
//
// Band columns 0..B live in the low halves, columns B+1..2B in the high
// halves of R = B+1 registers; the high half of the last register is a
// padding column held at H = 0 (it is the out-of-band "up" of column 2B).
// At step t the low halves hold row t and the high halves row t-1, so the
// two cells of a register are never each other's neighbours:
//   low  (t, h):      diag/up from the same half of registers h, h+1 of step
//                     t-1; up of h = B is the high half of register 0 (row
//                     t-1, column B+1), computed earlier in this step;
//   high (t-1, B+1+h): diag/up from the same half of step t-1; left of h = 0
//                     is the low half of register B of step t-1 (row t-1,
//                     column B).
// Values: registers hold H; the E chain is carried as E - (go+ge), so
//   E' = max(E'_left + ge, H_up),
//   H  = max(H_diag + sub - (go+ge), E', H_left, -(go+ge)) + (go+ge).
// Without the max(E, 0) clamp E differs from the reference's E only in
// non-positive values, which never reach H (H takes max(.., 0)); the
// -1000000 start of the chain at column 0 becomes a large negative value.
// Bits: H <= 511 in every cell (the host checks match*(min(qlen, rlen) + 1)), all
// terms stay inside int16, and the first-maximum key H*128 + (127-column) fits
// an unsigned 16-bit half.
//
// What bounds it: instructions.  Issue saturates near 0.65 per cycle and scheduler,
// however the work is split between the integer ALU pipe (the DPX maxima, logic) and the
// FMA pipe (multiply-adds, fp16), each two cycles per instruction; so the step is built
// for few of them, 5.5 per register and 0.5 for its substitution term, and both pipes
// are kept near 65%:
//  - the substitution terms of four registers (eight cells) are one 16-byte load from a
//    table in shared memory, its row picked by one byte permutation from the word that
//    interleaves the equality bits of both rows (a logic op and a 32-bit high product per
//    register before);
//  - all values lie in [0, 1021], where the bits of the fp16 number n * 2^-24 are the
//    integer n: additions may run as fp16 on the FMA pipe, and one fp16 multiply-add with
//    relu subtracts |go+ge| and takes max(.., 0).  Even registers use it and leave two
//    DPX maxima; odd ones use three DPX maxima, the floor among them, and one addition.
//    (All registers the one way 2.04 ms, the other 2.05, in turn 1.95.)
//  - cells outside the matrix need no masks of their own: their equality bits are off, and
//    then they change nothing (see sw_split.cu; the host's conditions are the same).
// Multipliers are kernel arguments so that the compiler cannot turn the multiply-adds
// into shifts.  256 threads per block, two blocks per SM: the table takes 64 KB a block
// (192 x 3 and 320 x 2 threads: 2.12, 2.11 ms).
// 1,000,000 reads of 150 bp, band 32: 2.51 -> 1.79 ms (band 16 with results to pageable
// memory: 1.61 -> 1.28); instructions per row of band 32: 361 -> 275.
// Sequences are read as 16-base (32-bit) words, reloaded every 16 rows; the query word is
// consumed two bits per row by multiplication.
// ---------------------------------------------------------------------------
// Constants of sw_pack16_kernel, built by the host from SwParams.
struct Pack16Consts {
    uint32_t x4, x8, x128, half;
    uint32_t dm_pad;   // (match - mismatch) * 4
    uint32_t dm;       // match - mismatch
    uint32_t mmg2;     // mismatch - (go+ge) in both halves
    uint32_t ge2;      // ge in both halves
    uint32_t ng2;      // -(go+ge) in both halves
    uint32_t one_f;    // 1.0 in both halves
    uint32_t neg_g_f;  // -|go+ge| * 2^-24 in both halves
};

// Halves as fp16 numbers n * 2^-24, whose bits are the integer n for 0 <= n <= 2047.
__device__ __forceinline__ uint32_t add_f16x2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// max(a * b + c, 0)
__device__ __forceinline__ uint32_t fma_relu_f16x2(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

__device__ __forceinline__ uint32_t mad_hi_u32(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// 16-base word k (bases 16k..16k+15, first base in the top two bits) of the
// 2-bit MSB-first sequence starting at 64-bit word `off`; k is clamped into
// the packed array (the clamped words are never read by an in-matrix cell).
__device__ __forceinline__ uint32_t seq_word16(const SeqView &s, int64_t off, int64_t k)
{
    int64_t i = 2 * off + (k ^ 1);
    const int64_t last = 2 * s.n_words - 1;
    i = i < 0 ? 0 : (i > last ? last : i);
    return __ldg(reinterpret_cast<const uint32_t *>(s.packed) + i);
}

// One step of sw_pack16_kernel over all R registers.  cw[k]: the equality bits of
// columns 16k .. 16k+15 of row t (column 16k+c at bit 30-2c) with those of row t-1,
// columns B+1+16k .., one bit above them; e_pad: row t's word that starts at column B.
// tab, l16: the score table and the lane's place in its rows.  Returns the packed row
// keys: low half row t, high half row t-1.
template <int B>
__device__ __forceinline__ uint32_t pack16_cells(uint32_t (&Hr)[B + 1], const uint32_t *cw,
                                                 uint32_t e_pad, const char *tab, uint32_t l16,
                                                 uint32_t &e_last, const Pack16Consts &c)
{
    constexpr int NL = B + 1, R = NL;
    const uint32_t SENT = 0x0000C000u;
    uint32_t hl = Hr[R - 1] << 16;                    // low: band edge 0; high: H(t-1, B)
    uint32_t el = __byte_perm(SENT, e_last, 0x5410);  // low: chain start; high: E'(t-1, B)
    uint32_t h0new = 0;
    uint32_t rk = 0, kpend = 0;
    uint32_t sub[4];
#pragma unroll
    for (int h = 0; h < R; ++h) {
        if (h == R - 1) {
            sub[0] = mad_hi_u32(e_pad & 0x40000000u, c.dm_pad, c.mmg2);
        } else if ((h & 3) == 0) {  // row of the table: the byte of these four columns
            const uint32_t at = __byte_perm(cw[h >> 4], l16, 0x7704 | ((3 - ((h >> 2) & 3)) << 4));
            const uint4 v = *reinterpret_cast<const uint4 *>(tab + at);
            sub[0] = v.x;
            sub[1] = v.y;
            sub[2] = v.z;
            sub[3] = v.w;
        }
        const uint32_t up = (h + 1 < R) ? Hr[h + 1 < R ? h + 1 : h] : (h0new >> 16);
        const uint32_t e = __viaddmax_s16x2(el, c.ge2, up);
        uint32_t hn;
        if (h & 1) {
            const uint32_t tt = __vimax3_s16x2(e, hl, c.ng2);
            hn = add_f16x2(__viaddmax_s16x2(Hr[h], sub[h & 3], tt), c.neg_g_f);
        } else {
            const uint32_t tt = __vimax3_s16x2(add_f16x2(Hr[h], sub[h & 3]), e, hl);
            hn = fma_relu_f16x2(tt, c.one_f, c.neg_g_f);
        }
        hl = hn;
        if (h == R - 1)
            hn &= 0x0000FFFFu;  // padding column stays 0
        if (h == 0)
            h0new = hn;
        Hr[h] = hn;
        el = e;
        const uint32_t key =
            hn * c.x128 + (((uint32_t)(127 - h)) | ((uint32_t)(127 - NL - h) << 16));
        if (h & 1)
            rk = __vimax3_u16x2(rk, kpend, key);
        else
            kpend = key;
    }
    if ((R - 1) % 2 == 0)
        rk = __vimax3_u16x2(rk, kpend, kpend);
    e_last = el;
    return rk;
}

// Fields [lo, hi) of 16-column equality word i (column 16i + f at bit 30-2f).
__device__ __forceinline__ uint32_t eq_fields(int32_t lo, int32_t hi, int i)
{
    const uint32_t a = (uint32_t)min(max(lo - 16 * i, 0), 16) * 2;
    const uint32_t b = (uint32_t)min(max(hi - 16 * i, 0), 16) * 2;
    return __funnelshift_rc(0x55555555u, 0u, a) & ~__funnelshift_rc(0xFFFFFFFFu, 0u, b);
}

constexpr int kPackThreads = 256;

template <int B>
__global__ void __launch_bounds__(kPackThreads, 2)
sw_pack16_kernel(SeqView q, SeqView r, Pack16Consts c, PairList pl, gb2_sw_result *__restrict__ out)
{
    static_assert(B % 16 == 0, "band must be a multiple of 16");
    constexpr int W = 2 * B + 1;
    constexpr int NL = B + 1;           // columns in low halves
    constexpr int R = NL;               // registers
    constexpr int NE = (W + 15) / 16;   // 16-column equality words of one row
    constexpr int BW0 = NL / 16;        // first word of columns B+1.. (offset one column)
    constexpr int NBW = B / 16;         // shifted words of the previous row
    constexpr int RW0 = NE - B / 16;    // 16-base word entering the window at t = 0
    static_assert(W <= 127, "column index must fit the key");
    static_assert(NL % 16 == 1 && BW0 + NBW < NE, "word layout");

    int64_t n;
    const int32_t *__restrict__ queue = pairs_resolve(pl, n);
    int *const queue_counter = pl.counter;
    const int lane = threadIdx.x & 31;
    const int64_t warp_global = warp_rank();
    const int64_t warps_total = (int64_t)gridDim.x * (kPackThreads / 32);
    const uint32_t SENT = 0x0000C000u;  // -16384 in the low half

    extern __shared__ uint4 tab[];
    score_table_fill(tab, c.mmg2, c.dm, kPackThreads);
    __syncthreads();
    const uint32_t l16 = (uint32_t)(lane & 15) * 16;

    int64_t base = warp_global * 32;
    for (;;) {
        if (queue_counter) {
            int64_t b0 = 0;
            if (lane == 0)
                b0 = atomicAdd(queue_counter, 32);
            base = __shfl_sync(0xffffffffu, b0, 0);
        }
        if (base >= n)
            break;
        const bool valid = base + lane < n;
        const int64_t slot = valid ? base + lane : base;
        const int64_t pi = queue ? (int64_t)queue[slot] : slot;
        const int64_t qoff = q.offsets[pi] - q.word_base;
        const int64_t roff = r.offsets[pi] - r.word_base;
        const int32_t qlen = (int32_t)q.lengths[pi], rlen = (int32_t)r.lengths[pi];
        uint32_t Hr[R];
#pragma unroll
        for (int h = 0; h < R; ++h)
            Hr[h] = 0;
        // The reference window of row t, r[t-B .. t-B+16*NE), one 16-base word
        // per entry, slid by one base per row; the base entering at the bottom
        // is the top of `rw`, the word of positions t-B+16*NE.., reloaded every
        // 16 rows (t-B+16*NE is a multiple of 16 exactly when t is).  Words
        // before the reference start are zero and masked below.
        // em: the columns of row t inside the matrix; ep, eo: equality bits of two rows.
        uint32_t win[NE], em[NE], ep[NE], eo[NE];
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            win[i] = (i < B / 16) ? 0u : seq_word16(r, roff, i - B / 16);
            em[i] = eq_fields(B + 1, max(B + 1, rlen + B + 1), i);
            ep[i] = 0;
        }
        uint32_t e_last = SENT;
        uint32_t saved_lowkey = 0, bestkey = 0, thr = 127;
        int32_t bq = 0;
        uint32_t qw = 0, rw = 0;
        uint32_t qn = seq_word16(q, qoff, 0), rn = seq_word16(r, roff, RW0);  // next words
        // rows [B+1, B+1+inner) have all their columns inside, and rows [0, tail) none
        // past the reference end
        const int32_t tail = min(qlen, rlen - B);
        const uint32_t inner = (uint32_t)max(tail - (B + 1), 0);
        const int32_t steps = __reduce_max_sync(0xffffffffu, qlen > 0 ? qlen + 1 : 0);
        auto one_row = [&](int32_t t, uint32_t(&eq)[NE], const uint32_t(&ep)[NE]) {
            if ((uint32_t)(t - (B + 1)) >= inner) {
                if (t < tail) {  // the start of the reference: a column more than at t-1
#pragma unroll
                    for (int i = 0; i < NE; ++i)
                        em[i] = __funnelshift_l(i + 1 < NE ? em[i + 1 < NE ? i + 1 : i] : 0x55555555u,
                                                em[i], 2);
                } else {
                    const int32_t lo = max(B - t, 0), hi = t < qlen ? rlen - t + B : 0;
#pragma unroll
                    for (int i = 0; i < NE; ++i)
                        em[i] = eq_fields(lo, max(hi, lo), i);
                }
            }
            // equality bits of row t against its window r[t-B .. t+B]
            const uint32_t qrep = mad_hi_u32(qw, c.x4, 0u) * 0x55555555u;
            qw *= c.x4;
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                const uint32_t x = win[i] ^ qrep;
                eq[i] = ~(x | mad_hi_u32(x, c.half, 0u)) & em[i];
            }
            // slide the window one base for row t+1
#pragma unroll
            for (int i = 0; i < NE; ++i)
                win[i] = __funnelshift_l(i + 1 < NE ? win[i + 1 < NE ? i + 1 : i] : rw, win[i], 2);
            rw *= c.x4;
            // both rows' bits: the previous row's shifted so column NL+h sits one
            // bit above column h
            uint32_t cw[NBW];
#pragma unroll
            for (int i = 0; i < NBW; ++i)
                cw[i] = ep[BW0 + i] * c.x8 + mad_hi_u32(ep[BW0 + i + 1], c.x8, eq[i]);
            const uint32_t rk =
                pack16_cells<B>(Hr, cw, eq[NBW], (const char *)tab, l16, e_last, c);
            // row t-1 is complete: its first half came one step earlier; a key
            // above thr = bestkey | 127 has a larger H than the best so far
            const uint32_t rowkey = max(saved_lowkey, rk >> 16);
            if (rowkey > thr) {
                bestkey = rowkey;
                bq = t - 1;
            }
            thr = max(thr, rowkey | 127u);
            saved_lowkey = rk & 0xFFFFu;
        };
        for (int32_t t0 = 0; t0 < steps; t0 += 16) {
            qw = qn;  // words of rows t0 .. t0+15; fetch the following ones
            rw = rn;
            qn = seq_word16(q, qoff, (t0 >> 4) + 1);
            rn = seq_word16(r, roff, (t0 >> 4) + RW0 + 1);
            const int32_t t1 = min(t0 + 16, steps);
            for (int32_t t = t0; t < t1; t += 2) {  // an odd count runs one empty row more
                one_row(t, eo, ep);
                one_row(t + 1, ep, eo);
            }
        }
        const int32_t best = (int32_t)(bestkey >> 7);
        const int32_t bcol = 127 - (int32_t)(bestkey & 127u);
        if (valid) {
            gb2_sw_result res;
            res.score = best;
            res.query_end = best > 0 ? bq : 0;
            res.ref_end = best > 0 ? bq - B + bcol : 0;
            out[pi] = res;
        }
        if (!queue_counter)
            base += warps_total * 32;
    }
}

// Literal per-pair kernel: one thread per pair, int64 arithmetic, rows in
// global scratch.  Statement order follows align_cpu.mojo:239-309 exactly,
// so it is exact for every configuration and band.
__global__ void __launch_bounds__(128)
sw_literal_kernel(SeqView q, SeqView r, SwParams p, int32_t band, const int32_t *__restrict__ bands,
                  PairList pl, gb2_sw_result *__restrict__ out, int64_t *__restrict__ scratch,
                  int64_t stride)
{
    int64_t n;
    const int32_t *__restrict__ queue = pairs_resolve(pl, n);
    // few pairs: their warps spread over the blocks (each takes its own cache)
    const int64_t tid = warp_rank() * 32 + (threadIdx.x & 31);
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    int64_t *hp = scratch + tid * stride;
    for (int64_t slot = tid; slot < n; slot += nth) {
        const int64_t pi = queue ? (int64_t)queue[slot] : slot;
        const int64_t b = bands ? bands[pi] : band;
        const int64_t width = 2 * b + 1;
        int64_t *hc = hp + width, *ec = hp + 2 * width;
        const int64_t qlen = q.lengths[pi], rlen = r.lengths[pi];
        const uint64_t *qw = q.packed + (q.offsets[pi] - q.word_base);
        const uint64_t *rw = r.packed + (r.offsets[pi] - r.word_base);
        int64_t best = 0, bq = 0, br = 0;
        if (width > 0) {
            for (int64_t j = 0; j < width; ++j)
                hp[j] = 0;
            for (int64_t qi = 0; qi < qlen; ++qi) {
                for (int64_t j = 0; j < width; ++j) {
                    hc[j] = 0;
                    ec[j] = 0;
                }
                const int64_t qb = (int64_t)((qw[qi >> 5] >> (62 - 2 * (qi & 31))) & 3u);
                for (int64_t off = 0; off < width; ++off) {
                    const int64_t ri = qi - b + off;
                    if (ri < 0 || ri >= rlen)
                        continue;
                    const int64_t rb = (int64_t)((rw[ri >> 5] >> (62 - 2 * (ri & 31))) & 3u);
                    const int64_t sub = (qb == rb) ? p.match : p.mismatch;
                    const int64_t h_diag = hp[off];
                    const int64_t h_up = (off + 1 < width) ? hp[off + 1] : 0;
                    const int64_t h_left = (off > 0) ? hc[off - 1] : 0;
                    int64_t e1 = (off > 0) ? ec[off - 1] + p.ge : -1000000LL;
                    int64_t e2 = h_up + p.go + p.ge;
                    const int64_t e_val = e1 > e2 ? e1 : e2;
                    const int64_t f_val = h_left + p.go + p.ge;
                    int64_t cell = h_diag + sub;
                    cell = cell > e_val ? cell : e_val;
                    cell = cell > f_val ? cell : f_val;
                    cell = cell > 0 ? cell : 0;
                    hc[off] = cell;
                    ec[off] = e_val;
                    if (cell > best) {
                        best = cell;
                        bq = qi;
                        br = ri;
                    }
                }
                for (int64_t j = 0; j < width; ++j)
                    hp[j] = hc[j];
            }
        }
        gb2_sw_result res;
        res.score = (int32_t)best;
        res.query_end = (int32_t)bq;
        res.ref_end = (int32_t)br;
        out[pi] = res;
    }
}

// Naive baseline (GB2_FLAG_NAIVE): one 128-thread block per pair, launched
// over all pairs in input order with no planning, as the reference's
// launch_banded_sw does (genomics/gpu/align_gpu.mojo:482-492) -- but computing
// the CPU recurrence exactly.  Cell (qi, j) of the band runs at step
// s = 2*qi + j: its diag (qi-1, j) ran at s-2, its up (qi-1, j+1) and left
// (qi, j-1) at s-1, so the cells of one step (one parity of j) are
// independent and one row of H and E per band column, in shared memory, holds
// every value a step reads; a barrier separates the steps.  Skipped cells
// (reference position outside [0, rlen)) hold 0 as the reference's reset rows
// do (align_cpu.mojo:261-268).  int32 values (the host bounds every score).
__global__ void __launch_bounds__(128)
sw_naive_kernel(SeqView q, SeqView r, SwParams p, int32_t band, const int32_t *__restrict__ bands,
                int64_t n, gb2_sw_result *__restrict__ out)
{
    extern __shared__ int32_t nsm[];
    __shared__ unsigned long long red[4];
    const int64_t pi = blockIdx.x;
    if (pi >= n)
        return;
    const int32_t b = bands ? bands[pi] : band;
    const int32_t W = 2 * b + 1;
    int32_t *const Hs = nsm;
    int32_t *const Es = nsm + W;
    const int32_t qlen = (int32_t)q.lengths[pi], rlen = (int32_t)r.lengths[pi];
    const uint64_t *qw = q.packed + (q.offsets[pi] - q.word_base);
    const uint64_t *rw = r.packed + (r.offsets[pi] - r.word_base);
    for (int32_t j = threadIdx.x; j < W; j += blockDim.x) {
        Hs[j] = 0;
        Es[j] = 0;
    }
    __syncthreads();
    unsigned long long best = 0;  // H << 42 | (2^21-1 - qi) << 21 | (2^21-1 - j)
    const int32_t steps = qlen > 0 ? 2 * (qlen - 1) + W : 0;
    const int32_t goe = p.go + p.ge;
    for (int32_t st = 0; st < steps; ++st) {
        // active columns: parity of st, qi = (st - j) / 2 in [0, qlen)
        const int32_t jlo = max(st & 1, st - 2 * (qlen - 1));
        const int32_t jhi = min(W - 1, st);
        for (int32_t j = jlo + 2 * (int32_t)threadIdx.x; j <= jhi; j += 2 * (int32_t)blockDim.x) {
            const int32_t qi = (st - j) >> 1;
            const int32_t ri = qi - b + j;
            int32_t h = 0, e = 0;
            if (ri >= 0 && ri < rlen) {
                const int32_t qb = (int32_t)((qw[qi >> 5] >> (62 - 2 * (qi & 31))) & 3u);
                const int32_t rb = (int32_t)((rw[ri >> 5] >> (62 - 2 * (ri & 31))) & 3u);
                const int32_t sub = qb == rb ? p.match : p.mismatch;
                const int32_t h_diag = Hs[j];
                const int32_t h_up = j + 1 < W ? Hs[j + 1] : 0;
                const int32_t h_left = j > 0 ? Hs[j - 1] : 0;
                const int32_t e1 = j > 0 ? Es[j - 1] + p.ge : -1000000;
                e = max(e1, h_up + goe);
                h = max(max(h_diag + sub, e), max(h_left + goe, 0));
                if (h > 0) {
                    const unsigned long long key =
                        ((unsigned long long)h << 42) |
                        ((unsigned long long)(0x1FFFFF - qi) << 21) |
                        (unsigned long long)(0x1FFFFF - j);
                    best = key > best ? key : best;
                }
            }
            Hs[j] = h;
            Es[j] = e;
        }
        __syncthreads();
    }
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, off);
        best = o > best ? o : best;
    }
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i)
            best = red[i] > best ? red[i] : best;
        sw_store(out, pi, best, b);
    }
}

cudaError_t launch_sw_naive(SeqView q, SeqView r, SwParams p, int32_t band, const int32_t *bands,
                            int32_t max_band, int64_t n, gb2_sw_result *out, cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    if (n > 0x7fffffff || max_band > kSwNaiveMaxBand)
        return cudaErrorInvalidValue;
    static std::atomic<uint64_t> done{0};
    const cudaError_t attr = allow_smem(
        sw_naive_kernel, (int)(2 * (2 * kSwNaiveMaxBand + 1) * sizeof(int32_t)), done);
    if (attr != cudaSuccess)
        return attr;
    const size_t smem = (size_t)2 * (2 * (size_t)max_band + 1) * sizeof(int32_t);
    sw_naive_kernel<<<(unsigned)n, 128, smem, st>>>(q, r, p, band, bands, n, out);
    return cudaGetLastError();
}

template <int B, int G, int K>
static cudaError_t launch_band(SeqView q, SeqView r, SwParams p, PairList pl, gb2_sw_result *out,
                               int grid, cudaStream_t st)
{
    const int block = 128;
    const int64_t pairs_per_block = (block / 32) * (32 / G);
    int g = grid;
    if (g <= 0) {  // one pass over a host-known count
        if (pl.seg || pl.n <= 0)
            return pl.n <= 0 && !pl.seg ? cudaSuccess : cudaErrorInvalidValue;
        const int64_t need = (pl.n + pairs_per_block - 1) / pairs_per_block;
        g = (int)(need < 0x7fffffff ? need : 0x7fffffff);
    }
    sw_band_kernel<B, G, K><<<g, block, 0, st>>>(q, r, p, pl, out);
    return cudaGetLastError();
}

template <int B, int G, int K>
static int occ_band()
{
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sw_band_kernel<B, G, K>, 128, 0);
    return nb > 0 ? nb : 1;
}

template <int B>
static cudaError_t pack16_smem()
{
    static std::atomic<uint64_t> done{0};
    return allow_smem(sw_pack16_kernel<B>, kScoreTableBytes, done);
}

template <int B>
static int occ_pack16()
{
    int nb = 0;
    if (pack16_smem<B>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sw_pack16_kernel<B>, kPackThreads,
                                                      kScoreTableBytes) != cudaSuccess)
        cudaGetLastError();
    return nb > 0 ? nb : 1;
}

int sw_blocks_per_sm(int band_class, int variant)
{
    switch (band_class) {
    case 16 | kPack16: return occ_pack16<16>();
    case 32 | kPack16: return occ_pack16<32>();
    case 16: return variant == 1 ? occ_band<16, 2, 17>() : occ_band<16, 1, 33>();
    case 32:
        return variant == 1 ? occ_band<32, 2, 33>()
                            : (variant == 2 ? occ_band<32, 4, 17>() : occ_band<32, 1, 65>());
    case 64: return variant == 1 ? occ_band<64, 4, 33>() : occ_band<64, 2, 65>();
    case 128: return variant == 1 ? occ_band<128, 8, 33>() : occ_band<128, 4, 65>();
    default: return 4;
    }
}

int sw_pairs_per_block(int band_class, int variant)
{
    int G = 1;
    switch (band_class) {
    case 16 | kPack16:
    case 32 | kPack16: return kPackThreads;
    case 16: G = variant == 1 ? 2 : 1; break;
    case 32: G = variant == 1 ? 2 : (variant == 2 ? 4 : 1); break;
    case 64: G = variant == 1 ? 4 : 2; break;
    case 128: G = variant == 1 ? 8 : 4; break;
    default: return 128;
    }
    return 4 * (32 / G);
}

double sw_pack16_cost(int band, const SplitLoad &l)
{
    // 425 cycles per warp and row at band 32 (1,000,000 reads)
    return split_time(12.9 * (band + 1), 24.5 * (band + 1) + 200,
                      (double)l.pairs / 32 / (4.0 * l.sm_count), 1, l);
}

// variant selects (G, K) for a band class: 0 = default.
cudaError_t launch_sw(int band_class, int variant, SeqView q, SeqView r, SwParams p, int32_t band,
                      const int32_t *bands, PairList pl, gb2_sw_result *out, int64_t *scratch,
                      int64_t scratch_stride, int grid, cudaStream_t st)
{
    switch (band_class) {
    case 16 | kPack16:
    case 32 | kPack16: {
        int g = grid;
        if (g <= 0) {
            if (pl.seg || pl.n <= 0)
                return pl.n <= 0 && !pl.seg ? cudaSuccess : cudaErrorInvalidValue;
            g = (int)((pl.n + kPackThreads - 1) / kPackThreads);
        }
        const uint32_t gg = (uint32_t)(-(p.go + p.ge)), dm = (uint32_t)(p.match - p.mismatch);
        Pack16Consts c;
        c.x4 = 4;
        c.x8 = 8;
        c.x128 = 128;
        c.half = 0x80000000u;
        c.dm_pad = dm * 4;
        c.dm = dm;
        c.mmg2 = ((uint32_t)p.mismatch + gg) * 0x00010001u;
        c.ge2 = (uint32_t)(uint16_t)p.ge * 0x00010001u;
        c.ng2 = gg * 0x00010001u;
        c.one_f = 0x3C003C00u;
        c.neg_g_f = (0x8000u | gg) * 0x00010001u;
        const auto go = [&](auto kern) {
            kern<<<g, kPackThreads, kScoreTableBytes, st>>>(q, r, c, pl, out);
        };
        const bool b16 = band_class == (16 | kPack16);
        const cudaError_t e = b16 ? pack16_smem<16>() : pack16_smem<32>();
        if (e != cudaSuccess)
            return e;
        if (b16)
            go(sw_pack16_kernel<16>);
        else
            go(sw_pack16_kernel<32>);
        return cudaGetLastError();
    }
    case 16:
        if (variant == 1)
            return launch_band<16, 2, 17>(q, r, p, pl, out, grid, st);
        return launch_band<16, 1, 33>(q, r, p, pl, out, grid, st);
    case 32:
        if (variant == 1)
            return launch_band<32, 2, 33>(q, r, p, pl, out, grid, st);
        if (variant == 2)
            return launch_band<32, 4, 17>(q, r, p, pl, out, grid, st);
        return launch_band<32, 1, 65>(q, r, p, pl, out, grid, st);
    case 64:
        if (variant == 1)
            return launch_band<64, 4, 33>(q, r, p, pl, out, grid, st);
        return launch_band<64, 2, 65>(q, r, p, pl, out, grid, st);
    case 128:
        if (variant == 1)
            return launch_band<128, 8, 33>(q, r, p, pl, out, grid, st);
        return launch_band<128, 4, 65>(q, r, p, pl, out, grid, st);
    default: {
        if (grid <= 0)
            return cudaErrorInvalidValue;  // the literal kernel needs a sized scratch grid
        static std::atomic<uint64_t> done{0};
        const cudaError_t attr = prefer_l1(sw_literal_kernel, done);
        if (attr != cudaSuccess)
            return attr;
        sw_literal_kernel<<<grid, 128, 0, st>>>(q, r, p, band, bands, pl, out, scratch,
                                                scratch_stride);
        return cudaGetLastError();
    }
    }
}

}  // namespace gb2
